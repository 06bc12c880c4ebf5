// The recurrent KDA step on B200 (sm_100a): decode, draft verification, commit replay.
//
// One persistent, warp-specialised block per SM walks a list of units, unit = (request, head) of one layer (or
// (request, layer, head) for the commit replay).  Four roles, connected by mbarrier rings in shared memory:
//
//   mover (1 warp)      bulk-copies (cp.async.bulk) each unit's 128x128 state and each row's raw inputs from global
//                       memory into shared-memory rings, two or three units ahead of the arithmetic (replay: three or five);
//   prologue (2 to 8 warps)  turns a row's raw inputs into q, k, v, the decay multipliers, beta and sigmoid(gate)
//                       (short conv + SiLU, L2 norms, gates for the layer entry points, on four or eight warps; exp(g) for the core
//                       ones, on two; see kProWarpsOf);
//   recurrence (16 warps) keeps the unit's state in registers across its rows: warp w owns value rows 8w..8w+7,
//                       lane l key columns 4l..4l+3; per row the delta rule and the read-out; afterwards each warp
//                       stores its own 8 rows, a whole contiguous row per instruction;
//   epilogue (1 warp)   gated RMSNorm, bf16 outputs, replay saves.
//
// The state therefore crosses HBM once in each direction -- in as bulk transfers that are always that many
// units deep in flight, out as coalesced vector stores from the registers.  What roles load from global memory themselves (a unit's metadata, the
// layer prologue's conv weights and biases) is fetched ahead of the wait for the row or unit it belongs to.
//
// Arithmetic contract (what makes this a drop-in for the reference's kernels/kda.cu): every sum over the 128 key
// channels is formed as the reference forms it -- a lane's four consecutive channels added in order from zero,
// then the five-step xor butterfly over 32 lanes -- and nothing is contracted into an FMA (this file is compiled
// with --fmad=false --ftz=false --prec-div=true --prec-sqrt=true, the reference's build.rs flags).  The butterfly
// is evaluated as a reduce-scatter (kda.cu:30-33 applied to eight rows at once): the same additions in the same
// pairing, so the same bits, with 9 shuffles for eight rows instead of 40.  The kernels on small blocks further down lay a row
// across eight lanes (recurrence_octet.cuh) and add the same numbers in the same pairs, so a replayed prefix of a
// window has the bits of serial single-row steps
// (reference kernels/glm53f_kda.h:111-116, 166-168).
//
// Reference lines restated here: kernels/kda.cu:38-53 (update), 98-210 (chain_kernel), 214-253 (replay_kernel),
// 290-460 (argument checks and entry points).

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include "common.cuh"
#include "glm53f_kda.h"
#include "kda_internal.h"
#include "recurrence.cuh"
#include "recurrence_octet.cuh"

namespace kda {

__device__ int g_status = 0;
// Host-side settings of the diagnostic hook glm53f_kda_debug_wait_test: the bound of the recurrent kernels' waits, and
// a one-shot request that the next launch's block 0 leaves its first unit's state unfetched.
static unsigned long long g_wait_limit_ns = kWaitLimitNs;
// How glm53f_kda_chain_batch_bf16state runs a verify call (read-only states, saves on): 0 = the exact row-by-row form,
// 1 = the chunked tensor-core form; GLM53F_KDA_VERIFY=chunked makes 1 the default.
static std::atomic<int> g_layer_verify_mode{[] {
    const char* e = getenv("GLM53F_KDA_VERIFY");
    return e != nullptr && strcmp(e, "chunked") == 0 ? 1 : 0;
}()};
// How the bf16-state replays run: 0 = the exact row-by-row form, 1 = chunks of 16 rows on the tensor cores;
// GLM53F_KDA_COMMIT=chunked makes 1 the default.
static std::atomic<int> g_commit_mode{[] {
    const char* e = getenv("GLM53F_KDA_COMMIT");
    return e != nullptr && strcmp(e, "chunked") == 0 ? 1 : 0;
}()};
static int g_skip_first_state = 0;

int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0)
            n = v;
        else {
            cudaGetLastError();
            return 1;
        }
    }
    return n;
}

namespace {

enum Mode : int { kLayer = 0, kCore = 1, kReplay = 2 };

constexpr int kRecThreads = kRecWarps * 32;
// Prologue warps per mode.  The layer prologue (conv + SiLU, decay, gate: ~740 warp instructions per row in dependent
// chains of divisions and exponentials) on two warps was the slowest stage of a layer call (measured: decode through
// the layer symbol 0.746 -> 0.657 ms per step with four, the exact verify 24.5 -> 19.1 ms, an exact prefill lane
// 2.05 -> 1.57 ms, the replay 4.97 -> 4.72 ms); the core prologue is a widening and one exponential per channel, and
// there two more warps only take registers and issue slots from the recurrence (0.538 -> 0.566 ms).
// Single rows of bf16 states are cooked by two teams of four, a unit each in turn: a unit's 64 KiB take an SM 1.4 us at the copy rate, its row
// four warps as long or longer (16 slots bf16: 674 -> 594 us a step of 34 layers; f32 states, 2.9 us a unit, 916 -> 937 with two teams,
// and the exact verify's windows 1,346 -> 1,420, its recurrence being short of issue slots; one unit a block: 191 -> 203).
template <typename S, int MODE, bool ONE_UNIT = false>
constexpr int kProWarpsOf = MODE == 1 /* kCore */ ? 2 : MODE == 0 /* kLayer */ && sizeof(S) == 2 && !ONE_UNIT ? 8 : 4;
template <typename S, int MODE, bool ONE_UNIT = false>
constexpr int kThreadsOf = kRecThreads + kProWarpsOf<S, MODE, ONE_UNIT> * 32 + 64;  // + epilogue warp + mover warp

struct Params {
    int H, layers;
    long long units;
    const int32_t* cu_rows;
    const int32_t* keep;
    int rows1;
    // layer entry points
    const uint16_t* P;
    long long p_stride, b_off;
    const uint16_t* A;
    long long a_stride;
    const uint16_t* G;  // output-gate rows (layer: stride g_stride; core: dense, may be null)
    long long g_stride;
    const uint16_t* conv;
    const long long* conv_off;
    const uint16_t* cw;
    const float* a_log;
    const float* dt_bias;
    const uint16_t* norm_w;
    float eps, lower;
    // core entry points
    const uint16_t *q, *k, *v;
    const float* glog;
    const float* beta;
    int flags;
    // states
    const void* state_in;
    void* state_out;
    long long state_stride;
    const long long* state_off;
    // outputs (for the replay the saves are inputs)
    uint16_t* out;
    long long out_stride;
    float* k_save;
    uint16_t* v_save;
    float* g_save;
    float* b_save;
    long long kv_stride, b_stride;
    unsigned long long neg_zero2;  // two -0.0f: see mul2
    unsigned long long wait_limit_ns;  // bound of every device-side wait (no progress for this long: give up)
    int skip_first_state;  // diagnostic (glm53f_kda_debug_wait_test): block 0 does not fetch its first unit's state
};

// Raw-row slot layouts, byte offsets.
struct RawLayer {
    static constexpr int X = 0;                 // bf16 [4 taps][3 parts][128]
    static constexpr int A = X + 4 * 3 * 256;   // bf16 [128]
    static constexpr int GATE = A + 256;        // bf16 [128]
    static constexpr int B = GATE + 256;        // the 16 aligned bytes that hold the beta logit
    static constexpr int BYTES = B + 16;
};
struct RawCore {
    static constexpr int Q = 0, K = 256, V = 512;  // bf16 [128] each
    static constexpr int GLOG = 768;               // f32 [128]
    static constexpr int GATE = GLOG + 512;        // bf16 [128]
    static constexpr int B = GATE + 256;           // the 16 aligned bytes that hold beta (f32)
    static constexpr int BYTES = B + 16;
};
struct RawReplay {
    static constexpr int K = 0, G = 512;  // f32 [128] each
    static constexpr int V = 1024;        // bf16 [128]
    static constexpr int B = V + 256;     // the 16 aligned bytes that hold beta (f32)
    static constexpr int BYTES = B + 16;
};
template <int MODE>
struct RawOf;
template <>
struct RawOf<kLayer> { using T = RawLayer; };
template <>
struct RawOf<kCore> { using T = RawCore; };
template <>
struct RawOf<kReplay> { using T = RawReplay; };

constexpr int align_up(int x, int a) { return (x + a - 1) / a * a; }

// A cooked row: what the recurrence and the epilogue read.
struct Cooked {
    float q[DK], k[DK], v[DV], g[DK], sg[DV], ys[DV];
    float beta;
    int pad[3];
};

// What the recurrence needs to know of a unit, left by the mover beside its state; rows < 0: no more units.  (Read from global
// memory by the sixteen warps themselves, it queued behind their own stores of the state before.)
struct __align__(16) UnitInfo {
    long long s_elem;
    int rows;
};

template <typename S, int MODE>
struct Smem {
    static constexpr int kStateBytes = DV * DK * (int)sizeof(S);
    // States in flight: 96 KiB (bf16) or 128 KiB (f32); the replay of saves off their 16 bytes has 160 and 192.  More slow a long launch down, its reads then crowd out its writes (bf16 core, 5 and
    // 3 slots of the ring: 48 requests 1,303 and 1,220 us a step of 34 layers, 16 requests 462 and 459; 2: 1,214 and 488).
    static constexpr int kStateSlots = MODE == kReplay ? (sizeof(S) == 4 ? 3 : 5) : sizeof(S) == 4 ? 2 : 3;
    static constexpr int kRawSlots = MODE == kLayer ? (sizeof(S) == 4 ? 6 : 10) : sizeof(S) == 4 ? 3 : 4;  // raw-row ring depth
    static constexpr int kRowSlots = MODE == kLayer ? (sizeof(S) == 4 ? 6 : 10) : sizeof(S) == 4 ? 3 : 4;  // cooked-row ring depth
    static constexpr int kRawBytes = align_up(RawOf<MODE>::T::BYTES, 128);
    static constexpr int oState = 0;
    static constexpr int oRaw = oState + kStateSlots * kStateBytes;
    static constexpr int oCooked = oRaw + kRawSlots * kRawBytes;
    static constexpr int oScratch = oCooked + kRowSlots * (int)sizeof(Cooked);  // prologue scratch: q, k before norm
    static constexpr int oBars = oScratch + 4 * DK * 4;
    // barriers: st_full[S], st_empty[S], raw_full[R], raw_empty[R], row_full[C], y_full[C], row_empty[C]
    static_assert(MODE != kLayer || kRawSlots == kRowSlots, "layer_prologue_role: a free cooked slot implies a finished raw slot");
    // A warp sees its slots' parities only at its own rows; between two of them lie at most the other warps' windows' rows and a
    // single row of the other team, and no parity may come round in that time.
    static_assert(MODE != kLayer || kRowSlots > kProWarpsOf<S, kLayer>, "layer_prologue_role: rows between two of a warp's own");
    static constexpr int kBars = 2 * kStateSlots + 2 * kRawSlots + 3 * kRowSlots;
    static constexpr int oCtl = oBars + kBars * 8;  // progress, abort
    static constexpr int oUnits = align_up(oCtl + 16, (int)alignof(UnitInfo));  // UnitInfo per state slot
    static constexpr int kBytes = oUnits + kStateSlots * (int)sizeof(UnitInfo);
    static_assert(oUnits % alignof(UnitInfo) == 0, "a UnitInfo is read and written whole");
    static_assert(kBytes <= 232448, "shared memory budget");
};

struct Unit {
    int b, h, layer, rows;
    long long row0;
    long long s_elem;    // element offset of this head's state inside state_in / state_out
    long long conv_off;  // layer entry points: element offset of the request's conv window
    float a_log;         // layer entry points: A_log of the head
};

// The units of this block, u = blockIdx.x, blockIdx.x + gridDim.x, ...: (request, head) with the head fastest, or
// (request, layer, head) for the replay.  Indices advance by 32-bit arithmetic; the metadata of the next unit
// (row range, state and window offsets: loads from global memory) is fetched while the current one is processed, and stays as
// loaded until that unit's turn: arithmetic on it right after the loads would wait for them there, 1,500 cycles a unit and role.
// Every role waits for itself, behind what it can work out from the launch's parameters alone: with the index arithmetic and the
// first reads of the parameters behind the wait, a unit's metadata came 930 ns after it, 300 ns so.
__device__ __forceinline__ void predecessors_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <int MODE>
struct UnitIter {
    unsigned long long u;
    unsigned b, h, layer;
    unsigned step_b, step_h;  // gridDim.x = step_b * H + step_h
    bool ok;
    int r0, r1, kept;
    long long s_off, c_off;
    float a_log;

    __device__ __forceinline__ explicit UnitIter(const Params& p) {
        u = blockIdx.x;
        ok = u < (unsigned long long)p.units;
        const unsigned H = (unsigned)p.H, L = (unsigned)p.layers;
        h = blockIdx.x % H;
        step_b = gridDim.x / H;
        step_h = gridDim.x - step_b * H;
        const unsigned q = blockIdx.x / H;
        layer = MODE == kReplay ? q % L : 0u;
        b = MODE == kReplay ? q / L : q;
        r0 = r1 = kept = 0;
        s_off = c_off = 0;
        a_log = 0.0f;
    }
    // Behind the launch's predecessors: nothing global is read before this.
    __device__ __forceinline__ void begin(const Params& p) {
        predecessors_done();
        if (ok) fetch(p);
    }
    __device__ __forceinline__ void fetch(const Params& p) {
        if (p.cu_rows) {
            r0 = p.cu_rows[b];
            if (MODE != kReplay) r1 = p.cu_rows[b + 1];
        }
        if (MODE != kCore && p.keep) kept = p.keep[b];
        if (p.state_off) s_off = p.state_off[b];
        if (MODE == kLayer) {
            if (p.conv_off) c_off = p.conv_off[b];
            a_log = p.a_log[h];
        }
    }
    __device__ __forceinline__ bool valid() const { return ok; }
    __device__ __forceinline__ Unit current(const Params& p) const {
        Unit cur;
        cur.b = (int)b;
        cur.h = (int)h;
        cur.layer = (int)layer;
        cur.row0 = p.cu_rows ? r0 : 0;
        if (MODE == kReplay) {
            cur.rows = p.keep ? kept : p.rows1;
        } else {
            cur.rows = p.cu_rows ? r1 - r0 : p.rows1;
            // a commit by recomputation: only the request's first keep[b] rows
            if (MODE == kLayer && p.cu_rows && p.keep && kept < cur.rows) cur.rows = kept;
        }
        if (cur.rows < 0) cur.rows = 0;
        cur.s_elem = (long long)layer * p.state_stride + s_off + (long long)h * DV * DK;
        cur.conv_off = c_off;
        cur.a_log = a_log;
        return cur;
    }
    // The current unit; advances to the next one and starts fetching its metadata.
    __device__ __forceinline__ Unit take(const Params& p) {
        const Unit cur = current(p);
        u += gridDim.x;
        ok = u < (unsigned long long)p.units;
        const unsigned H = (unsigned)p.H;
        if (MODE == kReplay) {
            const unsigned nh = h + gridDim.x, dq = nh / H;
            h = nh - dq * H;
            const unsigned L = (unsigned)p.layers, nl = layer + dq, lq = nl / L;
            layer = nl - lq * L;
            b += lq;
        } else {  // the stride in (request, head) is fixed for the launch: no division per unit
            h += step_h;
            b += step_b;
            if (h >= H) {
                h -= H;
                ++b;
            }
        }
        if (ok) fetch(p);
        return cur;
    }
};

// Whether a unit without rows still has to move its state (out of place copy).
__device__ __forceinline__ bool copies_state(const Params& p) { return p.state_out != nullptr && p.state_out != p.state_in; }

struct Ring {
    int idx = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next(int n) {
        if (++idx == n) {
            idx = 0;
            phase ^= 1u;
        }
    }
};

// ---- the mover -----------------------------------------------------------------------------------------------
// The pieces of a row's raw inputs, one per lane: a lane works out its own piece's address and issues its own copy.  (Issued one
// after the other by one lane, the twenty pieces of a layer row took 3,500 cycles a row, longer than any other stage of a
// single-row launch.)  Pieces are 16-byte multiples except the "scalar chunk" (beta or its logit): for that one `src` is the
// element's own address and the mover copies the aligned 16 bytes around it, so the element lands at off + (address & 15).
struct Piece {
    int off, bytes;  // its place in the slot; bytes == 0: this lane has none
    bool scalar;
    int tap;                        // conv inputs: the tap; others 3, the row itself
    const unsigned char* base;      // the piece of row 0, head 0, layer 0
    long long row, head, layer;     // bytes from one row, head, layer to the next
    const unsigned char* window;    // conv inputs: the piece of head 0 in the first row of the window at offset 0
    long long window_row;
    __device__ __forceinline__ const unsigned char* at(const Unit& u, int r) const {
        const int x = r + tap;
        return (x < WINDOW ? window + u.conv_off * 2 + x * window_row : base + (u.row0 + x - WINDOW) * row) + u.h * head + u.layer * layer;
    }
};
// What does not depend on the unit, worked out while the launch's predecessors finish; a row is then one address a lane.  (As a branch
// for every kind of piece behind the metadata, 1 slot 204 -> 186 us a step of 34 layers, 16 slots core 495 -> 464.)
template <int MODE>
__device__ __forceinline__ Piece piece_of(const Params& p, int lane) {
    Piece x{0, 0, false, WINDOW, nullptr, 0, 0, 0, nullptr, 0};
    auto set = [&](int off, int bytes, bool scalar, const void* base, long long row, long long head, long long layer) {
        x.off = off; x.bytes = bytes; x.scalar = scalar;
        x.base = reinterpret_cast<const unsigned char*>(base);
        x.row = row; x.head = head; x.layer = layer;
    };
    if constexpr (MODE == kLayer) {
        if (lane < 3 * TAPS) {
            const long long from = (long long)(lane % 3) * p.H * DK;
            set(RawLayer::X + lane * 256, 256, false, p.P + from, p.p_stride * 2, 2 * DK, 0);
            x.tap = lane / 3;
            x.window = reinterpret_cast<const unsigned char*>(p.conv + from);
            x.window_row = 3LL * p.H * DK * 2;
        } else if (lane == 3 * TAPS) {
            set(RawLayer::A, 256, false, p.A, p.a_stride * 2, 2 * DK, 0);
        } else if (lane == 3 * TAPS + 1) {
            set(RawLayer::GATE, 256, false, p.G, p.g_stride * 2, 2 * DV, 0);
        } else if (lane == 3 * TAPS + 2) {
            set(RawLayer::B, 2, true, p.P + p.b_off, p.p_stride * 2, 2, 0);
        }
    } else if constexpr (MODE == kCore) {
        const long long row2 = 2LL * p.H * DK;
        if (lane == 0) set(RawCore::Q, 256, false, p.q, row2, 2 * DK, 0);
        else if (lane == 1) set(RawCore::K, 256, false, p.k, row2, 2 * DK, 0);
        else if (lane == 2) set(RawCore::V, 256, false, p.v, row2, 2 * DK, 0);
        else if (lane == 3) set(RawCore::GLOG, 512, false, p.glog, 2 * row2, 4 * DK, 0);
        else if (lane == 4) set(RawCore::B, 4, true, p.beta, 4LL * p.H, 4, 0);
        else if (lane == 5 && p.G) set(RawCore::GATE, 256, false, p.G, row2, 2 * DK, 0);
    } else {
        const long long row2 = 2LL * p.H * DK;
        if (lane == 0) set(RawReplay::K, 512, false, p.k_save, 2 * row2, 4 * DK, 4 * p.kv_stride);
        else if (lane == 1) set(RawReplay::G, 512, false, p.g_save, 2 * row2, 4 * DK, 4 * p.kv_stride);
        else if (lane == 2) set(RawReplay::V, 256, false, p.v_save, row2, 2 * DK, 2 * p.kv_stride);
        else if (lane == 3) set(RawReplay::B, 4, true, p.b_save, 4LL * p.H, 4, 4 * p.b_stride);
    }
    return x;
}

template <int MODE>
__device__ __forceinline__ uint32_t raw_row_bytes(const Params& p) {
    return MODE == kLayer ? (3 * TAPS + 2) * 256 + 16 : MODE == kCore ? 3 * 256 + 512 + 16 + (p.G ? 256 : 0) : 2 * 512 + 256 + 16;
}

// A block's first row (layer calls), issued by the prologue's first four warps, four pieces each, as soon as they know the unit: bulk copies
// of several lanes are issued one after the other, and the fifteen of a row took the mover 0.7 us, the state behind them (5 slots 338 ->
// 326 us a step of 34 layers, 16 slots 593 -> 578).  The mover counts their bytes (before or after they land); a row that is not
// aligned it copies itself, and all of a launch of one unit a block, whose prologue has the weights to fetch meanwhile (2 slots 205,
// so 223).
template <typename L>
__device__ __forceinline__ void first_row(const Params& p, unsigned char* smem, uint64_t* raw_full, const Piece& x, const Unit& un, int warp, int lane) {
    if (un.rows == 0 || warp >= 4) return;
    const uintptr_t src = reinterpret_cast<uintptr_t>(x.at(un, 0));
    if (__any_sync(0xffffffffu, !x.scalar && (src & 15) != 0)) return;
    if (x.bytes && (lane >> 2) == warp)
        bulk_load(smem + L::oRaw + x.off, reinterpret_cast<const void*>(src & ~uintptr_t(15)), x.scalar ? 16 : x.bytes, raw_full);
    __syncwarp();
}

template <typename S, int MODE, bool ONE_UNIT>
__device__ void mover_role(const Params& p, unsigned char* smem, uint64_t* bars, const WaitCtx& ctx, int lane) {
    using L = Smem<S, MODE>;
    uint64_t* st_full = bars;
    uint64_t* st_empty = st_full + L::kStateSlots;
    uint64_t* raw_full = st_empty + L::kStateSlots;
    uint64_t* raw_empty = raw_full + L::kRawSlots;
    UnitInfo* info = reinterpret_cast<UnitInfo*>(smem + L::oUnits);
    Ring st, raw;
    const bool copy0 = copies_state(p);
    UnitIter<MODE> units(p);
    const Piece x = piece_of<MODE>(p, lane);
    units.begin(p);
    auto row_in = [&](const Unit& un, int r) -> bool {
        if (!mbar_wait(&raw_empty[raw.idx], raw.phase ^ 1u, ctx, kStatusWaitRawEmpty)) return false;
        unsigned char* dst = smem + L::oRaw + raw.idx * L::kRawBytes;
        const uintptr_t src = reinterpret_cast<uintptr_t>(x.at(un, r));
        if (!__any_sync(0xffffffffu, !x.scalar && (src & 15) != 0)) {
            if (lane == 0) mbar_arrive_expect_tx(&raw_full[raw.idx], raw_row_bytes<MODE>(p));
            __syncwarp();
            if (x.bytes) bulk_load(dst + x.off, reinterpret_cast<const void*>(src & ~uintptr_t(15)), x.scalar ? 16 : x.bytes, &raw_full[raw.idx]);
        } else {  // unaligned rows: 2-byte copies, a lane its piece
            uint16_t* d = reinterpret_cast<uint16_t*>(dst + x.off + (x.scalar ? (int)(src & 15) : 0));
            for (int e = 0; e < x.bytes / 2; ++e) d[e] = reinterpret_cast<const uint16_t*>(src)[e];
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_full[raw.idx]);
        }
        __syncwarp();
        raw.next(L::kRawSlots);
        if (lane == 0) atomicAdd(const_cast<uint32_t*>(ctx.progress), 1u);
        return true;
    };
    constexpr bool kRowFirst = MODE == kLayer;  // a core row is cooked in no time (16 slots 459 us a step; 473 with the row first)
    // A block's second f32 state waits for its first one: windows of two or three rows leave room in the ring of rows, so that it is asked for at
    // once, and every SM's first state is then late (4 slots x 3 rows core 402 us a step of 34 layers, 420 without, 6 x 2 441 and 461; single
    // rows, where the second state is wanted soon, 319 both ways).
    constexpr bool kPaced = MODE == kCore && sizeof(S) == 4;
    bool first = true;
    for (; units.valid(); first = false) {
        const Unit un = units.take(p);
        if (un.rows == 0 && !copy0) continue;
        // A layer call's first row goes ahead of its state: the row has to be cooked before the state is wanted (5 slots 352 us a step, behind
        // it 369).
        if (kRowFirst && first && un.rows > 0) {
            const uintptr_t src = reinterpret_cast<uintptr_t>(x.at(un, 0));
            if (ONE_UNIT || __any_sync(0xffffffffu, !x.scalar && (src & 15) != 0)) {
                if (!row_in(un, 0)) return;
            } else {  // the prologue's warps issue its copies (first_row)
                if (lane == 0) mbar_arrive_expect_tx(&raw_full[raw.idx], raw_row_bytes<MODE>(p));
                __syncwarp();
                raw.next(L::kRawSlots);
            }
        }
        // The unit's state.
        if (!mbar_wait(&st_empty[st.idx], st.phase ^ 1u, ctx, kStatusWaitStateEmpty)) return;
        if (lane == 0) info[st.idx] = {un.s_elem, un.rows};
        if (p.skip_first_state && blockIdx.x == 0 && first) {
            // Diagnostic launch: nothing is copied and nobody is told, so the recurrence's wait for this state runs out.
        } else {
            unsigned char* dst = smem + L::oState + st.idx * L::kStateBytes;
            const unsigned char* src = reinterpret_cast<const unsigned char*>(p.state_in) + un.s_elem * (long long)sizeof(S);
            if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
                if (lane == 0) {
                    mbar_arrive_expect_tx(&st_full[st.idx], L::kStateBytes);
                    bulk_load(dst, src, L::kStateBytes, &st_full[st.idx]);
                }
            } else {  // a state that is not 16-byte aligned: element-wise copy by the whole warp
                const S* s = reinterpret_cast<const S*>(src);
                S* d = reinterpret_cast<S*>(dst);
                for (int e = lane; e < DV * DK; e += 32) d[e] = s[e];
                __syncwarp();
                if (lane == 0) mbar_arrive(&st_full[st.idx]);
            }
        }
        st.next(L::kStateSlots);
        // The other rows.
        for (int r = kRowFirst && first ? 1 : 0; r < un.rows; ++r)
            if (!row_in(un, r)) return;
        if constexpr (kPaced) {
            if (first && un.rows > 1 && !mbar_wait(&st_full[0], 0, ctx, kStatusWaitStateFull)) return;
        }
    }
    if (!mbar_wait(&st_empty[st.idx], st.phase ^ 1u, ctx, kStatusWaitStateEmpty)) return;
    if (lane == 0) {
        info[st.idx] = {0, -1};
        mbar_arrive(&st_full[st.idx]);
    }
}

// ---- the prologue --------------------------------------------------------------------------------------------
// L2 norm of scratch[0..127] by one warp in the reference's order (kda.cu:151-165): lane partial over 4
// consecutive channels from zero, butterfly, times 1/sqrt(ss + 1e-6), q also times 128^-0.5.
__device__ __forceinline__ void l2norm_warp(const float* x, float* y, int lane, bool is_q) {
    float v4[4], ss = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v4[i] = x[lane * 4 + i];
        ss = ss + v4[i] * v4[i];
    }
    ss = butterfly1(ss);
    const float inv = 1.0f / sqrtf(ss + 1e-6f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float t = v4[i] * inv;
        if (is_q) t = t * (1.0f / sqrtf((float)DK));
        y[lane * 4 + i] = t;
    }
}

template <typename S, int MODE>
__device__ void prologue_role(const Params& p, unsigned char* smem, uint64_t* bars, const WaitCtx& ctx, int t) {
    using L = Smem<S, MODE>;
    constexpr int kProThreads = kProWarpsOf<S, MODE> * 32;
    uint64_t* raw_full = bars + 2 * L::kStateSlots;
    uint64_t* raw_empty = raw_full + L::kRawSlots;
    uint64_t* row_full = raw_empty + L::kRawSlots;
    uint64_t* row_empty = row_full + 2 * L::kRowSlots;
    float* scratch = reinterpret_cast<float*>(smem + L::oScratch);
    const int warp = t >> 5, lane = t & 31;
    Ring raw, row;
    const bool copy0 = copies_state(p);
    // Whether the role's threads meet at barriers in every row (the L2 norms go through shared scratch).
    const bool syncs = MODE == kCore && (p.flags & GLM53F_KDA_CORE_L2NORM) != 0;
    UnitIter<MODE> units(p);
    units.begin(p);
    while (units.valid()) {
        const Unit un = units.take(p);
        if (un.rows == 0 && !copy0) continue;
        for (int r = 0; r < un.rows; ++r) {
            // A thread that gave up on a wait may not simply leave when the role synchronises below: the threads that got
            // through would wait for it at the role's barrier for ever.  There the decision is taken by all at that barrier.
            bool ready = mbar_wait(&raw_full[raw.idx], raw.phase, ctx, kStatusWaitRawFull);
            if (ready) ready = mbar_wait(&row_empty[row.idx], row.phase ^ 1u, ctx, kStatusWaitRowEmpty);
            if (!syncs && !ready) return;
            const unsigned char* in = smem + L::oRaw + raw.idx * L::kRawBytes;
            Cooked& ck = *reinterpret_cast<Cooked*>(smem + L::oCooked + row.idx * sizeof(Cooked));
            const long long gr = un.row0 + r;
            bool normalise = true;
            if (!ready) {
                // nothing to read: go to the vote
            } else if constexpr (MODE == kCore) {
                normalise = (p.flags & GLM53F_KDA_CORE_L2NORM) != 0;
                for (int c = t; c < DK; c += kProThreads) {
                    const float qv = bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(in + RawCore::Q)[c]);
                    const float kv = bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(in + RawCore::K)[c]);
                    if (normalise) {
                        scratch[c] = qv;
                        scratch[DK + c] = kv;
                    } else {
                        ck.q[c] = qv;
                        ck.k[c] = kv;
                    }
                    ck.v[c] = bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(in + RawCore::V)[c]);
                    ck.g[c] = expf(reinterpret_cast<const float*>(in + RawCore::GLOG)[c]);
                    if (p.G) ck.sg[c] = sigmoidf_(bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(in + RawCore::GATE)[c]));
                }
                if (t == 0) {
                    const uintptr_t addr = reinterpret_cast<uintptr_t>(p.beta + gr * p.H + un.h);
                    ck.beta = *reinterpret_cast<const float*>(in + RawCore::B + (addr & 15));
                }
            } else {
                normalise = false;
                for (int c = t; c < DK; c += kProThreads) {
                    ck.k[c] = reinterpret_cast<const float*>(in + RawReplay::K)[c];
                    ck.g[c] = reinterpret_cast<const float*>(in + RawReplay::G)[c];
                    ck.v[c] = bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(in + RawReplay::V)[c]);
                }
                if (t == 0) {
                    const uintptr_t addr = reinterpret_cast<uintptr_t>(p.b_save + un.layer * p.b_stride + gr * p.H + un.h);
                    ck.beta = *reinterpret_cast<const float*>(in + RawReplay::B + (addr & 15));
                }
            }
            if (syncs) {
                if (!named_bar_all(1, kProThreads, ready)) return;
                if (warp == 0) l2norm_warp(scratch, ck.q, lane, true);
                else if (warp == 1) l2norm_warp(scratch + DK, ck.k, lane, false);
                named_bar_sync(2, kProThreads);  // scratch may be overwritten by the next row
            }
            mbar_arrive(&row_full[row.idx]);   // one arrival per prologue thread: every thread's writes are released
            mbar_arrive(&raw_empty[raw.idx]);
            raw.next(L::kRawSlots);
            row.next(L::kRowSlots);
        }
    }
}

// The layer entry points' prologue.  Windows of several rows: a warp cooks a whole row (a lane four consecutive channels, so the
// norms stay in the warp and nothing meets at a barrier), the warps take rows in turn.  A row is a chain of about 1,000
// instructions, most of them divisions and exponentials; with all four warps on the same row a row left every 4,500 cycles and the
// recurrence, 1,600 a row, waited (6 slots x 4 to 8 rows, f32: 37 -> 32 us a layer).
// A warp skips the others' rows, so it has not itself seen the row that held the raw slot before, whose copy may land after later
// rows' copies: raw_full can be a phase behind what its parity says.  So every row waits for its cooked slot first.  The two rings
// are equally deep, and that slot is free only when the row before has been through the whole pipeline, its raw copy included.
//
// A launch of one unit a block (ONE_UNIT, an instance of the kernel to itself: the rule inside cost 16 single-row slots 1.5 %) waits for its
// first rows, and there four warps on a row are the shorter way: windows of 2, 4 and 8 rows of one slot 7.9, 10.6 and 15.4 us with
// a row per warp, 6.6, 9.3 and 14.7 so (two units a block, 4 rows: 16.4 against 17.2).
constexpr int kTogetherRows = 8, kTeamWarps = 4;
template <typename S, bool ONE_UNIT>
__device__ void layer_prologue_role(const Params& p, unsigned char* smem, uint64_t* bars, const WaitCtx& ctx, int warp, int lane) {
    using L = Smem<S, kLayer>;
    uint64_t* raw_full = bars + 2 * L::kStateSlots;
    uint64_t* raw_empty = raw_full + L::kRawSlots;
    uint64_t* row_full = raw_empty + L::kRawSlots;
    uint64_t* row_empty = row_full + 2 * L::kRowSlots;
    Ring raw, row;
    const bool copy0 = copies_state(p);
    const bool vec = ((reinterpret_cast<uintptr_t>(p.cw) | reinterpret_cast<uintptr_t>(p.dt_bias)) & 15) == 0;
    UnitIter<kLayer> units(p);
    if constexpr (ONE_UNIT) {
        units.begin(p);
    } else {
        const Piece x = piece_of<kLayer>(p, lane);
        units.begin(p);
        if (units.valid()) first_row<L>(p, smem, raw_full, x, units.current(p), warp, lane);
    }
    constexpr int together = ONE_UNIT ? kTogetherRows : 1;
    constexpr int kTeams = kProWarpsOf<S, kLayer, ONE_UNIT> / kTeamWarps;
    int turn = 0, team_turn = 0;
    // A warp whose wait gave up does not leave: the single-row units further on are cooked by all four warps, which meet there at
    // barriers.  It takes no more rows and goes on through the units to the next vote, which then sends all four home.
    bool dead = false;
    auto widen = [](uint2 w, float (&x)[4]) {
        x[0] = __uint_as_float(w.x << 16);
        x[1] = __uint_as_float(w.x & 0xffff0000u);
        x[2] = __uint_as_float(w.y << 16);
        x[3] = __uint_as_float(w.y & 0xffff0000u);
    };
    while (units.valid()) {
        const Unit un = units.take(p);
        if (un.rows == 0 && !copy0) continue;
        if (un.rows <= together) {
            // A single row is cooked by all four warps, a thread a channel: with one row a unit the next state is waited for anyway,
            // and the row's latency counts (16 slots, bf16: 0.670 ms a step of 34 layers, 0.696 with a row per warp; 1 slot 0.215
            // against 0.263).  ONE_UNIT: so are up to eight, there being no other unit's rows to work on meanwhile.
            if (kTeams > 1 && (team_turn++ & (kTeams - 1)) != (warp >> 2)) {
                for (int r = 0; r < un.rows; ++r) {
                    raw.next(L::kRawSlots);
                    row.next(L::kRowSlots);
                }
                continue;
            }
            const int tw = warp & (kTeamWarps - 1), c = tw * 32 + lane, bar = 1 + 2 * (warp >> 2);
            uint2 w[3];
#pragma unroll
            for (int part = 0; part < 3; ++part) {
                const uint16_t* cw = p.cw + (((long long)part * p.H + un.h) * DK + c) * TAPS;
                w[part] = vec ? *reinterpret_cast<const uint2*>(cw) : make_uint2((uint32_t)cw[0] | ((uint32_t)cw[1] << 16), (uint32_t)cw[2] | ((uint32_t)cw[3] << 16));
            }
            const float* dtb = p.dt_bias + (long long)un.h * DK + (c & (DK / 2 - 1));
            const float db[2] = {dtb[0], dtb[DK / 2]}, decay_rate = expf(un.a_log);
            // A row alone is there the sooner for two warps forming the norms and two the gates; of a window's rows, which follow one another
            // at the pace of the slowest warp, every thread takes its own channel's gates (one slot, windows of 4 to 8 rows, bf16:
            // 672 us a round of 34 layers with two and two, 646 so; 1 slot, a row alone: 189, so 193).
            auto cook = [&](auto alone) {
                for (int r = 0; r < un.rows; ++r, raw.next(L::kRawSlots), row.next(L::kRowSlots)) {
                    const bool ready = !dead && mbar_wait(&row_empty[row.idx], row.phase ^ 1u, ctx, kStatusWaitRowEmpty) && mbar_wait(&raw_full[raw.idx], raw.phase, ctx, kStatusWaitRawFull);
                    const unsigned char* in = smem + L::oRaw + raw.idx * L::kRawBytes;
                    Cooked& ck = *reinterpret_cast<Cooked*>(smem + L::oCooked + row.idx * sizeof(Cooked));
                    float* scratch = reinterpret_cast<float*>(smem + L::oScratch) + (warp >> 2) * 2 * DK;
                    if (ready) {
                        const uint16_t* x = reinterpret_cast<const uint16_t*>(in + RawLayer::X);
#pragma unroll
                        for (int part = 0; part < 3; ++part) {
                            float wt[TAPS], acc = 0.0f;
                            widen(w[part], wt);
#pragma unroll
                            for (int tap = 0; tap < TAPS; ++tap) acc = acc + wt[tap] * bf16_bits_to_f32(x[(tap * 3 + part) * DK + c]);
                            (part == 2 ? ck.v : scratch + part * DK)[c] = bf16_round(acc / (1.0f + expf(-acc)));
                        }
                    }
                    if (!named_bar_all(bar, kTeamWarps * 32, ready)) return false;  // all four leave together
                    if (tw == 0) l2norm_warp(scratch, ck.q, lane, true);
                    else if (tw == 1) l2norm_warp(scratch + DK, ck.k, lane, false);
                    auto beta = [&] {
                        const uintptr_t addr = reinterpret_cast<uintptr_t>(p.P + (un.row0 + r) * p.p_stride + p.b_off + un.h);
                        ck.beta = bf16_round(sigmoidf_(bf16_bits_to_f32(*reinterpret_cast<const uint16_t*>(in + RawLayer::B + (addr & 15)))));
                    };
                    auto gates = [&](int d, float bias) {
                        ck.g[d] = expf(p.lower * sigmoidf_(decay_rate * (bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(in + RawLayer::A)[d]) + bias)));
                        ck.sg[d] = sigmoidf_(bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(in + RawLayer::GATE)[d]));
                    };
                    if constexpr (decltype(alone)::value) {  // the two warps that have no norm to form, two channels a thread
                        if (tw >= 2) {
                            gates(c & (DK / 2 - 1), db[0]);
                            gates((c & (DK / 2 - 1)) + DK / 2, db[1]);
                        }
                        if (tw == 2 && lane == 0) beta();
                    } else {
                        if (tw == 2 && lane == 0) beta();
                        gates(c, tw < 2 ? db[0] : db[1]);
                    }
                    named_bar_sync(bar + 1, kTeamWarps * 32);
                    if (tw == 0 && lane == 0) {
                        mbar_arrive(&row_full[row.idx]);
                        mbar_arrive(&raw_empty[raw.idx]);
                    }
                }
                return true;
            };
            if (!ONE_UNIT || un.rows == 1) {
                if (!cook(std::true_type{})) return;
            } else {
                if (!cook(std::false_type{})) return;
            }
            continue;
        }
        for (int r = 0; r < un.rows; ++r, raw.next(L::kRawSlots), row.next(L::kRowSlots)) {
            if ((turn++ & (kProWarpsOf<S, kLayer, ONE_UNIT> - 1)) != warp || dead) continue;
            // The head's weights come straight from global memory, on their way while the row's inputs are waited for.
            uint4 w[3][2];
            float4 dtb;
            {
                const uint16_t* cw = p.cw + ((long long)un.h * DK + lane * 4) * TAPS;
                const float* db = p.dt_bias + (long long)un.h * DK + lane * 4;
#pragma unroll
                for (int part = 0; part < 3; ++part, cw += (long long)p.H * DK * TAPS) {
                    if (vec) {
                        w[part][0] = reinterpret_cast<const uint4*>(cw)[0];
                        w[part][1] = reinterpret_cast<const uint4*>(cw)[1];
                    } else {
                        auto two = [&](int e) { return (uint32_t)cw[e] | ((uint32_t)cw[e + 1] << 16); };
                        w[part][0] = make_uint4(two(0), two(2), two(4), two(6));
                        w[part][1] = make_uint4(two(8), two(10), two(12), two(14));
                    }
                }
                dtb = vec ? *reinterpret_cast<const float4*>(db) : make_float4(db[0], db[1], db[2], db[3]);
            }
            const bool ready = mbar_wait(&row_empty[row.idx], row.phase ^ 1u, ctx, kStatusWaitRowEmpty) && mbar_wait(&raw_full[raw.idx], raw.phase, ctx, kStatusWaitRawFull);
            if (!__all_sync(FULL, ready)) {  // the warp as a whole: the norms below shuffle across it
                dead = true;
                continue;
            }
            const unsigned char* in = smem + L::oRaw + raw.idx * L::kRawBytes;
            Cooked& ck = *reinterpret_cast<Cooked*>(smem + L::oCooked + row.idx * sizeof(Cooked));
            // Short conv + SiLU, one bf16 rounding (kda.cu:129-142); q and k then through the L2 norm (kda.cu:151-165).
#pragma unroll
            for (int part = 0; part < 3; ++part) {
                const uint32_t ww[8] = {w[part][0].x, w[part][0].y, w[part][0].z, w[part][0].w, w[part][1].x, w[part][1].y, w[part][1].z, w[part][1].w};
                float act[4], acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int tap = 0; tap < TAPS; ++tap) {
                    float x[4];
                    widen(*reinterpret_cast<const uint2*>(in + RawLayer::X + (tap * 3 + part) * 256 + lane * 8), x);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t t2 = ww[2 * c + (tap >> 1)];
                        acc[c] = acc[c] + __uint_as_float(tap & 1 ? t2 & 0xffff0000u : t2 << 16) * x[c];
                    }
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) act[c] = bf16_round(acc[c] / (1.0f + expf(-acc[c])));
                if (part == 2) {
                    *reinterpret_cast<float4*>(&ck.v[lane * 4]) = make_float4(act[0], act[1], act[2], act[3]);
                } else {
                    float ss = 0.0f;
#pragma unroll
                    for (int c = 0; c < 4; ++c) ss = ss + act[c] * act[c];
                    const float inv = 1.0f / sqrtf(butterfly1(ss) + 1e-6f);
                    float y[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        y[c] = act[c] * inv;
                        if (part == 0) y[c] = y[c] * (1.0f / sqrtf((float)DK));
                    }
                    *reinterpret_cast<float4*>(part == 0 ? &ck.q[lane * 4] : &ck.k[lane * 4]) = make_float4(y[0], y[1], y[2], y[3]);
                }
            }
            // Decay multiplier (kda.cu:143-146), sigmoid of the output gate (kda.cu:199-200) and beta (kda.cu:147-149).
            float a[4], gt[4], d[4], sg[4];
            widen(*reinterpret_cast<const uint2*>(in + RawLayer::A + lane * 8), a);
            widen(*reinterpret_cast<const uint2*>(in + RawLayer::GATE + lane * 8), gt);
            const float db[4] = {dtb.x, dtb.y, dtb.z, dtb.w}, decay_rate = expf(un.a_log);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                d[c] = expf(p.lower * sigmoidf_(decay_rate * (a[c] + db[c])));
                sg[c] = sigmoidf_(gt[c]);
            }
            *reinterpret_cast<float4*>(&ck.g[lane * 4]) = make_float4(d[0], d[1], d[2], d[3]);
            *reinterpret_cast<float4*>(&ck.sg[lane * 4]) = make_float4(sg[0], sg[1], sg[2], sg[3]);
            if (lane == 0) {
                const uintptr_t addr = reinterpret_cast<uintptr_t>(p.P + (un.row0 + r) * p.p_stride + p.b_off + un.h);
                ck.beta = bf16_round(sigmoidf_(bf16_bits_to_f32(*reinterpret_cast<const uint16_t*>(in + RawLayer::B + (addr & 15)))));
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&row_full[row.idx]);
                mbar_arrive(&raw_empty[raw.idx]);
            }
        }
    }
}

// ---- the recurrence ------------------------------------------------------------------------------------------
template <typename S, int MODE, bool LATE>
__device__ void recurrence_role(const Params& p, unsigned char* smem, uint64_t* bars, const WaitCtx& ctx, int warp, int lane) {
    using L = Smem<S, MODE>;
    uint64_t* st_full = bars;
    uint64_t* st_empty = st_full + L::kStateSlots;
    uint64_t* row_full = st_empty + L::kStateSlots + 2 * L::kRawSlots;
    uint64_t* y_full = row_full + L::kRowSlots;
    uint64_t* row_empty = y_full + L::kRowSlots;
    Ring st, row;
    const UnitInfo* info = reinterpret_cast<const UnitInfo*>(smem + L::oUnits);
    predecessors_done();
    for (;;) {
        if (!mbar_wait(&st_full[st.idx], st.phase, ctx, kStatusWaitStateFull)) return;
        const UnitInfo un = info[st.idx];
        if (un.rows < 0) return;
        unsigned char* slot = smem + L::oState + st.idx * L::kStateBytes;
        f32x2 s[kPairs][4];
        load_rows<S>(slot, warp, lane, s);
        const bool writes = p.state_out != nullptr;
        __syncwarp();  // the slot is free as soon as every lane's registers hold the state
        if (!LATE && lane == 0) mbar_arrive(&st_empty[st.idx]);
        for (int r = 0; r < un.rows; ++r) {
            if (!mbar_wait(&row_full[row.idx], row.phase, ctx, kStatusWaitRowFull)) return;
            Cooked& ck = *reinterpret_cast<Cooked*>(smem + L::oCooked + row.idx * sizeof(Cooked));
            f32x2 kk[4], gg[4];
            {
                const float4 k4 = *reinterpret_cast<const float4*>(&ck.k[lane * 4]);
                const float4 g4 = *reinterpret_cast<const float4*>(&ck.g[lane * 4]);
                kk[0] = pack2(k4.x, k4.x); kk[1] = pack2(k4.y, k4.y); kk[2] = pack2(k4.z, k4.z); kk[3] = pack2(k4.w, k4.w);
                gg[0] = pack2(g4.x, g4.x); gg[1] = pack2(g4.y, g4.y); gg[2] = pack2(g4.z, g4.z); gg[3] = pack2(g4.w, g4.w);
            }
            delta_rule(s, kk, gg, ck.v, warp, lane, ck.beta, p.neg_zero2);
            if constexpr (MODE != kReplay) {
                // Read-out y = S q, rounded to bf16 (kda.cu:172-179).
                const float4 q4 = *reinterpret_cast<const float4*>(&ck.q[lane * 4]);
                const f32x2 qq[4] = {pack2(q4.x, q4.x), pack2(q4.y, q4.y), pack2(q4.z, q4.z), pack2(q4.w, q4.w)};
                const float o = rows_dot(s, qq, lane, p.neg_zero2);
                if ((lane & 3) == 0) ck.ys[warp * kRowsPerLane + (lane >> 2)] = bf16_round(o);
            }
            // A bf16 state is rounded after every row, after its read-out; after the last row the store rounds.
            if constexpr (sizeof(S) == 2) {
                if (r + 1 < un.rows || !writes) round_rows(s);
            }
            __syncwarp();
            if (lane == 0) {
                if (MODE != kReplay) mbar_arrive(&y_full[row.idx]);
                else mbar_arrive(&row_empty[row.idx]);
                if (warp == 0) atomicAdd(const_cast<uint32_t*>(ctx.progress), 1u);
            }
            row.next(L::kRowSlots);
        }
        if constexpr (LATE) {  // see late_release
            __syncwarp();
            if (lane == 0) mbar_arrive(&st_empty[st.idx]);
        }
        if (writes) {
            // Straight from the registers: per row a lane stores its 4 consecutive elements (8 or 16 bytes), a warp a
            // whole contiguous row.  Each warp wrote nothing but the rows it read, so in place is safe.
            S* dst = reinterpret_cast<S*>(p.state_out) + un.s_elem;
            store_rows_global<S>(dst, warp, lane, s);
        }
        st.next(L::kStateSlots);
    }
}

// ---- the epilogue --------------------------------------------------------------------------------------------
template <typename S, int MODE>
__device__ void epilogue_role(const Params& p, unsigned char* smem, uint64_t* bars, const WaitCtx& ctx, int lane) {
    using L = Smem<S, MODE>;
    uint64_t* y_full = bars + 2 * L::kStateSlots + 2 * L::kRawSlots + L::kRowSlots;
    uint64_t* row_empty = y_full + L::kRowSlots;
    Ring row;
    const bool copy0 = copies_state(p);
    const bool gated = MODE == kLayer || p.G != nullptr;
    float nw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    UnitIter<MODE> units(p);
    units.begin(p);
    if (gated)
#pragma unroll
        for (int i = 0; i < 4; ++i) nw[i] = bf16_bits_to_f32(p.norm_w[lane * 4 + i]);
    while (units.valid()) {
        const Unit un = units.take(p);
        if (un.rows == 0 && !copy0) continue;
        for (int r = 0; r < un.rows; ++r) {
            if (!mbar_wait(&y_full[row.idx], row.phase, ctx, kStatusWaitYFull)) return;
            const Cooked& ck = *reinterpret_cast<const Cooked*>(smem + L::oCooked + row.idx * sizeof(Cooked));
            const long long gr = un.row0 + r;
            float y[4];
            {
                const float4 y4 = *reinterpret_cast<const float4*>(&ck.ys[lane * 4]);
                y[0] = y4.x; y[1] = y4.y; y[2] = y4.z; y[3] = y4.w;
            }
            uint16_t o[4];
            if (gated) {  // kda.cu:188-201
                float ss = 0.0f;
#pragma unroll
                for (int i = 0; i < 4; ++i) ss = ss + y[i] * y[i];
                ss = butterfly1(ss);
                const float rinv = 1.0f / sqrtf(ss / (float)DV + p.eps);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float yn = y[i] * rinv;
                    const float yw = nw[i] * yn;
                    o[i] = f32_to_bf16_bits(yw * ck.sg[lane * 4 + i]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) o[i] = f32_to_bf16_bits(y[i]);
            }
            uint16_t* dst = p.out + gr * p.out_stride + (long long)un.h * DV + lane * 4;
            if ((reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
                *reinterpret_cast<uint2*>(dst) = make_uint2((uint32_t)o[0] | ((uint32_t)o[1] << 16), (uint32_t)o[2] | ((uint32_t)o[3] << 16));
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) dst[i] = o[i];
            }
            if (p.k_save != nullptr) {  // kda.cu:181-186
                const long long base = (gr * p.H + un.h) * DK + lane * 4;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    p.k_save[base + i] = ck.k[lane * 4 + i];
                    p.g_save[base + i] = ck.g[lane * 4 + i];
                    p.v_save[base + i] = f32_to_bf16_bits(ck.v[lane * 4 + i]);
                }
                if (lane == 0) p.b_save[gr * p.H + un.h] = ck.beta;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&row_empty[row.idx]);
            row.next(L::kRowSlots);
        }
    }
}

// ---- the kernel ----------------------------------------------------------------------------------------------
template <typename S, int MODE, bool ONE_UNIT = false, bool LATE = false>
__global__ void __launch_bounds__(kThreadsOf<S, MODE, ONE_UNIT>, 1) recurrent_kernel(const __grid_constant__ Params p) {
    using L = Smem<S, MODE>;
    constexpr int kProWarps = kProWarpsOf<S, MODE, ONE_UNIT>, kProThreads = kProWarps * 32;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::oBars);
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + L::oCtl);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        uint64_t* b = bars;
        for (int i = 0; i < L::kStateSlots; ++i) mbar_init(b++, 1);                                // st_full
        for (int i = 0; i < L::kStateSlots; ++i) mbar_init(b++, kRecWarps);                        // st_empty
        for (int i = 0; i < L::kRawSlots; ++i) mbar_init(b++, 1);                                     // raw_full
        for (int i = 0; i < L::kRawSlots; ++i) mbar_init(b++, MODE == kLayer ? 1 : kProThreads);         // raw_empty
        for (int i = 0; i < L::kRowSlots; ++i) mbar_init(b++, MODE == kLayer ? 1 : kProThreads);         // row_full
        for (int i = 0; i < L::kRowSlots; ++i) mbar_init(b++, kRecWarps);                             // y_full
        for (int i = 0; i < L::kRowSlots; ++i) mbar_init(b++, MODE == kReplay ? kRecWarps : 1);       // row_empty
        ctl[0] = 0u;
        ctl[1] = 0u;
        mbar_init_fence();
    }
    __syncthreads();
    // Programmatic dependent launch: let the next kernel of the stream be scheduled onto SMs as this grid's blocks
    // retire (its block set-up then overlaps this grid's tail); the roles touch no global memory before every earlier
    // grid of the stream has completed and flushed (predecessors_done).  Both are no-ops for a launch without the attribute.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const WaitCtx ctx{ctl, ctl + 1, &g_status, p.wait_limit_ns};
    if (warp < kRecWarps) {
        recurrence_role<S, MODE, LATE>(p, smem, bars, ctx, warp, lane);
    } else if (warp < kRecWarps + kProWarps) {
        if constexpr (MODE == kLayer) layer_prologue_role<S, ONE_UNIT>(p, smem, bars, ctx, warp - kRecWarps, lane);
        else prologue_role<S, MODE>(p, smem, bars, ctx, tid - kRecThreads);
    } else if (warp == kRecWarps + kProWarps) {
        if (MODE != kReplay) epilogue_role<S, MODE>(p, smem, bars, ctx, lane);
    } else {
        mover_role<S, MODE, ONE_UNIT>(p, smem, bars, ctx, lane);
    }
    // No thread leaves while bulk loads into this block's shared memory may still be in flight: the mover issues a
    // load only after its consumers freed the slot, and every consumer role waits for every load before it ends,
    // except after an abort -- then give outstanding loads a bounded time to land.
    if (ctl[1]) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 2000000ull) {
        }
    }
    __syncthreads();
}

// ---- the core step on many small blocks ------------------------------------------------------------------------
// The same arithmetic (recurrence_octet.cuh: the bits are those of the kernel above and of the reference) for the core entry
// points without fused norms, arranged for windows: a block of four warps owns HALF of a unit -- 64 of its 128 value rows, 16 a
// warp, which never interact with the others -- loads that part of the state straight from global memory into registers, cooks
// each row's inputs itself (128 threads, one channel each: widen q, k, v, exp of the log decay, beta; loaded a row ahead, into the other
// of two buffers, so a row takes one barrier), steps through the request's rows and stores its rows of the state back.  No rings, no
// bulk copies: four such blocks on an SM are two units' serial rows at once.  Used for the exact verify and, with more than one and at
// most two units an SM, for decode of any number of rows, the row-by-row fallback of the core prefill among it (core_entry).
constexpr int kSmallWarps = 4, kSmallThreads = kSmallWarps * 32, kR = 4, kSmallParts = DV / (4 * kR * kSmallWarps), kSmallPerSm = 4;

// DECODE: calls without saves.  A unit's halves are neighbours, which read the same rows; in a verify so are a request's units, in a decode
// those of different requests (a grid of heads by requests): neighbouring blocks share an SM when there are four for each, and one long
// request among single rows had its blocks on a few (288 units, one of 18 requests with 40 rows, 34 launches: bf16 2,465 -> 1,485 us, f32
// 2,244 -> 1,320).
template <typename S, bool DECODE>
__global__ void __launch_bounds__(kSmallThreads, kSmallPerSm) core_small_kernel(const __grid_constant__ Params p) {
    __shared__ __align__(16) float sq[2][DK], sk[2][DK], sg[2][DK], sv[2][DV];
    __shared__ float sbeta[2];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const long long unit = blockIdx.x / kSmallParts;
    const int part = blockIdx.x % kSmallParts, uw = part * kSmallWarps + warp;  // this warp's place among the unit's
    const int b = (int)(DECODE ? unit : unit / p.H), h = (int)(DECODE ? blockIdx.y : unit % p.H);
    const int r0 = p.cu_rows[b], rows = max(p.cu_rows[b + 1] - r0, 0);
    const bool writes = p.state_out != nullptr;
    if (rows == 0 && !copies_state(p)) return;
    const long long s_elem = p.state_off[b] + (long long)h * DV * DK;
    const int mine = uw * 4 * kR + oct::row_of_lane<kR>(lane);
    struct Raw {  // a row's inputs, this thread's channel
        uint16_t q, k, v;
        float g, beta;
    } next{};
    auto fetch = [&](int r) {
        const long long gr = (long long)r0 + r, at = (gr * p.H + h) * DK + t;
        next.q = p.q[at];
        next.k = p.k[at];
        next.v = p.v[at];
        next.g = p.glog[at];
        if (t == 0) next.beta = p.beta[gr * p.H + h];
    };
    // bf16: ahead of the state, and no rounding of a state that nobody reads: windows of one row of 6 slots 287 -> 246 us a step of 34
    // layers, of four rows 530 -> 491 (a quarter of a unit a block on the step of recurrence.cuh: 272 and 553).  f32: behind it (2 slots x
    // 16 rows 808 us, ahead 841).
    constexpr bool kRowFirst = sizeof(S) == 2;
    if (kRowFirst && rows > 0) fetch(0);
    f32x2 s[kR][oct::kRowPairs];
    oct::load_rows(reinterpret_cast<const S*>(p.state_in) + s_elem, uw, lane, s);
    if (!kRowFirst && rows > 0) fetch(0);
    for (int r = 0; r < rows; ++r) {
        const long long gr = (long long)r0 + r, at = (gr * p.H + h) * DK + t;
        const int buf = r & 1;  // the row before may still be read from the other buffer
        const float kf = bf16_bits_to_f32(next.k), gf = expf(next.g);
        sq[buf][t] = bf16_bits_to_f32(next.q);
        sk[buf][t] = kf;
        sg[buf][t] = gf;
        sv[buf][t] = bf16_bits_to_f32(next.v);
        if (t == 0) sbeta[buf] = next.beta;
        if (!DECODE && part == 0) {
            p.k_save[at] = kf;
            p.g_save[at] = gf;
            p.v_save[at] = next.v;
            if (t == 0) p.b_save[gr * p.H + h] = next.beta;
        }
        __syncthreads();
        if (r + 1 < rows) fetch(r + 1);
        {
            f32x2 kk[oct::kRowPairs], gg[oct::kRowPairs];
            oct::load_leaves(sg[buf], lane, gg);
            oct::load_leaves(sk[buf], lane, kk);
            oct::delta_rule(s, kk, gg, sv[buf][mine], lane, sbeta[buf], p.neg_zero2);
        }
        f32x2 qq[oct::kRowPairs];
        oct::load_leaves(sq[buf], lane, qq);
        const float o = oct::rows_dot(s, qq, lane, p.neg_zero2);
        if (oct::first_of_row<kR>(lane)) p.out[gr * p.out_stride + (long long)h * DV + mine] = f32_to_bf16_bits(o);
        if constexpr (sizeof(S) == 2) {
            if (r + 1 < rows) oct::round_rows(s);  // the last row's rounding is the store's, if there is one
        }
    }
    if (writes) oct::store_rows(reinterpret_cast<S*>(p.state_out) + s_elem, uw, lane, s);
}

template <typename S>
int launch_small(const Params& p, cudaStream_t stream) {
    Params q = p;
    q.neg_zero2 = 0x8000000080000000ull;
    cudaLaunchConfig_t cfg = {};
    const bool decode = p.k_save == nullptr;
    cfg.gridDim = decode ? dim3((unsigned)(p.units / p.H * kSmallParts), (unsigned)p.H) : dim3((unsigned)(p.units * kSmallParts));
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = early_attribute(attr[0]);
    return (int)cudaLaunchKernelEx(&cfg, decode ? core_small_kernel<S, true> : core_small_kernel<S, false>, q);
}

// ---- the replay on many small blocks ---------------------------------------------------------------------------
// A commit replays keep[b] saved rows onto every (request, layer, head) state: no read-out, no norms, inputs that are already
// cooked.  As above a block of four warps takes half of a unit; a row's saves come into shared memory by asynchronous copies, three
// rows ahead.  Same delta rule, same rounding points (a bf16 state is rounded after every row), so the bits are the persistent
// kernel's and the reference's.  Measured at 48 slots x 34 layers, accepted prefixes drawn from 0..16, bf16: 4.71 ms on the persistent
// kernel, 3.63 ms with eight value rows a warp read straight from global memory; see recurrence_octet.cuh for the step.
constexpr int kReplayAhead = 3;
struct __align__(16) ReplayRow {
    float k[DK], g[DK];
    uint16_t v[DV + 4];  // the 8-byte words that hold the row's values: they begin v_lead elements in
    float beta;
};

template <typename S>
__global__ void __launch_bounds__(kSmallThreads, kSmallPerSm) replay_small_kernel(const __grid_constant__ Params p) {
    static_assert((kReplayAhead & (kReplayAhead + 1)) == 0, "ring index");
    __shared__ ReplayRow ring[kReplayAhead + 1];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const long long unit = blockIdx.x / kSmallParts;
    const int uw = (int)(blockIdx.x % kSmallParts) * kSmallWarps + warp;  // this warp's place among the unit's
    const int h = (int)(unit % p.H), layer = (int)((unit / p.H) % p.layers), b = (int)(unit / ((long long)p.H * p.layers));
    const long long r0 = p.cu_rows ? p.cu_rows[b] : 0;
    int rows = p.keep ? p.keep[b] : p.rows1;
    if (rows < 0) rows = 0;
    if (rows == 0 && !copies_state(p)) return;
    const long long s_elem = (long long)layer * p.state_stride + (p.state_off ? p.state_off[b] : 0) + (long long)h * DV * DK;
    const long long kv_base = (long long)layer * p.kv_stride, b_base = (long long)layer * p.b_stride;
    // Values at any element: the aligned words around them are copied (rows and layers are multiples of four elements apart).
    const int v_lead = (int)((reinterpret_cast<uintptr_t>(p.v_save) & 7) / 2);
    auto fetch = [&](int r) {  // 16 bytes of k or of the decay a thread, 8 of v; beta
        if (r < rows) {
            const long long rh = (r0 + r) * p.H + h, at = kv_base + rh * DK;
            ReplayRow& x = ring[r & kReplayAhead];
            if (t < 32) oct::copy16(&x.k[t * 4], p.k_save + at + t * 4);
            else if (t < 64) oct::copy16(&x.g[(t - 32) * 4], p.g_save + at + (t - 32) * 4);
            else if (t < 96 || (t == 96 && v_lead != 0)) oct::copy8(&x.v[(t - 64) * 4], p.v_save + at - v_lead + (t - 64) * 4);
            else if (t == 97) oct::copy4(&x.beta, p.b_save + b_base + rh);
        }
        oct::copies_commit();
    };
#pragma unroll
    for (int r = 0; r < kReplayAhead; ++r) fetch(r);
    f32x2 s[kR][oct::kRowPairs];
    oct::load_rows(reinterpret_cast<const S*>(p.state_in) + s_elem, uw, lane, s);
    const int mine = uw * 4 * kR + oct::row_of_lane<kR>(lane);
    for (int r = 0; r < rows; ++r) {
        oct::copies_wait<kReplayAhead - 1>();
        __syncthreads();  // row r is there for all, and nobody reads row r - 1 any more
        fetch(r + kReplayAhead);
        const ReplayRow& x = ring[r & kReplayAhead];
        f32x2 kk[oct::kRowPairs], gg[oct::kRowPairs];
        oct::load_leaves(x.g, lane, gg);
        oct::load_leaves(x.k, lane, kk);
        oct::delta_rule(s, kk, gg, bf16_bits_to_f32(x.v[v_lead + mine]), lane, x.beta, p.neg_zero2);
        if constexpr (sizeof(S) == 2) {
            if (r + 1 < rows) oct::round_rows(s);  // the last row's rounding is the store's
        }
    }
    oct::store_rows(reinterpret_cast<S*>(p.state_out) + s_elem, uw, lane, s);
}

// A launch whose blocks find an SM each -- a layer's replay of a few heads -- is over when its longest chain of rows is.  A warp then
// takes eight value rows on the step of recurrence.cuh: what a lane needs of a saved row is a 16-byte piece of k and of the decay, one v and
// beta, loaded into registers while the row before is worked on; nothing is shared, so no row waits at a barrier.  (16 rows, 16 units, 34
// launches: 225 us f32, 265 bf16; on replay_small_kernel 340 and 382; rows two or three ahead in registers 240 to 270 and 272 to 406.)
constexpr int kFewParts = kRecWarps / kSmallWarps;
struct FewRow {
    float4 k, g;
    uint16_t v;  // bf16 bits, widened when the row's turn comes: a conversion at the load would wait for it there and then
    float beta;
};
__device__ __forceinline__ FewRow few_row(const Params& p, long long kv_base, long long b_base, long long gr, int h, int uw, int lane) {
    FewRow x;
    const long long at = kv_base + (gr * p.H + h) * DK;
    x.k = *reinterpret_cast<const float4*>(p.k_save + at + lane * 4);
    x.g = *reinterpret_cast<const float4*>(p.g_save + at + lane * 4);
    x.v = p.v_save[at + uw * kRowsPerLane + (lane >> 2)];
    x.beta = p.b_save[b_base + gr * p.H + h];
    return x;
}

template <typename S>
__global__ void __launch_bounds__(kSmallThreads, sizeof(S) == 4 ? 6 : 8) replay_few_kernel(const __grid_constant__ Params p) {
    grid_ready();
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const long long unit = blockIdx.x / kFewParts;
    const int uw = (int)(blockIdx.x % kFewParts) * kSmallWarps + warp;  // this warp's place among the unit's 16
    const int h = (int)(unit % p.H), layer = (int)((unit / p.H) % p.layers), b = (int)(unit / ((long long)p.H * p.layers));
    const long long r0 = p.cu_rows ? p.cu_rows[b] : 0;
    int rows = p.keep ? p.keep[b] : p.rows1;
    if (rows < 0) rows = 0;
    if (rows == 0 && !copies_state(p)) return;
    const long long s_elem = (long long)layer * p.state_stride + (p.state_off ? p.state_off[b] : 0) + (long long)h * DV * DK;
    const long long kv_base = (long long)layer * p.kv_stride, b_base = (long long)layer * p.b_stride;
    f32x2 s[kPairs][4];
    load_rows_global<S>(reinterpret_cast<const S*>(p.state_in) + s_elem, uw, lane, s);
    FewRow cur{};
    if (rows > 0) cur = few_row(p, kv_base, b_base, r0, h, uw, lane);
    for (int r = 0; r < rows; ++r) {
        FewRow nxt = cur;
        if (r + 1 < rows) nxt = few_row(p, kv_base, b_base, r0 + r + 1, h, uw, lane);
        const f32x2 kk[4] = {pack2(cur.k.x, cur.k.x), pack2(cur.k.y, cur.k.y), pack2(cur.k.z, cur.k.z), pack2(cur.k.w, cur.k.w)};
        const f32x2 gg[4] = {pack2(cur.g.x, cur.g.x), pack2(cur.g.y, cur.g.y), pack2(cur.g.z, cur.g.z), pack2(cur.g.w, cur.g.w)};
        delta_rule_v(s, kk, gg, bf16_bits_to_f32(cur.v), lane, cur.beta, p.neg_zero2);
        if constexpr (sizeof(S) == 2) {
            if (r + 1 < rows) round_rows(s);  // the last row's rounding is the store's
        }
        cur = nxt;
    }
    store_rows_global<S>(reinterpret_cast<S*>(p.state_out) + s_elem, uw, lane, s);
}

template <typename S>
int launch_replay_small(const Params& p, cudaStream_t stream) {
    Params q = p;
    q.neg_zero2 = 0x8000000080000000ull;
    // Up to a block an SM with bf16 states, to three on four SMs with f32 ones.  34 launches of 16 rows, bf16, 37 and 38 units: 319 and (three rounds
    // of four blocks) 805 us on the one, 374 and 374 on the other; f32, 24 and 32: 288 and 426 against 332 and 346.
    const long long sms = sm_count();
    const bool few = p.units * kFewParts * (sizeof(S) == 4 ? 4 : 3) <= 3 * sms;
    const long long blocks = p.units * (few ? kFewParts : kSmallParts);
    auto* kernel = few ? replay_few_kernel<S> : replay_small_kernel<S>;
    // Blocks that start while the launch before them still runs would crowd onto the SMs that it left free, and a launch takes as
    // long as the fullest SM: shared memory that nobody uses keeps it to its fair share of blocks an SM (34 launches of 16 rows, 64 units, f32 and
    // bf16: 729 and 800 us without it, 368 and 396 so).
    constexpr size_t kSmemPerSm = 227 * 1024, kMostPad = kSmemPerSm / 2 + 1024;
    const size_t own = few ? 0 : (kReplayAhead + 1) * sizeof(ReplayRow);
    const long long share = (blocks + sms - 1) / sms;
    const size_t pad = share < kSmallPerSm ? kSmemPerSm / (size_t)(share + 1) + 1024 - own : 0;
    static int configured[2] = {-1, -1};
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured[few] != dev) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostPad);
        if (e != cudaSuccess) return (int)e;
        configured[few] = dev;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = pad;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = early_attribute(attr[0]);
    return (int)cudaLaunchKernelEx(&cfg, kernel, q);
}

// Core launches: when a state's slot is free for the next one.  At once, the next read is as early as can be, which is what a launch of few
// units a block wants; many units are through sooner when reads keep less far ahead of the writes.  Single rows, us a step of 34 layers,
// early and late: bf16, 16, 32, 40 and 44 slots 458 and 484, 833 and 845, 1,031 and 1,038, 1,121 and 1,124; 46 slots 1,165 and
// 1,160; 48 and 56 the same within 0.2 %; 64 slots 1,587 and 1,558.  f32, 8, 12 and 15 slots 460 and 504, 657 and 687, 817 and 819; 16, 20 and 32 slots 852 and 844, 1,067 and
// 1,045, 1,655 and 1,599.  So the lines: 19.5 bf16 units a block (44 slots of 64 heads are 19.0, 46 are 19.9) and 6.75 f32 ones (15 are 6.5, 16 are 6.9).
// (An instance of the kernel to itself: the choice inside cost 16 slots 1 %.)
template <typename S>
bool late_release(long long units, long long sms) { return 4 * units > sms * (sizeof(S) == 4 ? 27 : 78); }

template <typename S, int MODE, bool ONE_UNIT = false, bool LATE = false>
int launch(const Params& p, cudaStream_t stream) {
    using L = Smem<S, MODE>;
    const long long sms = sm_count();
    if constexpr (MODE == kLayer && !ONE_UNIT) {
        if (p.units <= sms) return launch<S, MODE, true>(p, stream);
    }
    if constexpr (MODE == kCore && !LATE) {
        if (late_release<S>(p.units, sms)) return launch<S, MODE, false, true>(p, stream);
    }
    static bool configured = false;  // per process; the attribute is per device, so set it on every device change
    static int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured || configured_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(recurrent_kernel<S, MODE, ONE_UNIT, LATE>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes);
        if (e != cudaSuccess) return (int)e;
        configured = true;
        configured_dev = dev;
    }
    const unsigned grid = (unsigned)(p.units < sms ? p.units : sms);
    Params q = p;
    q.neg_zero2 = 0x8000000080000000ull;
    q.wait_limit_ns = g_wait_limit_ns;
    q.skip_first_state = g_skip_first_state;
    g_skip_first_state = 0;
    // Launched with programmatic stream serialization: the kernel itself waits for its predecessors before its first
    // global access, so ordering is what a plain launch gives.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreadsOf<S, MODE, ONE_UNIT>);
    cfg.dynamicSmemBytes = L::kBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = early_attribute(attr[0]);
    return (int)cudaLaunchKernelEx(&cfg, recurrent_kernel<S, MODE, ONE_UNIT, LATE>, q);
}

template <int MODE>
int launch_typed(const Params& p, bool bf16_state, cudaStream_t stream) {
    return bf16_state ? launch<__nv_bfloat16, MODE>(p, stream) : launch<float, MODE>(p, stream);
}

bool saves_ok(const void* k, const void* v, const void* g, const void* b) {
    const int n = (k != nullptr) + (v != nullptr) + (g != nullptr) + (b != nullptr);
    return n == 0 || n == 4;
}

// Reference kda.cu:290-299, 310-312, 329-332.
int chain_entry(int32_t heads, int32_t batch, bool batched, const int32_t* cu_rows, const int32_t* keep, int32_t rows, const glm53f_bf16* p,
                int64_t p_stride, int64_t b_off, const glm53f_bf16* a, int64_t a_stride, const glm53f_bf16* g,
                int64_t g_stride, const glm53f_bf16* conv, const int64_t* conv_off, const glm53f_bf16* conv_w,
                const void* state_in, void* state_out, const int64_t* state_off, bool bf16_state, const float* a_log,
                const float* dt_bias, const glm53f_bf16* norm_w, float eps, float lower, glm53f_bf16* out,
                int64_t out_stride, float* k_save, glm53f_bf16* v_save, float* g_save, float* b_save,
                glm53f_stream_t stream) {
    if (heads < 1 || heads > 65535) return kInvalid;
    if (!p || !a || !g || !conv || !conv_w || !state_in || !a_log || !dt_bias || !norm_w || !out) return kInvalid;
    if (!saves_ok(k_save, v_save, g_save, b_save)) return kInvalid;
    if (batched) {
        if (batch < 1 || batch > 65535 || !cu_rows || !conv_off || !state_off) return kInvalid;
    } else if (rows < 1) {
        return kInvalid;
    }
    if (batched && bf16_state && state_out == nullptr && k_save != nullptr && keep == nullptr && g_layer_verify_mode.load() == 1) {
        // The chunked form of a verify call: eligible when every row the two kernels touch by vector is aligned and the outputs,
        // which hold q between them, do not go over the gate rows; any other call runs the exact form below.
        auto al = [](const void* x, int bytes) { return (reinterpret_cast<uintptr_t>(x) & (bytes - 1)) == 0; };
        if (al(p, 8) && al(a, 8) && al(g, 8) && al(conv, 8) && al(conv_w, 16) && al(dt_bias, 16) && al(out, 16) && al(k_save, 16) && al(v_save, 16) &&
            al(g_save, 16) && al(state_in, 16) && (out != g || out_stride != g_stride) && p_stride % 4 == 0 && a_stride % 4 == 0 && g_stride % 4 == 0 && out_stride % 8 == 0) {
            cudaStream_t st = (cudaStream_t)stream;
            const int rc = verify_prologue_launch(heads, batch, cu_rows, p, p_stride, b_off, a, a_stride, conv, conv_off, conv_w, a_log, dt_bias,
                                                  lower, out, out_stride, k_save, v_save, g_save, b_save, st);
            if (rc != 0) return rc;
            return layer_verify_tc_launch(heads, batch, cu_rows, state_in, state_off, g, g_stride, norm_w, eps, out, out_stride, k_save, v_save,
                                          g_save, b_save, st);
        }
    }
    Params q{};
    q.H = heads;
    q.layers = 1;
    q.units = (long long)heads * batch;
    q.cu_rows = cu_rows;
    q.keep = keep;
    q.rows1 = rows;
    q.P = p; q.p_stride = p_stride; q.b_off = b_off;
    q.A = a; q.a_stride = a_stride;
    q.G = g; q.g_stride = g_stride;
    q.conv = conv; q.conv_off = reinterpret_cast<const long long*>(conv_off); q.cw = conv_w;
    q.a_log = a_log; q.dt_bias = dt_bias; q.norm_w = norm_w; q.eps = eps; q.lower = lower;
    q.state_in = state_in; q.state_out = state_out; q.state_stride = 0;
    q.state_off = reinterpret_cast<const long long*>(state_off);
    q.out = out; q.out_stride = out_stride;
    q.k_save = k_save; q.v_save = v_save; q.g_save = g_save; q.b_save = b_save;
    return launch_typed<kLayer>(q, bf16_state, (cudaStream_t)stream);
}

// Reference kda.cu:381-383, 412, 424.
int replay_entry(int32_t heads, int32_t layers, int32_t batch, bool batched, const int32_t* cu_rows, const int32_t* keep,
                 int32_t rows, const void* state_in, void* state_out, int64_t state_stride, const int64_t* state_off,
                 bool bf16_state, const float* k_save, const glm53f_bf16* v_save, const float* g_save,
                 const float* b_save, int64_t kv_stride, int64_t b_stride, glm53f_stream_t stream) {
    if (batched && (!cu_rows || !keep || !state_off)) return kInvalid;
    if (heads < 1 || layers < 1 || batch < 1 || batch > 65535 || (long long)heads * layers > 0x7fffffffLL || !state_in ||
        !state_out || !k_save || !v_save || !g_save || !b_save || rows < 0)
        return kInvalid;
    Params q{};
    q.H = heads;
    q.layers = layers;
    q.units = (long long)heads * layers * batch;
    q.cu_rows = cu_rows;
    q.keep = keep;
    q.rows1 = rows;
    q.state_in = state_in; q.state_out = state_out; q.state_stride = state_stride;
    q.state_off = reinterpret_cast<const long long*>(state_off);
    q.k_save = const_cast<float*>(k_save); q.v_save = const_cast<glm53f_bf16*>(v_save);
    q.g_save = const_cast<float*>(g_save); q.b_save = const_cast<float*>(b_save);
    q.kv_stride = kv_stride; q.b_stride = b_stride;
    if (bf16_state && g_commit_mode.load() == 1)
        return commit_tc_launch(heads, layers, batch, cu_rows, keep, rows, state_in, state_out, state_stride, state_off, k_save, v_save, g_save,
                                b_save, kv_stride, b_stride, (cudaStream_t)stream);
    // The small-block kernel takes k and decays on 16 bytes and grids that fit; GLM53F_KDA_REPLAY=pipeline keeps the
    // persistent kernel.
    static const bool small = [] {
        const char* e = getenv("GLM53F_KDA_REPLAY");
        return !(e != nullptr && strcmp(e, "pipeline") == 0);
    }();
    auto al16 = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
    if (small && al16(k_save) && al16(g_save) && kv_stride % 4 == 0 && q.units * kSmallParts <= 0x7fffffffLL)
        return bf16_state ? launch_replay_small<__nv_bfloat16>(q, (cudaStream_t)stream) : launch_replay_small<float>(q, (cudaStream_t)stream);
    return launch_typed<kReplay>(q, bf16_state, (cudaStream_t)stream);
}

int core_entry(int32_t heads, int32_t batch, const int32_t* cu_rows, const glm53f_bf16* q, const glm53f_bf16* k,
               const glm53f_bf16* v, const float* g, const float* beta, const void* state_in, void* state_out,
               const int64_t* state_off, int32_t state_bf16, int32_t flags, const glm53f_bf16* gate,
               const glm53f_bf16* norm_w, float eps, glm53f_bf16* out, float* k_save, glm53f_bf16* v_save,
               float* g_save, float* b_save, glm53f_stream_t stream) {
    if (heads < 1 || heads > 65535 || batch < 1 || batch > 65535) return kInvalid;
    if (!cu_rows || !q || !k || !v || !g || !beta || !state_in || !state_off || !out) return kInvalid;
    if (gate && !norm_w) return kInvalid;
    if (flags & ~(GLM53F_KDA_CORE_L2NORM | GLM53F_KDA_CORE_TENSOR)) return kInvalid;
    if (!saves_ok(k_save, v_save, g_save, b_save)) return kInvalid;
    if (flags & GLM53F_KDA_CORE_TENSOR) {
        // The chunked verify takes read-only bf16 states, inputs as given (no fused norms) and aligned rows; any other
        // call runs the exact form, whose results are always valid.
        auto al = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
        if (state_bf16 != 0 && state_out == nullptr && gate == nullptr && !(flags & GLM53F_KDA_CORE_L2NORM) && al(q) && al(k) && al(v) && al(g))
            return core_verify_tc_launch(heads, batch, cu_rows, q, k, v, g, beta, state_in, state_off, out, k_save, v_save, g_save, b_save,
                                         (cudaStream_t)stream);
        flags &= ~GLM53F_KDA_CORE_TENSOR;
    }
    Params x{};
    x.H = heads;
    x.layers = 1;
    x.units = (long long)heads * batch;
    x.cu_rows = cu_rows;
    x.q = q; x.k = k; x.v = v; x.glog = g; x.beta = beta; x.flags = flags;
    x.G = gate; x.norm_w = norm_w; x.eps = eps;
    x.state_in = state_in; x.state_out = state_out;
    x.state_off = reinterpret_cast<const long long*>(state_off);
    x.out = out; x.out_stride = (long long)heads * DV;
    x.k_save = k_save; x.v_save = v_save; x.g_save = g_save; x.b_save = b_save;
    // The exact verify (saves requested, inputs used as given, no fused output norm) runs on the small-block kernel: two
    // units' serial rows at once wait less on their own latencies than the persistent kernel's one (48 slots x 16 rows x 34 layers, bf16,
    // 9.6 against 11.9 ms; 6 slots x 8 rows 841 against 990 us, f32 757 and 901; a single slot's windows are the exception, four rows
    // 335 against 254).  Decode stays on the persistent kernel, which keeps more bytes in flight (bf16, 16 slots 458 against 635 us, 48
    // slots 1,208 and 1,704; f32 single rows 845 and 786, 2,335 and 2,117, but windows of two rows 880 and 924), except with more than
    // one and at most two units an SM: some of its blocks have two then, one after the other, and the rest wait (single rows of 160,
    // 192, 256 and 288 units, f32 285 -> 244 us for 34 launches, 301 -> 256, 319 -> 280, 325 -> 292, bf16 221 -> 195, 230 -> 201, 238 -> 210, 240 -> 215; windows
    // of two to six rows 3 to 15 % less, of 16, 64 and 1,000 rows 9 to 19 %, one request of 40 rows among single ones 1 to 10 %; rows
    // of four and one in turn 160 units up to 10 % more, 288 7 to 17 % less, half of the requests empty 1 to 5 % more where states are
    // written; single rows of 320 units 372 -> 311 and 275 -> 287).  GLM53F_KDA_DECODE=pipeline / small forces one
    // or the other; the bits are the same either way.
    static const int forced = [] {
        const char* e = getenv("GLM53F_KDA_DECODE");
        return e == nullptr ? 0 : (strcmp(e, "pipeline") == 0 ? 1 : (strcmp(e, "small") == 0 ? 2 : 0));
    }();
    const long long sms = sm_count();
    // A unit's two small blocks read all of a row's q and k each, and for the saves one of them all of v, and neither waits for the other before
    // it stores its half of the outputs: outputs over these rows stay on the persistent kernel, where one block has the unit.  Outputs
    // over other rows' inputs meet other units' on any kernel, except those of a single request over its earlier rows.
    const bool over_inputs = out == q || out == k || (k_save != nullptr && out == v);
    const bool two_units = x.units > sms && x.units <= 2 * sms && batch > 1;
    const bool small = !over_inputs && (forced == 2 || (forced == 0 && (k_save != nullptr || two_units)));
    if (small && flags == 0 && gate == nullptr && x.units * kSmallParts <= 0x7fffffffll)
        return state_bf16 != 0 ? launch_small<__nv_bfloat16>(x, (cudaStream_t)stream) : launch_small<float>(x, (cudaStream_t)stream);
    return launch_typed<kCore>(x, state_bf16 != 0, (cudaStream_t)stream);
}

}  // namespace

int layer_chain_launch(int32_t heads, int32_t batch, const int32_t* cu_rows, int32_t rows, const glm53f_bf16* p,
                       int64_t p_stride, int64_t b_off, const glm53f_bf16* a, int64_t a_stride, const glm53f_bf16* g,
                       int64_t g_stride, const glm53f_bf16* conv, const int64_t* conv_off, const glm53f_bf16* conv_w,
                       const void* state_in, void* state_out, const int64_t* state_off, bool bf16_state,
                       const float* a_log, const float* dt_bias, const glm53f_bf16* norm_w, float eps, float lower,
                       glm53f_bf16* out, int64_t out_stride, cudaStream_t stream) {
    Params q{};
    q.H = heads;
    q.layers = 1;
    q.units = (long long)heads * batch;
    q.cu_rows = cu_rows;
    q.rows1 = rows;
    q.P = p; q.p_stride = p_stride; q.b_off = b_off;
    q.A = a; q.a_stride = a_stride;
    q.G = g; q.g_stride = g_stride;
    q.conv = conv; q.conv_off = reinterpret_cast<const long long*>(conv_off); q.cw = conv_w;
    q.a_log = a_log; q.dt_bias = dt_bias; q.norm_w = norm_w; q.eps = eps; q.lower = lower;
    q.state_in = state_in; q.state_out = state_out;
    q.state_off = reinterpret_cast<const long long*>(state_off);
    q.out = out; q.out_stride = out_stride;
    return launch_typed<kLayer>(q, bf16_state, stream);
}

int core_chain_launch(int32_t heads, int32_t batch, const int32_t* cu_rows, const glm53f_bf16* q, const glm53f_bf16* k,
                      const glm53f_bf16* v, const float* g, const float* beta, const void* state_in, void* state_out,
                      const int64_t* state_off, bool bf16_state, int32_t flags, const glm53f_bf16* gate,
                      const glm53f_bf16* norm_w, float eps, glm53f_bf16* out, cudaStream_t stream) {
    return core_entry(heads, batch, cu_rows, q, k, v, g, beta, state_in, state_out, state_off, bf16_state ? 1 : 0, flags, gate,
                      norm_w, eps, out, nullptr, nullptr, nullptr, nullptr, (glm53f_stream_t)stream);
}

}  // namespace kda

using namespace kda;

extern "C" int glm53f_kda_chain(int32_t heads, int32_t rows, const glm53f_bf16* p, int64_t p_stride, int64_t b_off,
                                const glm53f_bf16* a, int64_t a_stride, const glm53f_bf16* g, int64_t g_stride,
                                const glm53f_bf16* conv, const glm53f_bf16* conv_w, const float* state_in,
                                float* state_out, const float* a_log, const float* dt_bias, const glm53f_bf16* norm_w,
                                float eps, float lower, glm53f_bf16* out, int64_t out_stride, float* k_save,
                                glm53f_bf16* v_save, float* g_save, float* b_save, glm53f_stream_t stream) {
    return chain_entry(heads, 1, false, nullptr, nullptr, rows, p, p_stride, b_off, a, a_stride, g, g_stride, conv, nullptr, conv_w,
                       state_in, state_out, nullptr, false, a_log, dt_bias, norm_w, eps, lower, out, out_stride, k_save,
                       v_save, g_save, b_save, stream);
}

extern "C" int glm53f_kda_chain_batch(int32_t heads, int32_t batch, const int32_t* cu_rows, const glm53f_bf16* p,
                                      int64_t p_stride, int64_t b_off, const glm53f_bf16* a, int64_t a_stride,
                                      const glm53f_bf16* g, int64_t g_stride, const glm53f_bf16* conv,
                                      const int64_t* conv_off, const glm53f_bf16* conv_w, const float* state_in,
                                      float* state_out, const int64_t* state_off, const float* a_log,
                                      const float* dt_bias, const glm53f_bf16* norm_w, float eps, float lower,
                                      glm53f_bf16* out, int64_t out_stride, float* k_save, glm53f_bf16* v_save,
                                      float* g_save, float* b_save, glm53f_stream_t stream) {
    return chain_entry(heads, batch, true, cu_rows, nullptr, 0, p, p_stride, b_off, a, a_stride, g, g_stride, conv, conv_off,
                       conv_w, state_in, state_out, state_off, false, a_log, dt_bias, norm_w, eps, lower, out,
                       out_stride, k_save, v_save, g_save, b_save, stream);
}

extern "C" int glm53f_kda_chain_batch_bf16state(int32_t heads, int32_t batch, const int32_t* cu_rows,
                                                const glm53f_bf16* p, int64_t p_stride, int64_t b_off,
                                                const glm53f_bf16* a, int64_t a_stride, const glm53f_bf16* g,
                                                int64_t g_stride, const glm53f_bf16* conv, const int64_t* conv_off,
                                                const glm53f_bf16* conv_w, const glm53f_bf16* state_in,
                                                glm53f_bf16* state_out, const int64_t* state_off, const float* a_log,
                                                const float* dt_bias, const glm53f_bf16* norm_w, float eps,
                                                float lower, glm53f_bf16* out, int64_t out_stride, float* k_save,
                                                glm53f_bf16* v_save, float* g_save, float* b_save,
                                                glm53f_stream_t stream) {
    return chain_entry(heads, batch, true, cu_rows, nullptr, 0, p, p_stride, b_off, a, a_stride, g, g_stride, conv, conv_off,
                       conv_w, state_in, state_out, state_off, true, a_log, dt_bias, norm_w, eps, lower, out, out_stride,
                       k_save, v_save, g_save, b_save, stream);
}

extern "C" int glm53f_kda_chain_commit_batch(int32_t heads, int32_t batch, const int32_t* cu_rows, const int32_t* keep,
                                             const glm53f_bf16* p, int64_t p_stride, int64_t b_off, const glm53f_bf16* a,
                                             int64_t a_stride, const glm53f_bf16* g, int64_t g_stride, const glm53f_bf16* conv,
                                             const int64_t* conv_off, const glm53f_bf16* conv_w, void* state,
                                             const int64_t* state_off, int32_t state_bf16, const float* a_log,
                                             const float* dt_bias, const glm53f_bf16* norm_w, float eps, float lower,
                                             glm53f_bf16* out, int64_t out_stride, glm53f_stream_t stream) {
    if (!keep || !state) return kInvalid;
    return chain_entry(heads, batch, true, cu_rows, keep, 0, p, p_stride, b_off, a, a_stride, g, g_stride, conv, conv_off, conv_w,
                       state, state, state_off, state_bf16 != 0, a_log, dt_bias, norm_w, eps, lower, out, out_stride, nullptr,
                       nullptr, nullptr, nullptr, stream);
}

extern "C" int glm53f_kda_replay(int32_t heads, int32_t rows, const float* state_in, float* state_out,
                                 const float* k_save, const glm53f_bf16* v_save, const float* g_save,
                                 const float* b_save, glm53f_stream_t stream) {
    return replay_entry(heads, 1, 1, false, nullptr, nullptr, rows, state_in, state_out, 0, nullptr, false, k_save,
                        v_save, g_save, b_save, 0, 0, stream);
}

extern "C" int glm53f_kda_replay_layers(int32_t heads, int32_t layers, int32_t rows, const float* state_in,
                                        float* state_out, int64_t state_stride, const float* k_save,
                                        const glm53f_bf16* v_save, const float* g_save, const float* b_save,
                                        int64_t kv_stride, int64_t b_stride, glm53f_stream_t stream) {
    return replay_entry(heads, layers, 1, false, nullptr, nullptr, rows, state_in, state_out, state_stride, nullptr,
                        false, k_save, v_save, g_save, b_save, kv_stride, b_stride, stream);
}

extern "C" int glm53f_kda_replay_batch(int32_t heads, int32_t layers, int32_t batch, const int32_t* cu_rows,
                                       const int32_t* keep, const float* state_in, float* state_out,
                                       int64_t state_stride, const int64_t* state_off, const float* k_save,
                                       const glm53f_bf16* v_save, const float* g_save, const float* b_save,
                                       int64_t kv_stride, int64_t b_stride, glm53f_stream_t stream) {
    return replay_entry(heads, layers, batch, true, cu_rows, keep, 0, state_in, state_out, state_stride, state_off, false,
                        k_save, v_save, g_save, b_save, kv_stride, b_stride, stream);
}

extern "C" int glm53f_kda_replay_batch_bf16state(int32_t heads, int32_t layers, int32_t batch, const int32_t* cu_rows,
                                                 const int32_t* keep, const glm53f_bf16* state_in,
                                                 glm53f_bf16* state_out, int64_t state_stride,
                                                 const int64_t* state_off, const float* k_save,
                                                 const glm53f_bf16* v_save, const float* g_save, const float* b_save,
                                                 int64_t kv_stride, int64_t b_stride, glm53f_stream_t stream) {
    return replay_entry(heads, layers, batch, true, cu_rows, keep, 0, state_in, state_out, state_stride, state_off, true,
                        k_save, v_save, g_save, b_save, kv_stride, b_stride, stream);
}

extern "C" int glm53f_kda_core_decode_batch(int32_t heads, int32_t batch, const int32_t* cu_rows, const glm53f_bf16* q,
                                            const glm53f_bf16* k, const glm53f_bf16* v, const float* g,
                                            const float* beta, const void* state_in, void* state_out,
                                            const int64_t* state_off, int32_t state_bf16, int32_t flags,
                                            const glm53f_bf16* gate, const glm53f_bf16* norm_w, float eps,
                                            glm53f_bf16* out, glm53f_stream_t stream) {
    return core_entry(heads, batch, cu_rows, q, k, v, g, beta, state_in, state_out, state_off, state_bf16, flags, gate,
                      norm_w, eps, out, nullptr, nullptr, nullptr, nullptr, stream);
}

extern "C" int glm53f_kda_core_verify_batch(int32_t heads, int32_t batch, const int32_t* cu_rows, const glm53f_bf16* q,
                                            const glm53f_bf16* k, const glm53f_bf16* v, const float* g,
                                            const float* beta, const void* state_in, void* state_out,
                                            const int64_t* state_off, int32_t state_bf16, int32_t flags,
                                            const glm53f_bf16* gate, const glm53f_bf16* norm_w, float eps,
                                            glm53f_bf16* out, float* k_save, glm53f_bf16* v_save, float* g_save,
                                            float* b_save, glm53f_stream_t stream) {
    return core_entry(heads, batch, cu_rows, q, k, v, g, beta, state_in, state_out, state_off, state_bf16, flags, gate,
                      norm_w, eps, out, k_save, v_save, g_save, b_save, stream);
}

extern "C" int glm53f_kda_core_commit_batch(int32_t heads, int32_t layers, int32_t batch, const int32_t* cu_rows,
                                            const int32_t* keep, const void* state_in, void* state_out,
                                            int64_t state_stride, const int64_t* state_off, int32_t state_bf16,
                                            const float* k_save, const glm53f_bf16* v_save, const float* g_save,
                                            const float* b_save, int64_t kv_stride, int64_t b_stride,
                                            glm53f_stream_t stream) {
    return replay_entry(heads, layers, batch, true, cu_rows, keep, 0, state_in, state_out, state_stride, state_off,
                        state_bf16 != 0, k_save, v_save, g_save, b_save, kv_stride, b_stride, stream);
}

int* kda::status_word() {
    int* p = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_status) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

extern "C" int glm53f_kda_device_status(void) {
    int v = 0, zero = 0;
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return (int)e;
    e = cudaMemcpyFromSymbol(&v, g_status, sizeof v);
    if (e != cudaSuccess) return (int)e;
    if (v != 0) cudaMemcpyToSymbol(g_status, &zero, sizeof zero);
    return v;
}

extern "C" int32_t glm53f_kda_verify_mode(int32_t mode) {
    const int prev = kda::g_layer_verify_mode.load();
    if (mode == 0 || mode == 1) kda::g_layer_verify_mode.store(mode);
    return prev;
}

extern "C" int32_t glm53f_kda_commit_mode(int32_t mode) {
    const int prev = kda::g_commit_mode.load();
    if (mode == 0 || mode == 1) kda::g_commit_mode.store(mode);
    return prev;
}

extern "C" int glm53f_kda_debug_wait_test(uint64_t wait_limit_ns, int32_t skip_first_state) {
    if (wait_limit_ns != 0 && (wait_limit_ns < 100000ull || wait_limit_ns > 60000000000ull)) return kda::kInvalid;  // 0.1 ms .. 60 s
    kda::g_wait_limit_ns = wait_limit_ns == 0 ? kda::kWaitLimitNs : wait_limit_ns;
    kda::g_skip_first_state = skip_first_state != 0 ? 1 : 0;
    return 0;
}
