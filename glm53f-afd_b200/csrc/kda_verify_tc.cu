// Draft verification on the tensor cores: a verify window of up to 16 rows is one 16-row chunk.
//
// The exact verify (kda_chain.cu) walks a window's rows one after the other through the delta rule, each row a full
// pass over the 128 x 128 state in registers: 16 serial passes, bound by instruction issue.  The chunked form reads the
// state once and does the state-sized work as two small tensor-core products.  For the rows i = 0..15 of a window,
// with G the cumulative log decay, Gm = G_8 (the middle row: every decay factor formed below stays within e^+-47 for
// the model's gate bound of -5.8 per row) and S the window's incoming state [v][k]:
//
//   L = beta_i (k_i a_i).(k_j / a_j) for j < i,  M = (q_i a_i).(k_j / a_j) for j <= i,   a = exp(G - Gm)
//                         as L^T | M^T = Kc x [Kgb | Qgb]^T (tcgen05, M = 64 of which 16 rows are real, N = 32)
//   W = (I + L)^-1 diag(beta) Kg,  U = (I + L)^-1 diag(beta) V   forward substitution down the 16 rows, FP32 on the CUDA
//                         cores (thread = channel: 136 multiply-adds each; no explicit inverse), Kg = k exp(G)
//   (W S)^T | (Qg S)^T    = S x [W | Qg]^T: tcgen05, M = 128 value channels, N = 2 x 16 rows, K = 128 key channels; the
//                         bf16 state tile is the A operand exactly as it lies in HBM (rows of 128 key channels)
//   D = U - W S,  O = Qg S + M D   FP32, thread = value channel (its tensor-memory lane)
//
// The state is not written (a verify leaves it to the commit) and the replay saves are the exact path's, bit for bit
// (k widened, v copied, exp(g) by the same expf, beta copied), so verify + commit still leaves the states of serial
// decode steps; only the window's OUTPUTS differ from the serial steps', by the rounding of bf16 operands (within the
// task's tolerance: max-abs 2e-2, rel-L2 5e-3).  Selected by GLM53F_KDA_CORE_TENSOR on glm53f_kda_core_verify_batch.
//
// The layer form (LAYER = true; the chunked form of glm53f_kda_chain_batch_bf16state, glm53f_kda_verify_mode) runs after
// the verify prologue (kda_prologue.cu) and takes a unit's rows from where that kernel left them: k, v, the decay
// multiplier and beta from the replay saves, q as fp16 from the output rows; it writes no saves and fuses the gated
// RMSNorm into its outputs.
//
// One block of 128 threads per (request, head) unit, three blocks per SM, blocks walk the units persistently.  A unit's
// rows arrive by asynchronous 16-byte copies, its state by two tensor copies straight into the 128-byte swizzle the tensor core
// reads, all issued one unit ahead, so one unit's arithmetic covers the next one's loads.  All waits are bounded.
//
// A unit's serial stages bound it, at twelve warps an SM.  What they took and take, cycles of a unit of the core form (48 requests of 8 to
// 16 rows): operand tiles 4,400 with two exponentials and a division an element and the saves between them, 1,800 as products of
// multipliers; the saves 1,300, beside the first products; the next rows' copies 1,800 with a load of beta to wait for, 570 without;
// products 870 + 880 as eight of N = 32 each instead of sixteen of N = 16; outputs 3,000 as two-byte stores, now sixteen bytes a unit
// later.  Verify and commit of 34 layers together, the same buffers in every call: 3,806 -> 3,183 us, 20 requests of 4 to 8 rows 1,625 -> 1,371;
// with the state in boxes, in both kernels and both ways, instead of 2,048 pieces that pass through the threads, 2,870 to 2,920 and 1,230 to 1,240
// (the commit's way out alone was 2,000 cycles of a unit's 14,000).  With buffers that change from call to call 48 requests take
// 3,065 to 3,120 us, before all of it 3,800.

#include <cuda_fp16.h>

#include "common.cuh"
#include "glm53f_kda.h"
#include "kda_internal.h"
#include "tc.cuh"
#include "tensor_map.cuh"

namespace kda {
namespace {

constexpr int WIN = 16, kVThreads = 128;
// Shared memory map (bytes).  Tiles are boxes of R rows x 128 bytes in the 128-byte swizzle (16-byte piece p of row r at
// piece p ^ (r & 7)), two boxes per tile (channels 0-63, 64-127).  The column-side tile Kc comes first: as the M = 128
// operand of L^T and M^T (M = 64) its descriptor walks 64 rows although 16 are real, and what follows it is the state tile.
// Once those two products are done Kc is dead, and L and M (FP32, 3 KB) take its place until the unit ends.
constexpr int vKc = 0, vS = 4096, vRow = vS + 32768, vRaw = vRow + 8192;
constexpr int kRowR = 2 * WIN;   // the row side: one tile of 32 rows, Kgb | Qgb and, once L^T and M^T are formed, W | Qg
constexpr int vStage = vRow;     // layer form: FP32 outputs [16][128] over W | Qg
constexpr int vL = vKc, vM = vL + WIN * WIN * 8;  // L twice in a row (see substitute), M transposed
static_assert(vM + WIN * WIN * 4 <= vS, "L and M fit the dead column-side tile");
// Raw rows of a unit.  Core form: q, k, v bf16 (256 bytes a row), log decay f32 (512), beta.  Layer form: q fp16, v bf16,
// k f32, the decay multiplier f32, beta.
template <bool LAYER>
struct Raw {
    static constexpr int Q = 0, V = 4096, K = 8192, G = LAYER ? 16384 : 12288, B = G + 8192, kBytes = B + 128;
};
template <bool LAYER>
struct Map {
    static constexpr int vOut = vRaw + Raw<LAYER>::kBytes;  // core form: a unit's outputs, bf16 [16][128], on their way out
    static constexpr int vBeta = vOut + (LAYER ? 0 : WIN * DV * 2), vBar = vBeta + 64 /* products, state */, vCtl = vBar + 16, kSmem = vCtl + 16;
    static_assert(vBar % 8 == 0 && kSmem <= 75 * 1024, "three blocks per SM");
};
constexpr uint32_t kVCols = 32;  // tensor memory: [0, 16) L^T then (W S)^T, [16, 32) M^T then (Qg S)^T

// A state buffer as rows of 128 elements in two halves, for copies of a unit's [128][128] that come in, and go out, in the tile's own
// swizzle: two boxes instead of 2,048 pieces, and nothing of them passes through the threads.  For buffers on 16 bytes and units at a
// multiple of a row; the others go piece by piece.
bool state_map(CUtensorMap* tm, const void* base) {
    EncodeTiled enc = encode_tiled();
    if (enc == nullptr || (reinterpret_cast<uintptr_t>(base) & 15) != 0) return false;
    const cuuint64_t dims[3] = {64u, 2u, 0x7fffffffu}, strides[2] = {128u, 256u};
    const cuuint32_t box[3] = {64u, 1u, (cuuint32_t)DV}, step[3] = {1u, 1u, 1u};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
__device__ __forceinline__ bool in_boxes(int mapped, long long s_elem) { return mapped && (s_elem & (DK - 1)) == 0 && s_elem >= 0 && s_elem <= (0x7fffffffll - DV) * DK; }
__device__ __forceinline__ void load_boxes(unsigned char* tile, const CUtensorMap* tm, long long s_elem, uint64_t* bar) {
    mbar_arrive_expect_tx(bar, DV * DK * 2);
    for (int x = 0; x < 2; ++x) tensor_load_3d(tile + x * 16384, tm, 0, x, (int)(s_elem / DK), bar);
}

// After an abort a unit's boxes may still be on their way into this block's shared memory: a bounded time for them.
__device__ __forceinline__ void abort_pause(volatile uint32_t* ctl) {
    if (ctl[1] == 0u) return;
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 2000000ull) {
    }
}

struct VParams {
    alignas(64) CUtensorMap tm_state;
    int mapped;
    int H;
    long long units;
    const int32_t* cu;
    const uint16_t *q, *k, *v;  // core form: bf16 rows
    const float* g;
    const float* beta;
    const uint16_t* state;
    const long long* state_off;
    uint16_t* out;              // layer form: holds q as fp16 on entry
    long long out_stride;
    float* k_save;              // layer form: the sources of k, v, decay and beta
    uint16_t* v_save;
    float* g_save;
    float* b_save;
    const uint16_t* gate;       // layer form: the output gate rows, the norm weight, eps
    long long gate_stride;
    const uint16_t* norm_w;
    float eps;
    int* status;
};

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gmem_src) : "memory");
}
// Zeros where !read (nothing is read then).
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src, bool read) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem_dst)), "l"(gmem_src), "r"(read ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src, bool read) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(smem_dst)), "l"(gmem_src), "r"(read ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Byte offset in a tile with R rows per box of the bf16 element (row r, channel c).
__device__ __forceinline__ int sw_elem(int R, int r, int c) {
    return (c >> 6) * R * 128 + r * 128 + (((((c & 63) >> 3) ^ (r & 7))) << 4) + (c & 7) * 2;
}
// The output gate: these outputs carry the rounding of bf16 operands already, so the hardware's approximate exponential
// and division do (the file's other divisions and exponentials keep IEEE arithmetic for the replay saves).
__device__ __forceinline__ float sigmoid_(float x) { return rcp_approx(1.0f + ex2_ftz(-kLog2e * x)); }

// The operand tiles are made two channels and eight rows a thread, outwards from the chunk's middle: lanes 0-15 have rows 7, 6, .. 0, lanes
// 16-31 rows 8, 9, .. 15.  Four-byte shared-memory accesses, packed conversions.  What a lane of the other half holds:
__device__ __forceinline__ float2 other_half(float2 x) {
    return make_float2(__shfl_xor_sync(0xffffffffu, x.x, 16), __shfl_xor_sync(0xffffffffu, x.y, 16));
}
__device__ __forceinline__ float2 widen_bf16x2(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ int row_of(int s, bool upper) { return upper ? WIN / 2 + s : WIN / 2 - 1 - s; }

// The decay factors of a thread's rows from their multipliers m[s] (the exponentials of the log decays): products of at most sixteen of
// them, no logarithms and no exponentials of sums.  Relative to the middle row (8), a row's factor is the product of the multipliers
// between, on the lower half its reciprocal.
struct Factors {
    float2 between[WIN / 2], out[WIN / 2];  // products of the rows from the middle up to a row, without the further end; from a row outwards
    float2 to_middle, beyond, all;
    bool upper;
    __device__ __forceinline__ Factors(const float2 (&m)[WIN / 2], bool up) : upper(up) {
        between[0] = {1.0f, 1.0f};
        out[WIN / 2 - 1] = m[WIN / 2 - 1];
#pragma unroll
        for (int s = 1; s < WIN / 2; ++s) between[s] = mul2(between[s - 1], {up ? m[s].x : m[s - 1].x, up ? m[s].y : m[s - 1].y});
#pragma unroll
        for (int s = WIN / 2 - 2; s >= 0; --s) out[s] = mul2(out[s + 1], m[s]);
        const float2 m8 = other_half(m[0]), rest = other_half(out[0]), x = mul2(rest, m[0]);
        to_middle = {up ? 1.0f : m8.x, up ? 1.0f : m8.y};
        beyond = {up ? x.x : rest.x, up ? x.y : rest.y};
        all = mul2(rest, out[0]);
    }
    // a = exp(G - G_8) and its reciprocal.  The smaller of the two stops at 2^-126, so that the other is finite (NaN stays NaN).
    __device__ __forceinline__ void relative(int s, float2& a, float2& inva) const {
        const float2 p = mul2(to_middle, between[s]), r = {rcp_approx(max_nan(p.x, 0x1p-126f)), rcp_approx(max_nan(p.y, 0x1p-126f))};
        a = {upper ? p.x : r.x, upper ? p.y : r.y};
        inva = {upper ? r.x : p.x, upper ? r.y : p.y};
    }
    // Whether the last rows' factors have stopped there: more decay than the products can be split for.
    __device__ __forceinline__ bool lost() const { return upper && (between[WIN / 2 - 1].x < 0x1p-126f || between[WIN / 2 - 1].y < 0x1p-126f); }
    __device__ __forceinline__ float2 from_start(int s) const {  // exp(G)
        const float2 x = mul2(beyond, between[s]);
        return {upper ? x.x : out[s].x, upper ? x.y : out[s].y};
    }
    __device__ __forceinline__ float2 to_end(int s) const {  // exp(G_last - G)
        const float2 x = mul2(beyond, between[s]), o = s + 1 < WIN / 2 ? out[s + 1] : float2{1.0f, 1.0f};
        return {upper ? o.x : x.x, upper ? o.y : x.y};
    }
};
// All 16 rows of one channel (c0 + upper) from the two halves' pairs of channels.
__device__ __forceinline__ void all_rows(const float2 (&x)[WIN / 2], bool upper, float (&y)[WIN]) {
#pragma unroll
    for (int s = 0; s < WIN / 2; ++s) {
        const float got = __shfl_xor_sync(0xffffffffu, upper ? x[s].x : x[s].y, 16);
        y[WIN / 2 - 1 - s] = upper ? got : x[s].x;
        y[WIN / 2 + s] = upper ? x[s].y : got;
    }
}

// (W, U) by forward substitution down the 16 rows, two-wide: x[i] = (beta_i kg_i, beta_i v_i) - sum_j L[i][j] x[j].  -L[i][j] lies
// twice in a row at Ln[i * LN + j], so one 16-byte read feeds two of the 136 two-wide multiply-adds.
constexpr int LN = WIN;
__device__ __forceinline__ void substitute(const float2* Ln, const float* betas, const float (&kg)[WIN], const float (&vv)[WIN], float2 (&x)[WIN]) {
#pragma unroll
    for (int i = 0; i < WIN; ++i) {
        const float bi = betas[i];
        float2 x0 = mul2({bi, bi}, {kg[i], vv[i]}), x1 = {0.0f, 0.0f};
#pragma unroll
        for (int j = 0; j < i; j += 2) {
            const float4 l = *reinterpret_cast<const float4*>(Ln + i * LN + j);
            x0 = fma2({l.x, l.y}, x[j], x0);
            if (j + 1 < i) x1 = fma2({l.z, l.w}, x[j + 1], x1);
        }
        x[i] = i > 1 ? fma2(x1, {1.0f, 1.0f}, x0) : x0;
    }
}

struct Unit {
    int b, h, n;
    long long row0, s_elem;
};
// The block's units, u = blockIdx.x, blockIdx.x + gridDim.x, ...  A unit's metadata is read two units ahead and stays as loaded until
// then: arithmetic right after the loads would wait for them behind the stores of a unit's results (1,900 cycles a unit).
struct Units {
    unsigned b, h, step_b, step_h;
    long long left;  // units from the one in the registers on
    int r0, r1;
    long long off;
    __device__ __forceinline__ explicit Units(const VParams& p) {
        const unsigned H = (unsigned)p.H;
        b = blockIdx.x / H;
        h = blockIdx.x % H;
        step_b = gridDim.x / H;
        step_h = gridDim.x % H;
        left = p.units - blockIdx.x;
        r0 = r1 = 0;
        off = 0;
        fetch(p);
    }
    __device__ __forceinline__ void fetch(const VParams& p) {
        if (left <= 0) return;
        r0 = p.cu[b];
        r1 = p.cu[b + 1];
        off = p.state_off[b];
    }
    __device__ __forceinline__ bool take(const VParams& p, Unit& x) {
        if (left <= 0) return false;
        x.b = (int)b;
        x.h = (int)h;
        x.row0 = r0;
        x.n = r1 - r0;
        x.s_elem = off + (long long)h * DV * DK;
        left -= gridDim.x;
        h += step_h;
        b += step_b;
        if (h >= (unsigned)p.H) {
            h -= (unsigned)p.H;
            ++b;
        }
        fetch(p);
        return true;
    }
};

// Offset in the state tile of the 16-byte piece pk of row v.
__device__ __forceinline__ int state_piece(int v, int pk) { return (pk >> 3) * 16384 + v * 128 + (((pk & 7) ^ (v & 7)) << 4); }

// The unit's raw rows; rows past the window's end become zero.
template <bool LAYER>
__device__ __forceinline__ void fetch_rows(const VParams& p, unsigned char* smem, const Unit& un, int t) {
    using R = Raw<LAYER>;
    const int n = min(max(un.n, 0), WIN);
    unsigned char* raw = smem + vRaw;
    const long long rs = (long long)p.H * DK, unit = (un.row0 * p.H + un.h) * DK;
    {  // 16-byte pieces of the 256-byte rows, eight rows a step
        const int r0 = t >> 4, pc = t & 15;
        const long long at = unit + r0 * rs + pc * 8;
        const uint16_t* qs = LAYER ? p.out + (un.row0 + r0) * p.out_stride + (long long)un.h * DK + pc * 8 : p.q + at;
        const uint16_t* vs = (LAYER ? p.v_save : p.v) + at;
        const uint16_t* ks = p.k + at;  // core form
#pragma unroll
        for (int i = 0; i < WIN / 8; ++i) {
            unsigned char* to = raw + (t + i * kVThreads) * 16;
            const bool in = r0 + 8 * i < n;
            cp_async16(to + R::Q, in ? qs + i * 8 * (LAYER ? p.out_stride : rs) : qs, in);
            if constexpr (!LAYER) cp_async16(to + R::K, in ? ks + i * 8 * rs : ks, in);
            cp_async16(to + R::V, in ? vs + i * 8 * rs : vs, in);
        }
    }
    {  // and of the 512-byte rows, four a step
        const int r0 = t >> 5;
        const long long at = unit + r0 * rs + (t & 31) * 4;
        const float *gs = (LAYER ? p.g_save : p.g) + at, *ks = p.k_save + at;
#pragma unroll
        for (int i = 0; i < WIN / 4; ++i) {
            unsigned char* to = raw + (t + i * kVThreads) * 16;
            const bool in = r0 + 4 * i < n;
            cp_async16(to + R::G, in ? gs + i * 4 * rs : gs, in);
            if constexpr (LAYER) cp_async16(to + R::K, in ? ks + i * 4 * rs : ks, in);
        }
    }
    if (t < WIN) {
        const float* src = LAYER ? p.b_save : p.beta;
        cp_async4(raw + R::B + t * 4, t < n ? src + (un.row0 + t) * p.H + un.h : src, t < n);
    }
    cp_async_commit();
}
// The unit's state, 2,048 pieces of 16 bytes, into the swizzled tile.
__device__ __forceinline__ void fetch_state(const VParams& p, unsigned char* smem, const Unit& un, int t, uint64_t* bar_state) {
    const uint16_t* src = p.state + un.s_elem;
    if (in_boxes(p.mapped, un.s_elem)) {
        if (t == 0) load_boxes(smem + vS, &p.tm_state, un.s_elem, bar_state);
    } else if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        unsigned char* to = smem + vS + state_piece(t >> 4, t & 15);  // eight rows a step: the swizzle stays
        src += t * 8;
#pragma unroll
        for (int i = 0; i < 16; ++i) cp_async16(to + i * 1024, src + i * kVThreads * 8);
    } else {  // a state that is not 16-byte aligned: element by element
        for (int e = t; e < DV * DK; e += kVThreads) *reinterpret_cast<uint16_t*>(smem + vS + sw_elem(DV, e >> 7, e & 127)) = src[e];
    }
    cp_async_commit();
}

// The core form's replay saves of a unit's n rows, the exact path's bits: k widened, v, exp(g), which stage A has left in place of g, beta.
__device__ __forceinline__ void save_rows(const VParams& p, const unsigned char* smem, const Unit& un, int n, int t, bool vec) {
    using R = Raw<false>;
    if (p.k_save == nullptr) return;
    const unsigned char* raw = smem + vRaw;
    const long long rs = (long long)p.H * DK, unit = (un.row0 * p.H + un.h) * DK;
    if (t < n) p.b_save[(un.row0 + t) * p.H + un.h] = reinterpret_cast<const float*>(raw + R::B)[t];
    if (vec) {
#pragma unroll
        for (int i = 0; i < WIN / 4; ++i) {  // four channels a thread, four rows a step
            const int r = (t >> 5) + 4 * i, c = (t & 31) * 4;
            if (r < n) {
                const uint2 kw = *reinterpret_cast<const uint2*>(raw + R::K + (r * DK + c) * 2);
                const float2 k0 = widen_bf16x2(kw.x), k1 = widen_bf16x2(kw.y);
                const float4 g4 = *reinterpret_cast<const float4*>(raw + R::G + (r * DK + c) * 4);
                *reinterpret_cast<float4*>(p.k_save + unit + r * rs + c) = make_float4(k0.x, k0.y, k1.x, k1.y);
                *reinterpret_cast<float4*>(p.g_save + unit + r * rs + c) = g4;
            }
        }
#pragma unroll
        for (int i = 0; i < WIN / 8; ++i) {
            const int r = (t >> 4) + 8 * i, c = (t & 15) * 8;
            if (r < n) *reinterpret_cast<uint4*>(p.v_save + unit + r * rs + c) = *reinterpret_cast<const uint4*>(raw + R::V + (r * DK + c) * 2);
        }
    } else {
        for (int r = 0; r < n; ++r) {
            const long long at = unit + r * rs + t;
            p.k_save[at] = bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(raw + R::K)[r * DK + t]);
            p.g_save[at] = reinterpret_cast<const float*>(raw + R::G)[r * DK + t];
            p.v_save[at] = reinterpret_cast<const uint16_t*>(raw + R::V)[r * DK + t];
        }
    }
}

template <bool LAYER>
__global__ void __launch_bounds__(kVThreads, 3) verify_tc_kernel(const __grid_constant__ VParams p) {
    using R = Raw<LAYER>;
    using MP = Map<LAYER>;
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + MP::vBar);
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + MP::vCtl);
    uint32_t* tmem_slot = const_cast<uint32_t*>(ctl) + 2;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 1, 1);
        ctl[0] = 0u;
        ctl[1] = 0u;
        mbar_init_fence();
    }
    if (warp == 0) tc::tmem_alloc(tmem_slot, kVCols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = *tmem_slot;
    grid_ready();
    const WaitCtx ctx{ctl, ctl + 1, p.status};
    uint32_t phase = 0, state_phase = 0;
    float2* Ln = reinterpret_cast<float2*>(smem + vL);
    float* Mf = reinterpret_cast<float*>(smem + vM);
    float* betas = reinterpret_cast<float*>(smem + MP::vBeta);
    float nw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if constexpr (LAYER) {
#pragma unroll
        for (int i = 0; i < 4; ++i) nw[i] = bf16_bits_to_f32(p.norm_w[lane * 4 + i]);
    }

    const bool vec_saves = ((reinterpret_cast<uintptr_t>(p.k_save) | reinterpret_cast<uintptr_t>(p.g_save) | reinterpret_cast<uintptr_t>(p.v_save)) & 15) == 0;
    // The core form's outputs leave sixteen bytes a thread (two bytes a thread, sixteen stores each, held up whatever came after them),
    // behind the next unit's first barrier.  An output buffer off 16 bytes takes them two bytes a thread, a row at a time.
    const bool vec_out = (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
    long long out_at = 0;
    int out_n = 0;
    auto out_rows = [&] {
        if (vec_out) {
#pragma unroll
            for (int i = 0; i < WIN / 8; ++i) {
                const int r = (t >> 4) + 8 * i, c = (t & 15) * 8;
                if (r < out_n) *reinterpret_cast<uint4*>(p.out + out_at + (long long)r * p.H * DV + c) = *reinterpret_cast<const uint4*>(smem + MP::vOut + (r * DV + c) * 2);
            }
        } else {
            for (int r = 0; r < out_n; ++r) p.out[out_at + (long long)r * p.H * DV + t] = reinterpret_cast<const uint16_t*>(smem + MP::vOut)[r * DV + t];
        }
    };
    Units units(p);
    Unit un, nxt;
    bool more = units.take(p, nxt);
    if (more) {
        fetch_rows<LAYER>(p, smem, nxt, t);
        fetch_state(p, smem, nxt, t, bar + 1);
    }
    while (more) {
        un = nxt;
        more = units.take(p, nxt);
        if (un.n > WIN && t == 0) atomicCAS(p.status, 0, kStatusVerifyWindow);
        const int n = min(max(un.n, 0), WIN);

        cp_async_wait<1>();  // this unit's rows have landed (its state may still be on the way)
        __syncthreads();     // and every thread is done with the previous unit's L, M and staged outputs
        if constexpr (!LAYER) out_rows();
        out_at = (un.row0 * p.H + un.h) * DV;
        out_n = n;

        // ---- A. the decay factors and the operand tiles: channels c0 and c0 + 1, eight rows -------------------------------------
        float kg[WIN], vv[WIN];
        float2 qe[WIN / 2];
        const bool upper = lane >= 16;
        const int c0 = warp * 32 + (lane & 15) * 2;
        {
            unsigned char* raw = smem + vRaw;
            float2 m[WIN / 2], kgp[WIN / 2];
#pragma unroll
            for (int s = 0; s < WIN / 2; ++s) {
                float2* x = reinterpret_cast<float2*>(raw + R::G + (row_of(s, upper) * DK + c0) * 4);
                m[s] = *x;
                if constexpr (LAYER) {  // the saved multipliers; the rows past the window decay by nothing
                    if (row_of(s, upper) >= n) m[s] = {1.0f, 1.0f};
                } else {  // of the log decays, by the exact path's expf; save_rows() takes them from here
                    m[s] = {expf(m[s].x), expf(m[s].y)};
                    *x = m[s];
                }
            }
            const Factors fac(m, upper);
            float amax = 0.0f;
#pragma unroll
            for (int s = 0; s < WIN / 2; ++s) {
                const int row = row_of(s, upper), at2 = (row * DK + c0) * 2;
                float2 kf, qf, a, inva;
                const uint32_t qw = *reinterpret_cast<const uint32_t*>(raw + R::Q + at2);
                if constexpr (LAYER) {
                    kf = *reinterpret_cast<const float2*>(raw + R::K + at2 * 2);
                    qf = __half22float2(*reinterpret_cast<const __half2*>(&qw));
                } else {
                    kf = widen_bf16x2(*reinterpret_cast<const uint32_t*>(raw + R::K + at2));
                    qf = widen_bf16x2(qw);
                }
                fac.relative(s, a, inva);
                const float2 e = fac.from_start(s);
                amax = fmaxf(amax, fmaxf(a.x, a.y));
                kgp[s] = mul2(kf, e);
                qe[s] = mul2(qf, e);  // the Qg rows are written when Qgb's have been read
                const float2 kb = mul2(kf, a), qb = mul2(qf, a), kc = mul2(kf, inva);
                *reinterpret_cast<uint32_t*>(smem + vRow + sw_elem(kRowR, row, c0)) = tc::bf16x2(kb.x, kb.y);
                *reinterpret_cast<uint32_t*>(smem + vRow + sw_elem(kRowR, WIN + row, c0)) = tc::bf16x2(qb.x, qb.y);
                *reinterpret_cast<uint32_t*>(smem + vKc + sw_elem(WIN, row, c0)) = tc::bf16x2(kc.x, kc.y);
            }
            all_rows(kgp, upper, kg);
#pragma unroll
            for (int r = 0; r < WIN; ++r) vv[r] = bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(raw + R::V)[r * DK + t]);
            if (!(amax < 1e37f) || fac.lost()) atomicCAS(p.status, 0, kStatusPrefillRange);
            if (t < WIN) {
                const float bt = reinterpret_cast<const float*>(raw + R::B)[t];
                betas[t] = bt;
            }
        }
        fence_proxy_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if constexpr (LAYER) {  // the raw rows are consumed: the next unit's may come in
            if (more) fetch_rows<LAYER>(p, smem, nxt, t);
            else cp_async_commit();
        }

        // ---- B. L^T and M^T -------------------------------------------------------------------------------------------------
        if (warp == 0) {
            const uint32_t leader = tc::elect_one();
            constexpr uint32_t id = tc::idesc_bf16(64, kRowR, 0, 0, 0);
#pragma unroll
            for (int k0 = 0; k0 < DK; k0 += 16)
                tc::mma_bf16_if(leader, tm, tc::desc_sw128_kmajor(smem + vKc, WIN, k0), tc::desc_sw128_kmajor(smem + vRow, kRowR, k0), id, k0 > 0);
            tc::mma_commit_if(leader, bar);
            if (leader) atomicAdd(const_cast<uint32_t*>(ctl), 1u);
            __syncwarp();
        }
        if constexpr (!LAYER) save_rows(p, smem, un, n, t, vec_saves);  // while the products run
        bool ok = mbar_wait(bar, phase, ctx, kStatusWaitPrefill);
        phase ^= 1u;
        if (!__syncthreads_and(ok)) break;
        tc::fence_after_sync();
        if constexpr (!LAYER) {  // the raw rows are consumed
            if (more) fetch_rows<LAYER>(p, smem, nxt, t);
            else cp_async_commit();
        }
        if (warp == 0) {  // tensor-memory lane = column j, column = row i of L, then of M.  Kc is dead: L, M go over it.
            uint32_t l16[8], m16[8];  // the fragment layout: columns j and j + 8, rows i = 8 g + 2 (lane % 4) and the next
            tc::tmem_ld_frag(tm, l16);
            tc::tmem_ld_frag(tm + 16, m16);
            tc::tmem_ld_wait();
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int j = (lane >> 2) + 8 * (x & 1), i = 8 * (x >> 1) + 2 * (lane & 3);
                const float l0 = i > j ? -betas[i] * __uint_as_float(l16[2 * x]) : 0.0f, l1 = i + 1 > j ? -betas[i + 1] * __uint_as_float(l16[2 * x + 1]) : 0.0f;
                Ln[i * LN + j] = make_float2(l0, l0);
                Ln[(i + 1) * LN + j] = make_float2(l1, l1);
                *reinterpret_cast<uint2*>(Mf + j * WIN + i) = make_uint2(i < j ? 0u : m16[2 * x], i + 1 < j ? 0u : m16[2 * x + 1]);
            }
        }
#pragma unroll
        for (int s = 0; s < WIN / 2; ++s) *reinterpret_cast<uint32_t*>(smem + vRow + sw_elem(kRowR, WIN + row_of(s, upper), c0)) = tc::bf16x2(qe[s].x, qe[s].y);
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();

        // ---- C. W = (I + L)^-1 diag(beta) Kg into its tile (thread = channel c0 + upper), U = (I + L)^-1 diag(beta) V in registers
        //         (thread = value channel), both by forward substitution down the 16 rows: the same multiply-adds as a product
        //         with an explicit inverse, without the inverse
        float2 wu[WIN];
        substitute(Ln, betas, kg, vv, wu);
#pragma unroll
        for (int i = 0; i < WIN; ++i) *reinterpret_cast<uint16_t*>(smem + vRow + sw_elem(kRowR, i, c0 + upper)) = f32_to_bf16_bits(wu[i].x);
        cp_async_wait<1>();  // this unit's state has landed (the next unit's rows may still be on the way)
        if (in_boxes(p.mapped, un.s_elem)) {
            ok = mbar_wait(bar + 1, state_phase, ctx, kStatusWaitPrefill);
            state_phase ^= 1u;
        }
        fence_proxy_async_smem();
        tc::fence_before_sync();
        if (!__syncthreads_and(ok)) break;
        tc::fence_after_sync();

        // ---- D. (W S)^T and (Qg S)^T: the state tile as it lies in memory is the M operand ---------------------------------------
        if (warp == 0) {
            const uint32_t leader = tc::elect_one();
            constexpr uint32_t id = tc::idesc_bf16(128, kRowR, 0, 0, 0);
#pragma unroll
            for (int k0 = 0; k0 < DK; k0 += 16)
                tc::mma_bf16_if(leader, tm, tc::desc_sw128_kmajor(smem + vS, DV, k0), tc::desc_sw128_kmajor(smem + vRow, kRowR, k0), id, k0 > 0);
            tc::mma_commit_if(leader, bar);
            if (leader) atomicAdd(const_cast<uint32_t*>(ctl), 1u);
            __syncwarp();
        }
        ok = mbar_wait(bar, phase, ctx, kStatusWaitPrefill);
        phase ^= 1u;
        if (!__syncthreads_and(ok)) break;
        tc::fence_after_sync();
        // The state tile is consumed: the next unit's may come in.
        if (more) fetch_state(p, smem, nxt, t, bar + 1);
        else cp_async_commit();

        // ---- E. D = U - W S,  O = Qg S + M D; thread = value channel = its tensor-memory lane -----------------------------------------
        uint2 gate[4] = {};  // layer form: the gate values of the four rows that this warp normalises, on their way meanwhile
        if constexpr (LAYER) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (warp * 4 + k < n) gate[k] = *reinterpret_cast<const uint2*>(p.gate + (un.row0 + warp * 4 + k) * p.gate_stride + (long long)un.h * DV + lane * 4);
        }
        {
            uint32_t ws[16], qs[16];
            tc::tmem_ld16(tc::tmem_addr(tm, warp, 0), ws);
            tc::tmem_ld16(tc::tmem_addr(tm, warp, 16), qs);
            tc::tmem_ld_wait();
            float2 o[WIN / 2];  // rows 2 p and 2 p + 1
#pragma unroll
            for (int q = 0; q < WIN / 2; ++q) o[q] = {__uint_as_float(qs[2 * q]), __uint_as_float(qs[2 * q + 1])};
#pragma unroll
            for (int j = 0; j < WIN; ++j) {  // M's column j: rows j .. 15, zero above
                const float d = wu[j].y - __uint_as_float(ws[j]);
#pragma unroll
                for (int i = j / 4 * 4; i < WIN; i += 4) {
                    const float4 m = *reinterpret_cast<const float4*>(Mf + j * WIN + i);
                    if (i + 1 >= j) o[i / 2] = fma2({m.x, m.y}, {d, d}, o[i / 2]);
                    o[i / 2 + 1] = fma2({m.z, m.w}, {d, d}, o[i / 2 + 1]);
                }
            }
#pragma unroll
            for (int i = 0; i < WIN; ++i) {
                const float x = i & 1 ? o[i / 2].y : o[i / 2].x;
                if constexpr (LAYER) reinterpret_cast<float*>(smem + vStage)[i * DV + t] = x;  // W and Qg are dead
                else reinterpret_cast<uint16_t*>(smem + MP::vOut)[i * DV + t] = f32_to_bf16_bits(x);
            }
        }
        tc::fence_before_sync();  // the next unit's products overwrite these tensor-memory columns
        if constexpr (LAYER) {
            // The gated RMSNorm (reference kda.cu:188-201): a warp takes four rows, a lane four value channels.
            __syncthreads();
            float y[4][4], ss[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // (rows past the window: sums of numbers that nobody takes)
                const float4 y4 = *reinterpret_cast<const float4*>(smem + vStage + ((warp * 4 + k) * DV + lane * 4) * 4);
                y[k][0] = y4.x; y[k][1] = y4.y; y[k][2] = y4.z; y[k][3] = y4.w;
                ss[k] = 0.0f;
#pragma unroll
                for (int x = 0; x < 4; ++x) ss[k] = ss[k] + y[k][x] * y[k][x];
            }
#pragma unroll
            for (int o = 16; o; o >>= 1)
#pragma unroll
                for (int k = 0; k < 4; ++k) ss[k] = ss[k] + __shfl_xor_sync(0xffffffffu, ss[k], o);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = warp * 4 + k;
                if (i >= n) break;
                const float rinv = rsqrtf(ss[k] * (1.0f / (float)DV) + p.eps);
                const long long gr = un.row0 + i;
                const float gt[4] = {__uint_as_float(gate[k].x << 16), __uint_as_float(gate[k].x & 0xffff0000u), __uint_as_float(gate[k].y << 16),
                                     __uint_as_float(gate[k].y & 0xffff0000u)};
                uint32_t o2[2];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float lo = (nw[2 * x] * (y[k][2 * x] * rinv)) * sigmoid_(gt[2 * x]);
                    const float hi = (nw[2 * x + 1] * (y[k][2 * x + 1] * rinv)) * sigmoid_(gt[2 * x + 1]);
                    o2[x] = tc::bf16x2(lo, hi);
                }
                *reinterpret_cast<uint2*>(p.out + gr * p.out_stride + (long long)un.h * DV + lane * 4) = make_uint2(o2[0], o2[1]);
            }
        }
    }
    cp_async_wait<0>();
    abort_pause(ctl);
    tc::fence_before_sync();
    __syncthreads();
    if constexpr (!LAYER) {
        if (ctl[1] == 0u) out_rows();
    }
    if (warp == 0) tc::tmem_dealloc(tm, kVCols);
}

// ---- the commit as chunks of 16 rows ---------------------------------------------------------------------------------
// The state after the first keep[b] saved rows, for every (request, layer, head): S <- E S + Kdec^T D per chunk of up to
// 16 rows, with D = U - W S as above, E = exp(G_last) and Kdec_i = k_i exp(G_last - G_i).  The inputs are the replay
// saves (k and the decay multiplier f32, v bf16, beta).  The bf16 state tile is the A operand of S W^T where it lies;
// the update D^T x Kdec (M = 128 value rows, N = 128 key channels, K = 16 rows) runs as three products of bf16 hi/lo
// halves (the path into the state keeps 16 bits of operand mantissa, as in the prefill), its FP32 accumulator is read
// back lane = value row, E S is added in FP32 and the rounded row goes back into the tile, which is then the next
// chunk's state or is copied out.  Unlike the exact replay this rounds the state to bf16 once per chunk instead of
// after every row, and its sums run in another order: the committed state agrees with serial decode steps to the last
// bits of bf16, not bit for bit (glm53f_kda_commit_mode).
// Three blocks per SM: the stages of a unit are serial, so what overlaps one unit's waits is the other resident blocks' work.  A
// chunk's saved rows arrive in shared memory by asynchronous copies issued one chunk (or unit) ahead, and the unit's metadata is
// read a unit ahead: taken straight from global memory, queued behind the state before's stores, they were 15,000 of a unit's
// 25,800 cycles, which a fourth block (no room for the rows) did not cover. 
// The hi half of D^T shares its 4 KB with Kc and L: Kc is read by the L^T product only, L by the forward substitution only, and
// D^T is written after the (W S)^T product, which comes after both.
constexpr int cS = 0, cDT = 32768, cKc = cDT, cKgb = cDT + 8192, cKdT = cKgb + 4096, cE = cKdT + 8192, cBeta = cE + 512;
constexpr int cBar = cBeta + 64 /* products, state */, cCtl = cBar + 16, cRawK = cCtl + 16, cRawG = cRawK + WIN * DK * 4, cRawV = cRawG + WIN * DK * 4, kCSmem = cRawV + WIN * DV * 2;
constexpr int cW = cKgb, cL = cKc;                    // W replaces Kgb, L replaces Kc once L^T is done
constexpr uint32_t kCCols = 128;                      // tensor memory: L^T, then (W S)^T, then the 128 x 128 update
constexpr int kCBlocks = 3;
static_assert(kCBlocks * (kCSmem + 1024) <= 228 * 1024 && kCBlocks * kCCols <= 512, "three blocks per SM");
static_assert(cRawK % 16 == 0 && WIN * LN * 8 <= 4096, "");

struct CParams {
    alignas(64) CUtensorMap tm_in, tm_out;
    int mapped;
    int H, layers, rows1;
    long long units;
    const int32_t* cu;
    const int32_t* keep;
    const uint16_t* state_in;
    uint16_t* state_out;
    long long state_stride;
    const long long* state_off;
    const float* k_save;
    const uint16_t* v_save;
    const float* g_save;
    const float* b_save;
    long long kv_stride, b_stride;
    int* status;
};

static_assert(cS == 0, "state_piece() is the place in the tile");

__global__ void __launch_bounds__(kVThreads, kCBlocks) commit_tc_kernel(const __grid_constant__ CParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + cBar);
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + cCtl);
    uint32_t* tmem_slot = const_cast<uint32_t*>(ctl) + 2;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 1, 1);
        ctl[0] = 0u;
        ctl[1] = 0u;
        mbar_init_fence();
    }
    if (warp == 0) tc::tmem_alloc(tmem_slot, kCCols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = *tmem_slot;
    grid_ready();
    const WaitCtx ctx{ctl, ctl + 1, p.status};
    uint32_t phase = 0, state_phase = 0;
    float2* Ln = reinterpret_cast<float2*>(smem + cL);
    float* En = reinterpret_cast<float*>(smem + cE);
    float* betas = reinterpret_cast<float*>(smem + cBeta);
    bool ok = true;

    // A unit's place and metadata; those of the next one are read a unit ahead, as they come (arithmetic would wait for them).
    const unsigned H = (unsigned)p.H, NL = (unsigned)p.layers;
    unsigned h = blockIdx.x % H, layer = blockIdx.x / H % NL, b = blockIdx.x / H / NL;
    int m_row = 0, m_keep = p.rows1;
    long long m_off = 0;
    auto fetch_meta = [&]() {
        if (p.cu) m_row = p.cu[b];
        if (p.keep) m_keep = p.keep[b];
        if (p.state_off) m_off = p.state_off[b];
    };
    const bool vec_rows = ((reinterpret_cast<uintptr_t>(p.k_save) | reinterpret_cast<uintptr_t>(p.v_save) | reinterpret_cast<uintptr_t>(p.g_save)) & 15) == 0 && p.kv_stride % 8 == 0;
    // Rows row .. row + n - 1 (n <= 16) of the saves; the places of the others keep what they hold.
    auto fetch_saves = [&](unsigned lay, unsigned head, long long row, int n) {
        const long long base = (long long)lay * p.kv_stride + (row * H + head) * DK;
        if (vec_rows) {
            const long long rs = (long long)H * DK, at = base + (t >> 5) * rs + (t & 31) * 4;  // four rows a step
#pragma unroll
            for (int i = 0; i < WIN / 4; ++i)
                if ((t >> 5) + 4 * i < n) {
                    cp_async16(smem + cRawK + (t + i * kVThreads) * 16, p.k_save + at + i * 4 * rs);
                    cp_async16(smem + cRawG + (t + i * kVThreads) * 16, p.g_save + at + i * 4 * rs);
                }
            const uint16_t* vs = p.v_save + base + (t >> 4) * rs + (t & 15) * 8;  // eight
#pragma unroll
            for (int i = 0; i < WIN / 8; ++i)
                if ((t >> 4) + 8 * i < n) cp_async16(smem + cRawV + (t + i * kVThreads) * 16, vs + i * 8 * rs);
        } else {
            for (int r = 0; r < n; ++r) {
                const long long at = base + (long long)r * H * DK + t;
                reinterpret_cast<float*>(smem + cRawK)[r * DK + t] = p.k_save[at];
                reinterpret_cast<float*>(smem + cRawG)[r * DK + t] = p.g_save[at];
                reinterpret_cast<uint16_t*>(smem + cRawV)[r * DV + t] = p.v_save[at];
            }
        }
        cp_async_commit();
    };
    if (blockIdx.x < p.units) {
        fetch_meta();
        fetch_saves(layer, h, m_row, min(max(m_keep, 0), WIN));
    }

    for (long long u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
        const long long row0 = m_row;
        const int n = max(m_keep, 0);
        const unsigned uh = h, ul = layer;
        const long long s_elem = (long long)ul * p.state_stride + m_off + (long long)uh * DV * DK;
        const uint16_t* src = p.state_in + s_elem;
        uint16_t* dst = p.state_out + s_elem;
        const bool more = u + gridDim.x < p.units;
        {
            const unsigned nh = h + gridDim.x, dq = nh / H, nl = layer + dq, lq = nl / NL;
            h = nh - dq * H;
            layer = nl - lq * NL;
            b += lq;
        }
        if (more) fetch_meta();
        auto fetch_next = [&]() { fetch_saves(layer, h, m_row, more ? min(max(m_keep, 0), WIN) : 0); };
        if (n == 0 && dst == src) {
            fetch_next();
            continue;
        }
        const long long b_base = (long long)ul * p.b_stride;
        __syncthreads();  // the previous unit's tile has been copied out
        // The unit's state into the swizzled tile.
        const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0, boxes = in_boxes(p.mapped, s_elem);
        if (t == 0) bulk_wait_read<0>();  // the unit before has left the tile
        if (boxes) {
            if (t == 0) load_boxes(smem + cS, &p.tm_in, s_elem, bar + 1);
        } else if (vec) {
            __syncthreads();
            unsigned char* to = smem + state_piece(t >> 4, t & 15);
#pragma unroll
            for (int i = 0; i < 16; ++i) cp_async16(to + i * 1024, src + (t + i * kVThreads) * 8);
        } else {
            __syncthreads();
            for (int e = t; e < DV * DK; e += kVThreads) *reinterpret_cast<uint16_t*>(smem + cS + sw_elem(DV, e >> 7, e & 127)) = src[e];
        }
        cp_async_commit();
        if (n == 0) fetch_next();
        bool landed = !boxes;
        auto state_lands = [&]() -> bool {
            if (landed) return true;
            landed = true;
            const bool there = mbar_wait(bar + 1, state_phase, ctx, kStatusWaitPrefill);
            state_phase ^= 1u;
            return there;
        };

        for (int c0 = 0; c0 < n && ok; c0 += WIN) {
            const int nr = min(WIN, n - c0);
            const float bt = t < nr ? p.b_save[b_base + (row0 + c0 + t) * H + uh] : 0.0f;  // (t < 16 uses it)
            if (c0 == 0) cp_async_wait<1>();  // its rows are there (the state may still be on the way)
            else cp_async_wait<0>();
            __syncthreads();
            // ---- A. the decay factors and the operand tiles: channels ch0 and ch0 + 1, eight rows; thread = value channel: v ---------
            float kg[WIN], vv[WIN];
            const bool upper = lane >= 16;
            const int ch0 = warp * 32 + (lane & 15) * 2;
            {
                float2 m[WIN / 2], kgp[WIN / 2];
                float amax = 0.0f;
#pragma unroll
                for (int s = 0; s < WIN / 2; ++s) {
                    m[s] = {1.0f, 1.0f};
                    if (row_of(s, upper) < nr) m[s] = *reinterpret_cast<const float2*>(smem + cRawG + (row_of(s, upper) * DK + ch0) * 4);
                }
                const Factors fac(m, upper);
                uint32_t dh[2][WIN / 4], dl[2][WIN / 4];
#pragma unroll
                for (int r = 0; r < WIN / 2; r += 2) {
                    float2 kd[2];
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const int s = r + x, row = row_of(s, upper), to = sw_elem(WIN, row, ch0);
                        const float2 kf = row < nr ? *reinterpret_cast<const float2*>(smem + cRawK + (row * DK + ch0) * 4) : float2{0.0f, 0.0f};
                        float2 a, inva;
                        fac.relative(s, a, inva);
                        amax = fmaxf(amax, fmaxf(a.x, a.y));
                        kgp[s] = mul2(kf, fac.from_start(s));
                        kd[x] = mul2(kf, fac.to_end(s));
                        const float2 kb = mul2(kf, a), kc = mul2(kf, inva);
                        *reinterpret_cast<uint32_t*>(smem + cKgb + to) = tc::bf16x2(kb.x, kb.y);
                        *reinterpret_cast<uint32_t*>(smem + cKc + to) = tc::bf16x2(kc.x, kc.y);
                    }
                    // in the order of the rows: the lower half counts down
                    const float2 d0 = upper ? kd[0] : kd[1], d1 = upper ? kd[1] : kd[0];
                    tc::split_bf16x2(d0.x, d1.x, dh[0][r / 2], dl[0][r / 2]);
                    tc::split_bf16x2(d0.y, d1.y, dh[1][r / 2], dl[1][r / 2]);
                }
                // Kdec^T: row = key channel, 16 row indices along K = two 16-byte cells, of which this thread has one
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    unsigned char* to = smem + cKdT + ((upper ? DK : 0) + ch0 + x) * 16;
                    *reinterpret_cast<uint4*>(to) = upper ? make_uint4(dh[x][0], dh[x][1], dh[x][2], dh[x][3]) : make_uint4(dh[x][3], dh[x][2], dh[x][1], dh[x][0]);
                    *reinterpret_cast<uint4*>(to + 4096) = upper ? make_uint4(dl[x][0], dl[x][1], dl[x][2], dl[x][3]) : make_uint4(dl[x][3], dl[x][2], dl[x][1], dl[x][0]);
                }
                if (!upper) *reinterpret_cast<float2*>(&En[ch0]) = fac.all;
                all_rows(kgp, upper, kg);
#pragma unroll
                for (int r = 0; r < WIN; ++r) vv[r] = r < nr ? bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(smem + cRawV)[r * DV + t]) : 0.0f;
                if (!(amax < 1e37f) || fac.lost()) atomicCAS(p.status, 0, kStatusPrefillRange);
                if (t < WIN) betas[t] = bt;
            }
            fence_proxy_async_smem();
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();

            // The saved rows are consumed: the next chunk's, or the next unit's first, may come in.
            if (c0 + WIN < n) fetch_saves(ul, uh, row0 + c0 + WIN, min(WIN, n - c0 - WIN));
            else fetch_next();

            // ---- B. L^T ---------------------------------------------------------------------------------------------------
            if (warp == 0) {
                const uint32_t leader = tc::elect_one();
                constexpr uint32_t id = tc::idesc_bf16(64, WIN, 0, 0, 0);
#pragma unroll
                for (int k0 = 0; k0 < DK; k0 += 16)
                    tc::mma_bf16_if(leader, tm, tc::desc_sw128_kmajor(smem + cKc, WIN, k0), tc::desc_sw128_kmajor(smem + cKgb, WIN, k0), id, k0 > 0);
                tc::mma_commit_if(leader, bar);
                if (leader) atomicAdd(const_cast<uint32_t*>(ctl), 1u);
                __syncwarp();
            }
            ok = mbar_wait(bar, phase, ctx, kStatusWaitPrefill);
            phase ^= 1u;
            ok = __syncthreads_and(ok);
            if (!ok) break;
            tc::fence_after_sync();
            if (warp == 0) {
                uint32_t l16[8];  // the fragment layout, as in the verify
                tc::tmem_ld_frag(tm, l16);
                tc::tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int j = (lane >> 2) + 8 * (x & 1), i = 8 * (x >> 1) + 2 * (lane & 3);
                    const float l0 = i > j ? -betas[i] * __uint_as_float(l16[2 * x]) : 0.0f, l1 = i + 1 > j ? -betas[i + 1] * __uint_as_float(l16[2 * x + 1]) : 0.0f;
                    Ln[i * LN + j] = make_float2(l0, l0);
                    Ln[(i + 1) * LN + j] = make_float2(l1, l1);
                }
            }
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();

            // ---- C. W and U by forward substitution ---------------------------------------------------------------------------
            float2 wu[WIN];
            substitute(Ln, betas, kg, vv, wu);
#pragma unroll
            for (int i = 0; i < WIN; ++i) *reinterpret_cast<uint16_t*>(smem + cW + sw_elem(WIN, i, ch0 + upper)) = f32_to_bf16_bits(wu[i].x);  // over Kgb, which is consumed
            cp_async_wait<1>();  // the state has landed (the next rows may still be on the way)
            ok = state_lands();
            fence_proxy_async_smem();
            tc::fence_before_sync();
            ok = __syncthreads_and(ok);
            if (!ok) break;
            tc::fence_after_sync();

            // ---- D. (W S)^T = S W^T --------------------------------------------------------------------------------------------
            if (warp == 0) {
                const uint32_t leader = tc::elect_one();
                constexpr uint32_t id = tc::idesc_bf16(128, WIN, 0, 0, 0);
                for (int k0 = 0; k0 < DK; k0 += 16)
                    tc::mma_bf16_if(leader, tm, tc::desc_sw128_kmajor(smem + cS, DV, k0), tc::desc_sw128_kmajor(smem + cW, WIN, k0), id, k0 > 0);
                tc::mma_commit_if(leader, bar);
                if (leader) atomicAdd(const_cast<uint32_t*>(ctl), 1u);
                __syncwarp();
            }
            ok = mbar_wait(bar, phase, ctx, kStatusWaitPrefill);
            phase ^= 1u;
            ok = __syncthreads_and(ok);
            if (!ok) break;
            tc::fence_after_sync();

            // ---- E. D = U - W S as the A operand D^T (row = value channel t, hi and lo halves) ------------------------------
            {
                uint32_t ws[16];
                tc::tmem_ld16(tc::tmem_addr(tm, warp, 0), ws);
                tc::tmem_ld_wait();
                uint32_t dh[WIN / 2], dl[WIN / 2];
#pragma unroll
                for (int i = 0; i < WIN; i += 2) {
                    tc::split_bf16x2(wu[i].y - __uint_as_float(ws[i]), wu[i + 1].y - __uint_as_float(ws[i + 1]), dh[i / 2], dl[i / 2]);
                }
                *reinterpret_cast<uint4*>(smem + cDT + (0 * DV + t) * 16) = make_uint4(dh[0], dh[1], dh[2], dh[3]);
                *reinterpret_cast<uint4*>(smem + cDT + (1 * DV + t) * 16) = make_uint4(dh[4], dh[5], dh[6], dh[7]);
                *reinterpret_cast<uint4*>(smem + cDT + 4096 + (0 * DV + t) * 16) = make_uint4(dl[0], dl[1], dl[2], dl[3]);
                *reinterpret_cast<uint4*>(smem + cDT + 4096 + (1 * DV + t) * 16) = make_uint4(dl[4], dl[5], dl[6], dl[7]);
            }
            fence_proxy_async_smem();
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();

            // ---- F. the update D^T x Kdec: [value row][key channel], three products of halves ------------------------------------
            if (warp == 0) {
                const uint32_t leader = tc::elect_one();
                constexpr uint32_t id = tc::idesc_bf16(128, 128, 0, 0, 0);
                tc::mma_bf16_if(leader, tm, tc::desc_kmajor_bf16(smem + cDT, DV, 0, 0), tc::desc_kmajor_bf16(smem + cKdT, DK, 0, 0), id, false);
                tc::mma_bf16_if(leader, tm, tc::desc_kmajor_bf16(smem + cDT, DV, 0, 0), tc::desc_kmajor_bf16(smem + cKdT + 4096, DK, 0, 0), id, true);
                tc::mma_bf16_if(leader, tm, tc::desc_kmajor_bf16(smem + cDT + 4096, DV, 0, 0), tc::desc_kmajor_bf16(smem + cKdT, DK, 0, 0), id, true);
                tc::mma_commit_if(leader, bar);
                if (leader) atomicAdd(const_cast<uint32_t*>(ctl), 1u);
                __syncwarp();
            }
            ok = mbar_wait(bar, phase, ctx, kStatusWaitPrefill);
            phase ^= 1u;
            ok = __syncthreads_and(ok);
            if (!ok) break;
            tc::fence_after_sync();

            // ---- G. S <- E S + update, rounded to bf16, back into the tile (thread = value row) ------------------------------
            uint32_t acc[2][32];  // a quarter of the row, and the next on its way
            tc::tmem_ld32(tc::tmem_addr(tm, warp, 0), acc[0]);
#pragma unroll
            for (int cg = 0; cg < DK / 32; ++cg) {
                tc::tmem_ld_wait();
                if (cg + 1 < DK / 32) tc::tmem_ld32(tc::tmem_addr(tm, warp, (cg + 1) * 32), acc[(cg + 1) & 1]);
                const uint32_t* a16 = acc[cg & 1];
#pragma unroll
                for (int half = 0; half < 4; ++half) {
                    unsigned char* at = smem + state_piece(t, cg * 4 + half);
                    const uint4 sv = *reinterpret_cast<const uint4*>(at);
                    const uint32_t sw[4] = {sv.x, sv.y, sv.z, sv.w};
                    uint32_t out[4];
#pragma unroll
                    for (int x = 0; x < 4; x += 2) {
                        const float4 e4 = *reinterpret_cast<const float4*>(&En[cg * 32 + half * 8 + 2 * x]);
                        const uint32_t* a4 = a16 + half * 8 + 2 * x;
                        const float2 s0 = fma2({e4.x, e4.y}, widen_bf16x2(sw[x]), {__uint_as_float(a4[0]), __uint_as_float(a4[1])});
                        const float2 s1 = fma2({e4.z, e4.w}, widen_bf16x2(sw[x + 1]), {__uint_as_float(a4[2]), __uint_as_float(a4[3])});
                        out[x] = tc::bf16x2(s0.x, s0.y);
                        out[x + 1] = tc::bf16x2(s1.x, s1.y);
                    }
                    *reinterpret_cast<uint4*>(at) = make_uint4(out[0], out[1], out[2], out[3]);
                }
            }
            fence_proxy_async_smem();  // the next chunk's S W^T reads the tile through the async proxy
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();
        }
        if (!ok) break;
        if (n == 0) {  // a unit without rows: its state is only copied
            cp_async_wait<1>();
            ok = state_lands();
            if (!__syncthreads_and(ok)) break;
        }
        // ---- the tile back to global memory, coalesced ------------------------------------------------------------------------
        if (boxes) {  // (the last chunk's end has published the tile to these copies)
            if (t == 0) {
                for (int x = 0; x < 2; ++x) tensor_store_3d(&p.tm_out, 0, x, (int)(s_elem / DK), smem + cS + x * 16384);
                bulk_commit();
            }
        } else if (vec) {
            const unsigned char* from = smem + state_piece(t >> 4, t & 15);
#pragma unroll
            for (int i = 0; i < 16; ++i) *reinterpret_cast<uint4*>(dst + (t + i * kVThreads) * 8) = *reinterpret_cast<const uint4*>(from + i * 1024);
        } else {
            for (int e = t; e < DV * DK; e += kVThreads) dst[e] = *reinterpret_cast<const uint16_t*>(smem + cS + sw_elem(DV, e >> 7, e & 127));
        }
    }
    if (t == 0) bulk_wait_all<0>();
    cp_async_wait<0>();
    abort_pause(ctl);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tm, kCCols);
}

template <bool LAYER>
int launch_verify(const VParams& p, cudaStream_t stream) {
    static int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(verify_tc_kernel<LAYER>, cudaFuncAttributeMaxDynamicSharedMemorySize, Map<LAYER>::kSmem);
        if (e != cudaSuccess) return (int)e;
        configured_dev = dev;
    }
    if (p.status == nullptr) return (int)cudaErrorUnknown;
    const long long cap = 3LL * sm_count();
    return launch_early(verify_tc_kernel<LAYER>, (unsigned)(p.units < cap ? p.units : cap), kVThreads, Map<LAYER>::kSmem, stream, p);
}

}  // namespace

// The chunked verify of the core entry point: bf16 states, no state written, no fused norm, q, k, v and g on 16 bytes (the
// caller checks); states, outputs and saves at any element.
int core_verify_tc_launch(int32_t heads, int32_t batch, const int32_t* cu_rows, const glm53f_bf16* q, const glm53f_bf16* k,
                          const glm53f_bf16* v, const float* g, const float* beta, const void* state_in, const int64_t* state_off,
                          glm53f_bf16* out, float* k_save, glm53f_bf16* v_save, float* g_save, float* b_save, cudaStream_t stream) {
    VParams p{};
    p.H = heads;
    p.units = (long long)heads * batch;
    p.cu = cu_rows;
    p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta;
    p.state = reinterpret_cast<const uint16_t*>(state_in);
    p.mapped = state_map(&p.tm_state, state_in);
    p.state_off = reinterpret_cast<const long long*>(state_off);
    p.out = out;
    p.out_stride = (long long)heads * DV;
    p.k_save = k_save; p.v_save = v_save; p.g_save = g_save; p.b_save = b_save;
    p.status = status_word();
    return launch_verify<false>(p, stream);
}

// The chunked verify of the layer entry point, after verify_prologue_launch on the same stream: the saves hold k, v, the
// decay multiplier and beta of every window row, `out` holds q as fp16 and receives the gated, normalised outputs.
int layer_verify_tc_launch(int32_t heads, int32_t batch, const int32_t* cu_rows, const void* state_in, const int64_t* state_off,
                           const glm53f_bf16* gate, int64_t gate_stride, const glm53f_bf16* norm_w, float eps, glm53f_bf16* out,
                           int64_t out_stride, float* k_save, glm53f_bf16* v_save, float* g_save, float* b_save, cudaStream_t stream) {
    VParams p{};
    p.H = heads;
    p.units = (long long)heads * batch;
    p.cu = cu_rows;
    p.state = reinterpret_cast<const uint16_t*>(state_in);
    p.mapped = state_map(&p.tm_state, state_in);
    p.state_off = reinterpret_cast<const long long*>(state_off);
    p.out = out;
    p.out_stride = out_stride;
    p.k_save = k_save; p.v_save = v_save; p.g_save = g_save; p.b_save = b_save;
    p.gate = gate; p.gate_stride = gate_stride; p.norm_w = norm_w; p.eps = eps;
    p.status = status_word();
    return launch_verify<true>(p, stream);
}

// The chunked commit (bf16 states; the caller checks that the saves are 4-byte aligned, which every float array is).
int commit_tc_launch(int32_t heads, int32_t layers, int32_t batch, const int32_t* cu_rows, const int32_t* keep, int32_t rows1, const void* state_in,
                     void* state_out, int64_t state_stride, const int64_t* state_off, const float* k_save, const glm53f_bf16* v_save,
                     const float* g_save, const float* b_save, int64_t kv_stride, int64_t b_stride, cudaStream_t stream) {
    static int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(commit_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCSmem);
        if (e != cudaSuccess) return (int)e;
        configured_dev = dev;
    }
    CParams p{};
    p.H = heads; p.layers = layers; p.rows1 = rows1;
    p.units = (long long)heads * layers * batch;
    p.cu = cu_rows; p.keep = keep;
    p.state_in = reinterpret_cast<const uint16_t*>(state_in);
    p.state_out = reinterpret_cast<uint16_t*>(state_out);
    p.mapped = state_map(&p.tm_in, state_in) && state_map(&p.tm_out, state_out);
    p.state_stride = state_stride;
    p.state_off = reinterpret_cast<const long long*>(state_off);
    p.k_save = k_save; p.v_save = v_save; p.g_save = g_save; p.b_save = b_save;
    p.kv_stride = kv_stride; p.b_stride = b_stride;
    p.status = status_word();
    if (p.status == nullptr) return (int)cudaErrorUnknown;
    const long long cap = (long long)kCBlocks * sm_count();
    return launch_early(commit_tc_kernel, (unsigned)(p.units < cap ? p.units : cap), kVThreads, kCSmem, stream, p);
}

}  // namespace kda
