// Chunk-64 KDA prefill on the 5th-generation tensor cores (tcgen05 + TMEM): in two roles over a caller-provided workspace (the core entry points
// that take one, and the chunked form of the layer prefill), or one block a chain without one (prefill_one_kernel).
//
// The head's 128 x 128 state stays in tensor memory (FP32) from a walk's first chunk to its last.  Per chunk (the algebra of the reference's CPU
// definition crates/glm53f-kda/src/chunked.rs:67-198, which itself restates chunk_kimi_delta_attention):
//
//   G_i   = g_0 + ... + g_i per key channel (FP32 scan), E = exp(G), E_last = exp(G_63)
//   Kg = k*E, Qg = q*E, Kinv = k/E, Kdec = k * E_last/E                       (operand tiles, written by hand)
//   L = Kg Kinv^T, M = Qg Kinv^T      64x64x128 MMAs; L strictly lower * beta_i, M lower incl. diagonal
//   T  = (I + L)^-1                   16 x 16 diagonal blocks by substitution, then the lower-left block of every
//                                     2sz x 2sz diagonal block is -T22 (L21 T11), sz = 16, 32;  T' = T diag(beta)
//   W  = T' Kg,  U = T' V             T' as bf16 hi + lo for U
//   D  = U - W S,  QS = Qg S          MMAs on a bf16 copy of S
//   O  = QS + M D
//   S <- E_last * S + Kdec^T D        Kdec and D as bf16 hi + lo (three products)
//
// Operand precision follows a CPU study of this exact scheme on the benchmark's input distribution: bf16
// operands are enough for every product that only reaches the output (M, QS, M D) and for L, W and W S, but not
// for U and Kdec^T D, which carry the state: those use two-term bf16 splits (16 mantissa bits).  With that mix
// the final state is within 5e-4 rel-L2 of the FP32 recurrence (limit 1e-3) and the bf16 outputs within 4e-3
// (limit 5e-3).
//
// Where it runs with a workspace.  Everything of a chunk that does not need the recurrent state -- the decay scan, the
// operand tiles, L, M, the triangular inverse, W = T'Kg and U = T'V, about two thirds of a chunk's time -- is
// independent from chunk to chunk, so the *intra role* spreads those (chain, chunk) items over every SM and leaves
// per item, in the workspace, exactly what the state recurrence consumes: Qg, W, M, Kdec hi/lo (bf16 cell tiles),
// U (FP32) and exp(G_last).  The *state role*, one block per chain, walks the chunks in order with the state in
// tensor memory and only the short dependent part per chunk: S as bf16 operand, QS = Qg S and -W S, D = U - W S,
// O = QS + M D, S <- E_last S + Kdec^T D.
//
// Where many chains are walked (WALK_U), T' as bf16 hi + lo goes into the workspace in U's place and the walk forms U itself, from V as the
// caller has it: 16 KiB less to write and to read an item, a product and a result less in the intra role, but eight products more in
// the walk, which only a walk that waits for memory does not notice.  The products and sums are the same, and so are the bits.  U in the items / in
// the walk, us: 262,144 rows x 64 heads 15,316 / 14,020, 8,192 rows x 64 heads in 8 sequences 517 / 484, the layer form's 4 x 2,048 rows 922 / 883.
// Of T', the quarter above the diagonal that is zero stays behind: another 2 to 4 % of the first two (65,536 rows 3,456 -> 3,383, 473 -> 454).  (M's
// likewise, for two products more: nothing.)
//
// The sequence is cut into segments sized by the workspace.  One kernel launch runs the state role for segment s-1
// (blocks 0..chains-1) and the intra role for segment s (every block, the chain blocks after their state work; items
// are handed out through a counter in the workspace), on two halves of the workspace that swap from launch to
// launch; stream order between launches is the only synchronisation.  With more chains than SMs, and for the layer entry
// points, one persistent launch a pass runs both roles over all the slots (fused_roles).
//
// Workspace slot of one (chain, chunk) item, bytes: U 0 (FP32, cells of four rows, [2][16][64 value channels]), or T' 4,096 (its columns 0-31 hi, lo: cells [4][64 rows],
// its columns 32-63 below the diagonal block's first row hi, lo: [4][32 rows]) and V 16,384 (boxes as they are staged: the layer prologue's, and of a sequence's partial chunk; any other V is read where the caller has it) | Qg 32,768 |
// W 49,152 (cells of eight rows, [8][128 key channels]) | M 65,536 | Kdec hi 73,728 | Kdec lo 90,112 | E_last 106,496 (128 floats); 107,008 per slot = 1,672 per row and head, inside
// the 2,176 the reference's prefill workspace formula provides (kernels/kda_prefill.cu:40-43, 695-698).  The last
// 256 bytes of the workspace hold the counters (kda_internal.h).

#include <cstdlib>

#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "glm53f_kda.h"
#include "kda_internal.h"
#include "prefill_common.cuh"
#include "tc.cuh"
#include "tensor_map.cuh"

namespace kda {
namespace {

using namespace pf;

// U is kept in FP32 as 16-byte cells of four rows of a value channel, the channels in two halves, so that both its writer (a
// thread holds a channel's rows) and its reader store and load consecutive cells.
__device__ __forceinline__ int u_cell(int row4, int v) { return (((v >> 6) * 16 + row4) * 64 + (v & 63)) * 16; }
// What the walk's loader brings in together lies together: U, or T' and V; Qg and W; M and Kdec.
constexpr int kTpBytes = 3 * kTile / 4, wU = 0, wTp = kTile - kTpBytes, wV = kTile, wQg = 2 * kTile, wW = 3 * kTile, wMm = 4 * kTile, wKdHi = wMm + kTile / 2, wKdLo = wKdHi + kTile;
constexpr int kUBytes = CH * DV * 4, wEgl = wKdLo + kTile, kSlotBytes = wEgl + 512;
static_assert(kSlotBytes == kPrefillSlotBytes && wV == kSlotInV && wTp >= kSlotInK && kSlotInK + kTile <= wV && wU + kUBytes == wQg, "a chunk's V stays where the layer prologue put it; T' goes over K");

// Staging of a chunk's raw rows in the intra kernel: dense boxes of 64 rows x 128 bytes written by tiled tensor copies
// with the 128-byte swizzle (16-byte piece p of row r sits at piece p ^ (r & 7)), so that threads walking down the
// rows of one column spread over all banks.  q, k, v: two boxes each (channels 0-63, 64-127); the log decays: four.
constexpr int kBox = CH * 128;  // 8 KiB
// Byte offset inside a tensor's staging of the 16-byte piece `piece` (0..15 for bf16 rows, 0..31 for f32 rows) of row r.
__device__ __forceinline__ int box_piece(int r, int piece) { return prefill_box_piece(r, piece); }

// Two 16-bit values of a q or k row to FP32: bf16 (the core entry points' inputs), or fp16 where the layer prologue produced
// them (normalised q and k lie in [-1, 1]; eleven mantissa bits instead of eight keep the rounding of k, which goes into
// the state through Kdec, below the state's error budget).
template <bool LAYER>
__device__ __forceinline__ float2 widen2(uint32_t w) {
    if constexpr (LAYER) return __half22float2(*reinterpret_cast<const __half2*>(&w));
    else return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

struct SpParams {
    alignas(64) CUtensorMap tm_q, tm_k, tm_v, tm_g;  // [rows][H][128] as (128, H, rows); boxes of 64 rows x 128 bytes, 128-byte swizzle
    alignas(64) CUtensorMap tm_out;                  // the shard-local output, the same way
    alignas(64) CUtensorMap tm_gate;                 // the gate rows, the same way (gate_boxes != 0)
    alignas(64) CUtensorMap tm_full[8];              // every rank's full output buffer: (128, heads_total, rows)
    int H, batch;
    const int32_t* cu;
    const uint16_t *q, *k, *v;
    const float* g;
    const float* beta;
    const void* state_in;   // segment 0 reads the caller's state, later segments the state written so far
    void* state_out;
    const long long* state_off;
    int state_bf16;
    const uint16_t* gate;
    long long gate_stride;  // elements between consecutive gate rows
    int longest_first;      // prefill_one_kernel: blocks take the longest sequences' chains first
    int gate_boxes;         // full chunks' gate values come by tiled tensor copies (base and stride on 16 bytes)
    const uint16_t* norm_w;
    float eps;
    uint16_t* out;
    int seg_chunks;          // chunks of every sequence per segment = slots per chain in a workspace half
    unsigned char* ws_intra; // intra role: chunks [intra_chunk0, intra_chunk0 + seg_chunks) of every sequence, or none
    int intra_chunk0, has_intra;
    unsigned char* ws_state; // state role: chunks [state_chunk0, state_chunk0 + seg_chunks) of every sequence, or none
    int state_chunk0, has_state;
    uint16_t* full[8];       // head-sharded launches: every rank's full [rows][heads_total][128] output buffer, or none
    int ranks, heads_total, head0;
    unsigned int* counters;  // [2] item counters: this launch hands items out of counters[ctr], and zeroes the other
    int ctr;
    // One persistent launch for both roles: items, then chains, are handed out from tail set ctr; chains form groups
    // of `group`, and a chain's state role starts when all items of its group are finished.
    int group;
    unsigned int* sets;
    // Blocks 0 .. early_blocks - 1, which will have a chain more to walk than the others, leave the last items, those from early_from on, to them.
    int early_blocks;
    long long early_from;
    int* status;
    // The scan over segments of the sequence (scan_pass != 0; FP32 states; the workspace holds every chunk).  Segment s of
    // a chain covers chunks [s * scan_chunks, (s + 1) * scan_chunks).
    //   pass 1  blocks (chain, s < K - 1, kind): the walk of segment s without outputs, from the zero state (kind 0: its
    //           end state is the segment's offset B_s) and from the identity with U = 0 (kind 1: its end state is the
    //           segment's transition A_s), written to scan_ab
    //   pass 2  blocks (chain, s): the walk of segment s with outputs from its true incoming state scan_start (composed
    //           from the A_s, B_s between the two passes); the last segment writes the final state
    int scan_pass, scan_k, scan_chunks;
    int scan_open;      // the last segment runs to the sequence's end (the call's last super-block), else to the end of
                        // this launch's chunk range [state_chunk0, state_chunk0 + seg_chunks)
    int scan_p1;        // segments pass 1 walks: K - 1, or K when the state after the range is wanted before pass 2 runs
    const float* scan_carry_in;  // super-blocks: the FP32 state before this launch's range, [chain][128 x 128] (NULL: state_in)
    float* scan_carry_out;       // super-blocks: the FP32 state after this launch's range (scan_p1 == K)
    float* scan_ab;     // [chain][K - 1][2][128 x 128]: B_s, A_s in the state's layout
    float* scan_start;  // [chain][K][128 x 128]: the state before each segment
};

__device__ __forceinline__ unsigned char* slot_of(unsigned char* ws, int seg_chunks, int chain, int jj) {
    return ws + ((size_t)chain * seg_chunks + jj) * kSlotBytes;
}

// Chain number n of a fused launch, in the order in which items and walks are handed out.  The layer form's goes backwards through the batch: its prologue has
// written the last requests' rows last, and those are still in L2.
__device__ __forceinline__ int chain_at(const SpParams& p, int n) { return p.v == nullptr ? p.batch * p.H - 1 - n : n; }

struct Item {
    int chain, jj, group;
};
// Chunk-major, neighbouring chains next to each other; in a fused launch so within each group of chains.
template <bool FUSED>
__device__ __forceinline__ Item item_of(const SpParams& p, int item) {
    const int chains = p.batch * p.H;
    if (!FUSED) return {item % chains, item / chains, 0};
    const int per = p.group * p.seg_chunks, g = item / per, rem = item - g * per, n = min(p.group, chains - g * p.group);
    return {chain_at(p, g * p.group + rem % n), rem / n, g};
}

// The state role's barriers sit behind every tile (set up once at kernel entry, never repurposed).  The intra role's
// live inside its two groups' areas, which the state role -- it runs first in a block -- uses as tile space, so they are
// set up when the intra role starts.
constexpr int oCtl = 14 * kTile;  // the block's control words
constexpr int oBarsState = oCtl + 32, oChain = oBarsState + 240, kSmemSp = oChain + 64;
// 16 compute warps, the loader warp, and (state role only) a warp that moves finished output rows to global memory and one that
// issues the tensor-core products.
constexpr int kThreadsSp = kCompute + 96, kLoaderWarp = kCompute / 32, kOutWarp = kCompute / 32 + 1, kMmaWarp = kCompute / 32 + 2;
static_assert(kSmemSp <= 232448, "shared memory budget");

// =====================================================================================================================
// Pass 1: the state-independent part of every (chain, chunk) item of the segment, items handed out by a counter.
//
// A block runs two items at a time: two groups of eight warps, each with its own staging, tensor-memory columns,
// barriers and loader warp, so that one group's waits (tensor-core rounds, tensor-memory reads, its own barriers) are
// filled by the other group's arithmetic.  To fit two items, a group keeps 96 KiB: q, k, v and the log decays arrive
// by tiled tensor copies in the 128-byte swizzle, which is an operand layout of the tensor core (K-major for the
// products over key channels, MN-major for the products over rows), so k and q are turned into Kg and Qg in place and
// v is used as it lands; the log decays become E in place; the inverse's FP32 scratch goes over E and Kinv once they
// are dead; and everything the state role needs leaves for the workspace straight from registers (Qg, Kdec hi/lo,
// E_last, M, W, U or T'), in the un-swizzled cell layout the state role reads, so no result tile lives in shared memory.
// =====================================================================================================================
constexpr int kGroupThreads = 256, kGroups = 2;
// Strong decays (core forms).  A thread sums its channel's decays over 32 rows, and what lies between two rows is a difference.  Of strong decays the rounding of long sums
// would pass through the exponential into the states.  So a thread whose first nine rows decay by more than e^-8.5 (as in a chunk of e^-60, from where on chunks take
// block-wise references) begins its sums anew at a block's first row and behind its middle row, and block-wise chunks form their tables once more, from the sums of
// just the decays between two rows.  The states' distance from 64 bits, decays of e^-4 and e^-5.8 a row that vary by a fifth: 4.5e-6 and 3.4e-6; from differences
// 1.1e-5 and 1.7e-5, of sums over sixteen rows 1.0e-5 and 1.5e-5; at e^-0.9 and milder the operands' rounding is all there is to see, either way.
// us, before / so: 8,192 rows in 8 sequences 463 / 463, 65,536 rows x 64 heads 3,555 / 3,559, 1,000 without a workspace 122.0 / 122.4; strong decays, 16,384 x 64 940 / 956, 1,000
// without 141.2 / 141.9.  The choice by a branch, or before the factors are formed, cost all chunks 1 to 3 %.
constexpr float kStrong = -8.5f * kLog2e;
// Decay range.  L and M hold exp(G_i - G_j) for every pair of rows j <= i of a chunk, and a tensor-core product can
// only form it as (row factor) x (column factor).  With the model's gate bound (log decay down to -5.8 per row, -371
// per chunk) neither exp(G) nor exp(-G) is representable, so the pair is split at a reference row r between j and i:
// exp(G_i - G_r) exp(G_r - G_j).  Rows are grouped in blocks of 16 and the reference of row block I is its middle row
// (16 I + 8).  The row side k_i exp(G_i - Gm_I) then stays within e^+-47; the column side for row block I is
// k_j exp(Gm_I - G_j) for every j below the end of block I: at most e^47 inside the block and at most 1 (vanishing
// harmlessly where the true product vanishes) in earlier blocks.  It depends on I, so there are four column-side
// tiles of 16, 32, 48 and 64 rows, and L^T, M^T are formed block column by block column (N = 16) with the column side
// as the M operand: rows past a tile's end produce entries above the diagonal, which are discarded.
constexpr int kKcBytes = 2 * 128 * (16 + 32 + 48 + 64);  // the four column-side tiles, boxes of R x 128 bytes
// Tile I starts at pf::kc_tile(I).  Byte offset inside tile I (R = 16 (I + 1) rows per box) of the 16-byte piece `piece` (0..15) of row r.
__device__ __forceinline__ int kc_piece(int I, int r, int piece) {
    return kc_tile(I) + (piece >> 3) * (I + 1) * 2048 + r * 128 + (((piece & 7) ^ (r & 7)) << 4);
}
constexpr int gK = 0, gV = kTile, gQ = 2 * kTile, gKb = 3 * kTile, gKc = 4 * kTile;  // K/Kg | V (unless WALK_U) | Q/Qgb | Kgb | the column-side tiles
// The log decays lie over the column-side tiles; the inverse's scratch and T' (hi | lo box, over L) over Q, Kgb and the 8 KiB before
// the log decays, so that the next item's log decays can arrive as soon as L and M are formed.
constexpr int gG = gKc + 8192, gT = gQ, gL = gT + CH * LS * 4, gTp = gL;
static_assert(gTp % 1024 == 0 && gKc % 1024 == 0, "swizzled tiles are 1024-byte aligned");
// Per-block decay factors, 128 channels each: E0[J] = exp(Gm_J), EL[J] = exp(G_last - Gm_J), F[I(I-1)/2 + J] =
// exp(Gm_I - Gm_J) for I > J.
constexpr int gTab = gKc + kKcBytes, gP = gTab, gBeta = gTab + kTabs * 512, gBars = gBeta + CH * 4, kGroupBars = 6, gItem = gBars + kGroupBars * 8, gGl = gItem + 16;  // gGl: exp(G_last) [128]
constexpr int kGroupBytes = 114688;
static_assert(gG + 4 * kBox <= gTab && gG % 1024 == 0 && 32 * PS * 4 <= kTabs * 512 && gL + CH * LS * 4 <= gG && gGl + 512 <= kGroupBytes && kGroupBytes % 1024 == 0, "group map");
static_assert(kGroups * kGroupBytes <= oCtl, "two groups must fit below the block's control words");
constexpr uint32_t gcL = 0, gcM = 64, gcW = 0, gcU = 64, kGroupCols = 128;

// prefill_one_kernel: one group's area, the slot (its U's place takes the outputs when U is consumed), sums of the norm, barriers.
enum : int { o1Full = 0, o1Free, o1WS, o1S16, o1SDec, o1D, o1SNew, o1O, o1OFree, o1OutFull, o1OutEmpty, o1Gate, kOneBars };
constexpr int oSlotOne = kGroupBytes, oRedOne = oSlotOne + kSlotBytes, oBarsOne = oRedOne + 4 * CH * 4, oCtlOne = oBarsOne + (kOneBars + 1) / 2 * 16, kSmemOne = oCtlOne + 16;
static_assert(oSlotOne % 1024 == 0 && wU == 0 && kSmemOne <= 232448, "shared memory of the single-pass kernel");

// LAYER: the items' inputs are in their slots (kda_internal.h), which the results then replace.  G = 0 or 1, a runtime value: both groups run the same instructions (one copy of this code in the instruction cache).
// ONE: the items are the chunks of the block's own chain, one after another, and the "slot" lies in the block's shared memory (prefill_one_kernel).
template <bool LAYER, bool FUSED, bool WALK_U, bool ONE = false>
__device__ __forceinline__ void intra_group(const SpParams& p, unsigned char* smem, const uint32_t tm_block, const WaitCtx& ctx, const int G) {
    // The issue loops stay loops in the layer form's instance and are unrolled in the core form's, whichever branch an item takes: 4 x 2,048
    // rows of the layer form 972 -> 944 us as loops; the core form's 8,192 rows in 8 sequences 462 both ways with mild gates, 548 and 555 with
    // strong ones, 32,768 rows in one sequence 1,968 and 1,995, 2,138 and 2,207.
    constexpr int kIssue = LAYER ? 1 : 8;
    const int BAR = 2 + G;
    unsigned char* gs = smem + G * kGroupBytes;
    const uint32_t tm = tm_block + G * kGroupCols;
    uint64_t* bar_raw = reinterpret_cast<uint64_t*>(gs + gBars);
    uint64_t* bar_mma = bar_raw + 1;
    uint64_t* bar_lm = bar_raw + 2;  // the eight products of L^T and M^T: eight issuing threads arrive
    uint64_t *bar_free = bar_raw + 3, *bar_g = bar_raw + 4, *bar_gfree = bar_raw + 5;
    volatile int* item_slot = reinterpret_cast<volatile int*>(gs + gItem);
    float* betas = reinterpret_cast<float*>(gs + gBeta);
    const int gt = threadIdx.x - G * kGroupThreads, gw = gt >> 5, lane = gt & 31;
    const int quad = gw & 3, cg = gw >> 2;  // a warp reaches tensor-memory lanes 32 * (warp % 4)..; cg picks a half of the columns
    auto group_sync = [&]() { named_bar_sync(BAR, kGroupThreads); };
    auto publish = [&]() {
        fence_proxy_async_smem();
        tc::fence_before_sync();
        group_sync();
        tc::fence_after_sync();
    };
    auto mma_issue = [&](uint64_t* bar, auto&& issue) {  // by one lane of the group's first warp, the warp converged
        if (gw == 0) {
            const uint32_t leader = tc::elect_one();
            issue(leader);
            tc::mma_commit_if(leader, bar);
            if (leader) atomicAdd(const_cast<uint32_t*>(ctx.progress), 1u);
            __syncwarp();
        }
    };
    uint32_t raw_phase = 0, mma_phase = 0, lm_phase = 0;
    // Fused launches count finished items.  The fence has to wait for the group's last stores, so an item is counted during the next
    // one's last products, when they have long landed.
    int unreported = -1;
    auto report = [&]() {
        if (FUSED && unreported >= 0 && gt == kGroupThreads - 1) {
            __threadfence();
            atomicAdd(p.sets + p.ctr * kTailSet + kTailDone + unreported, 1u);
        }
        unreported = -1;
    };
    auto mma_wait = [&](uint64_t* bar, uint32_t& phase) -> bool {
        if (!mbar_wait(bar, phase, ctx, kStatusWaitPrefill)) return false;
        phase ^= 1u;
        tc::fence_after_sync();
        return true;
    };

    for (;;) {
        if (!mbar_wait(bar_g, raw_phase, ctx, kStatusWaitPrefill)) break;
        const int item = item_slot[0], live = item_slot[1];  // (the next item's from when L and M are formed)
        if (item < 0) break;
        const Item at_item = ONE ? Item{0, item, 0} : item_of<FUSED>(p, item);
        unsigned char* slot = ONE ? smem + oSlotOne : slot_of(p.ws_intra, p.seg_chunks, at_item.chain, at_item.jj);
        uint64_t* one = reinterpret_cast<uint64_t*>(smem + oBarsOne);

        bool mild;
        // ---- 1. per key channel: the cumulative log decay; a = exp(G - Gm), every row relative to the middle row of its block of
        // 16, left in the staging boxes in place of g; then the per-block factor tables.  Thread (part, d): rows 32 part ..
        // 32 part + 31 of channel d, i.e. row blocks 2 part and 2 part + 1 (a needs nothing from the other half).
        {
            const int part = gt >> 7, d = gt & 127;
            // Row r of this thread's channel: box d / 32, piece (d % 32) / 4 swizzled by r & 7, float d % 4.
            unsigned char* col = gs + gG + (d >> 5) * kBox + part * 32 * 128 + (d & 3) * 4;
            const int pc = (d >> 2) & 7;
            float* tmp = reinterpret_cast<float*>(gs + gKb);  // totals [2][128], middles [4][128]; for strong decays, from a half's first middle to its second and on to its end [2][2][128]: the Kgb tile is not in use yet
            float run[32], acc = 0.0f;
            bool strong = false;
#pragma unroll
            for (int r = 0; r < 32; ++r) {
                if (!LAYER && r == 9) strong = acc < kStrong;
                if ((r & 15) == 9 || r == 16) acc = strong ? 0.0f : acc;
                acc = fmaf(*reinterpret_cast<const float*>(col + r * 128 + ((pc ^ (r & 7)) << 4)), kLog2e, acc);  // in powers of two from here on
                run[r] = acc;
            }
            const float mid0 = strong ? 0.0f : run[8], mid1 = strong ? 0.0f : run[24];
            const float upto = (run[8] + run[15]) + run[24], to_mid1 = strong ? upto : run[24];
            acc = strong ? upto + run[31] : acc;
            if (!LAYER) {
                tmp[(6 + 2 * part) * 128 + d] = run[15] + run[24];
                tmp[(7 + 2 * part) * 128 + d] = run[31];
            }
            tmp[part * 128 + d] = acc;
            tmp[(2 + 2 * part) * 128 + d] = run[8];
            tmp[(3 + 2 * part) * 128 + d] = to_mid1;
            float amax = 0.0f;
#pragma unroll
            for (int r = 0; r < 32; ++r) {
                const float av = ex2_ftz(max_nan(run[r] - ((r & 15) <= 8 ? run[(r & 16) | 8] : r < 16 ? mid0 : mid1), -126.0f));  // never 0: its reciprocal is taken
                amax = fmaxf(amax, av);
                *reinterpret_cast<float*>(col + r * 128 + ((pc ^ (r & 7)) << 4)) = av;
            }
            // Eight rows of decay must stay below e^85: per-row log decays below about -10.6 (or positive ones) do not.  (Behind the
            // middle the factors stop at 2^-126; a block's last row is the first to.)
            if (!(amax < 1e37f) || run[15] - mid0 < -126.0f || run[31] - mid1 < -126.0f) atomicCAS(p.status, 0, kStatusPrefillRange);
            group_sync();
            const float base1 = tmp[d];
            const float gm0 = tmp[2 * 128 + d], gm1 = tmp[3 * 128 + d], gm2 = base1 + tmp[4 * 128 + d], gm3 = base1 + tmp[5 * 128 + d];
            const float gl = base1 + tmp[128 + d];
            // (Denormals are wanted here: sixteen rows at the gate's bound decay by e^-93, and their factor meets others of e^+40 and e^+46.)
            float* tab = reinterpret_cast<float*>(gs + gTab) + d;
            if (part == 0) {
                tab[(tE0 + 0) * 128] = ex2_approx(gm0); tab[(tE0 + 1) * 128] = ex2_approx(gm1); tab[(tE0 + 2) * 128] = ex2_approx(gm2); tab[(tE0 + 3) * 128] = ex2_approx(gm3);
                tab[(tEL + 0) * 128] = ex2_approx(gl - gm0); tab[(tEL + 1) * 128] = ex2_approx(gl - gm1);
                tab[(tEL + 2) * 128] = ex2_approx(gl - gm2); tab[(tEL + 3) * 128] = ex2_approx(gl - gm3);
            } else {
                tab[(tF + 0) * 128] = ex2_approx(gm1 - gm0);
                tab[(tF + 1) * 128] = ex2_approx(gm2 - gm0); tab[(tF + 2) * 128] = ex2_approx(gm2 - gm1);
                tab[(tF + 3) * 128] = ex2_approx(gm3 - gm0); tab[(tF + 4) * 128] = ex2_approx(gm3 - gm1); tab[(tF + 5) * 128] = ex2_approx(gm3 - gm2);
                const float egl = ex2_approx(gl);
                if (!ONE) reinterpret_cast<float*>(slot + wEgl)[d] = egl;
                reinterpret_cast<float*>(gs + gGl)[d] = egl;
            }
            mild = gl > -60.0f * kLog2e;
        }
        // A chunk whose whole decay stays above e^-60 in every channel needs no block-wise references: exp(G) and exp(-G) from
        // the chunk's start are both representable with room for small q and k, one column-side tile serves every row, and L^T,
        // M^T are one product each.  The group decides together (the barrier carries the vote); the choice depends on the chunk's
        // own gates only, so it is the same however the call is batched or cut into passes.
        const bool narrow = named_bar_all(BAR, kGroupThreads, mild);

        // ---- 2., 3. operand tiles -------------------------------------------------------------------------------------------------
        if (ONE && !mbar_wait(one + o1Free, (uint32_t)(item + 1) & 1u, ctx, kStatusWaitPrefill)) break;  // the walk is through with the chunk before
        const float* tabs = reinterpret_cast<const float*>(gs + gTab);
        float a[32];
        // The block-wise form's share of a thread: a row of blocks J and 3 - J, sixteen channels each, so that every warp makes as many
        // column-side pieces (3 - J a piece; with one row of 32 channels a thread, half of the warps made three times the others').
        auto block = [&](int t) { return t < 2 ? gw & 1 : 3 - (gw & 1); };
        auto row = [&](int t) { return block(t) * 16 + (lane & 15); };
        auto piece = [&](int t) { return (gw >> 1) * 4 + (lane >> 4) * 2 + (t & 1); };
        if (narrow) {
            // One reference (the chunk's start): Kg = K exp(G) (over K) is the row side of L and the operand of W, Kinv = K exp(-G)
            // (in Kgb's place) the one column-side tile, Kdec = Kinv exp(G_last) as bf16 hi + lo out to the workspace, Qg = Q exp(G) (over Q and
            // out) the row side of M.  All from one read of a, in a loop that stays a loop: the group's instructions are more than
            // the cache next to the warps holds.
            if (!mbar_wait(bar_raw, raw_phase, ctx, kStatusWaitPrefill)) break;
            raw_phase ^= 1u;
            const int r = gt & 63, cq = gt >> 6, J = r >> 4;
#pragma unroll 1
            for (int c = cq * 4; c < cq * 4 + 4; ++c) {
                const uint4 k8 = *reinterpret_cast<const uint4*>(gs + gK + box_piece(r, c)), q8 = *reinterpret_cast<const uint4*>(gs + gQ + box_piece(r, c));
                const float4 aa = *reinterpret_cast<const float4*>(gs + gG + box_piece(r, 2 * c)), ab = *reinterpret_cast<const float4*>(gs + gG + box_piece(r, 2 * c + 1));
                const float4 e0a = *reinterpret_cast<const float4*>(tabs + (tE0 + J) * 128 + c * 8), e0b = *reinterpret_cast<const float4*>(tabs + (tE0 + J) * 128 + c * 8 + 4);
                const float4 gla = *reinterpret_cast<const float4*>(gs + gGl + c * 32), glb = *reinterpret_cast<const float4*>(gs + gGl + c * 32 + 16);
                const float2 A[4] = {{aa.x, aa.y}, {aa.z, aa.w}, {ab.x, ab.y}, {ab.z, ab.w}};
                const float2 E0[4] = {{e0a.x, e0a.y}, {e0a.z, e0a.w}, {e0b.x, e0b.y}, {e0b.z, e0b.w}};
                const float2 GL[4] = {{gla.x, gla.y}, {gla.z, gla.w}, {glb.x, glb.y}, {glb.z, glb.w}};
                const uint32_t kw[4] = {k8.x, k8.y, k8.z, k8.w}, qw[4] = {q8.x, q8.y, q8.z, q8.w};
                uint32_t kg[4], ki[4], dh[4], dl[4], qg[4];
#pragma unroll
                for (int u2 = 0; u2 < 4; ++u2) {
                    const float2 kf = widen2<LAYER>(kw[u2]), e = mul2(A[u2], E0[u2]);
                    const float2 v_kg = mul2(kf, e), v_ki = mul2(kf, {rcp_approx(e.x), rcp_approx(e.y)}), v_kd = mul2(v_ki, GL[u2]), v_qg = mul2(widen2<LAYER>(qw[u2]), e);
                    kg[u2] = tc::bf16x2(v_kg.x, v_kg.y);
                    ki[u2] = tc::bf16x2(v_ki.x, v_ki.y);
                    qg[u2] = tc::bf16x2(v_qg.x, v_qg.y);
                    tc::split_bf16x2(v_kd.x, v_kd.y, dh[u2], dl[u2]);
                }
                *reinterpret_cast<uint4*>(gs + gK + box_piece(r, c)) = make_uint4(kg[0], kg[1], kg[2], kg[3]);
                *reinterpret_cast<uint4*>(gs + gKb + box_piece(r, c)) = make_uint4(ki[0], ki[1], ki[2], ki[3]);
                *reinterpret_cast<uint4*>(gs + gQ + box_piece(r, c)) = make_uint4(qg[0], qg[1], qg[2], qg[3]);
                *reinterpret_cast<uint4*>(cell(slot + wKdHi, CH, c, r)) = make_uint4(dh[0], dh[1], dh[2], dh[3]);
                *reinterpret_cast<uint4*>(cell(slot + wKdLo, CH, c, r)) = make_uint4(dl[0], dl[1], dl[2], dl[3]);
                *reinterpret_cast<uint4*>(cell(slot + wQg, CH, c, r)) = make_uint4(qg[0], qg[1], qg[2], qg[3]);
            }
        } else {
            if constexpr (!LAYER) {  // the factors between two rows once more (kStrong)
                int thread = threadIdx.x - G * kGroupThreads;
                asm volatile("" : "+r"(thread));  // formed anew: kept from the sums on it costs registers all the way (with the norm, 1,000 rows 131.7 -> 136.1 us)
                const int part = thread >> 7, d = thread & 127;
                const float* tmp = reinterpret_cast<const float*>(gs + gKb) + d;
                float* tab = reinterpret_cast<float*>(gs + gTab) + d;
                const float end0 = tmp[0], end1 = tmp[128], m0 = tmp[2 * 128], m1 = tmp[3 * 128], m2 = tmp[4 * 128], m3 = tmp[5 * 128];
                const bool s0 = m0 < kStrong, s1 = m2 < kStrong;
                const float b01 = s0 ? tmp[6 * 128] : m1 - m0, b23 = s1 ? tmp[8 * 128] : m3 - m2;
                const float r1 = s0 ? tmp[7 * 128] : end0 - m1, r3 = s1 ? tmp[9 * 128] : end1 - m3, r0 = b01 + r1, r2 = b23 + r3;
                if (part == 0) {
                    tab[(tEL + 0) * 128] = ex2_approx(r0 + end1); tab[(tEL + 1) * 128] = ex2_approx(r1 + end1); tab[(tEL + 2) * 128] = ex2_approx(r2); tab[(tEL + 3) * 128] = ex2_approx(r3);
                } else {
                    tab[(tF + 0) * 128] = ex2_approx(b01);
                    tab[(tF + 1) * 128] = ex2_approx(r0 + m2); tab[(tF + 2) * 128] = ex2_approx(r1 + m2);
                    tab[(tF + 3) * 128] = ex2_approx(r0 + m3); tab[(tF + 4) * 128] = ex2_approx(r1 + m3); tab[(tF + 5) * 128] = ex2_approx(b23);
                }
            }
            // a into registers: the column-side tiles go over it.  Then the tiles made from k: row side Kgb = K a; Kg = K exp(G)
            // (over K) for W; Kdec = K exp(G_last - G) as bf16 hi + lo out to the workspace; column sides K exp(Gm_I - G) into the
            // tiles I >= J.
#pragma unroll
            for (int t = 0; t < 4; ++t)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 x = *reinterpret_cast<const float4*>(gs + gG + box_piece(row(t), 2 * piece(t) + h));
                    a[t * 8 + 4 * h + 0] = x.x; a[t * 8 + 4 * h + 1] = x.y; a[t * 8 + 4 * h + 2] = x.z; a[t * 8 + 4 * h + 3] = x.w;
                }
            group_sync();  // nobody reads the staged a (or the scan's scratch) any more: the tiles may go over them
            if (!mbar_wait(bar_raw, raw_phase, ctx, kStatusWaitPrefill)) break;
            raw_phase ^= 1u;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int c = piece(t), J = block(t), r = row(t);
                const uint4 k8 = *reinterpret_cast<const uint4*>(gs + gK + box_piece(r, c));
                const float4 e0a = *reinterpret_cast<const float4*>(tabs + (tE0 + J) * 128 + c * 8), e0b = *reinterpret_cast<const float4*>(tabs + (tE0 + J) * 128 + c * 8 + 4);
                const float4 ela = *reinterpret_cast<const float4*>(tabs + (tEL + J) * 128 + c * 8), elb = *reinterpret_cast<const float4*>(tabs + (tEL + J) * 128 + c * 8 + 4);
                const float2 E0[4] = {{e0a.x, e0a.y}, {e0a.z, e0a.w}, {e0b.x, e0b.y}, {e0b.z, e0b.w}};
                const float2 EL[4] = {{ela.x, ela.y}, {ela.z, ela.w}, {elb.x, elb.y}, {elb.z, elb.w}};
                const uint32_t kw[4] = {k8.x, k8.y, k8.z, k8.w};
                uint32_t kg[4], kgb[4], kcd[4], dh[4], dl[4];
                float2 kc[4];  // K exp(Gm_J - G): the column side inside the row's own block
#pragma unroll
                for (int u2 = 0; u2 < 4; ++u2) {
                    const float2 kf = widen2<LAYER>(kw[u2]), av = {a[t * 8 + 2 * u2], a[t * 8 + 2 * u2 + 1]};
                    const float2 v_kgb = mul2(kf, av), v_kg = mul2(kf, mul2(av, E0[u2]));
                    kc[u2] = mul2(kf, {rcp_approx(av.x), rcp_approx(av.y)});
                    const float2 v_kd = mul2(kc[u2], EL[u2]);
                    kg[u2] = tc::bf16x2(v_kg.x, v_kg.y);
                    kgb[u2] = tc::bf16x2(v_kgb.x, v_kgb.y);
                    kcd[u2] = tc::bf16x2(kc[u2].x, kc[u2].y);
                    tc::split_bf16x2(v_kd.x, v_kd.y, dh[u2], dl[u2]);
                }
                *reinterpret_cast<uint4*>(gs + gK + box_piece(r, c)) = make_uint4(kg[0], kg[1], kg[2], kg[3]);
                *reinterpret_cast<uint4*>(gs + gKb + box_piece(r, c)) = make_uint4(kgb[0], kgb[1], kgb[2], kgb[3]);
                *reinterpret_cast<uint4*>(cell(slot + wKdHi, CH, c, r)) = make_uint4(dh[0], dh[1], dh[2], dh[3]);
                *reinterpret_cast<uint4*>(cell(slot + wKdLo, CH, c, r)) = make_uint4(dl[0], dl[1], dl[2], dl[3]);
                *reinterpret_cast<uint4*>(gs + gKc + kc_piece(J, r, c)) = make_uint4(kcd[0], kcd[1], kcd[2], kcd[3]);
                for (int I = J + 1; I < 4; ++I) {  // the later row blocks see this row through exp(Gm_I - Gm_J) <= 1
                    const float* f = tabs + (tF + I * (I - 1) / 2 + J) * 128 + c * 8;
                    const float4 fa = *reinterpret_cast<const float4*>(f), fb = *reinterpret_cast<const float4*>(f + 4);
                    const float2 F[4] = {{fa.x, fa.y}, {fa.z, fa.w}, {fb.x, fb.y}, {fb.z, fb.w}};
                    uint32_t kcf[4];
#pragma unroll
                    for (int u2 = 0; u2 < 4; ++u2) {
                        const float2 x = mul2(kc[u2], F[u2]);
                        kcf[u2] = tc::bf16x2(x.x, x.y);
                    }
                    *reinterpret_cast<uint4*>(gs + gKc + kc_piece(I, r, c)) = make_uint4(kcf[0], kcf[1], kcf[2], kcf[3]);
                }
            }
        }
        publish();
        // ---- 3a. L^T, one block column of 16 rows i a warp: [64 j x 16 i] = column side (tile I) x row side (block I)^T.  The
        // eight warps issue the eight small products of L^T and M^T (one lane each), so none of them issues for long; each
        // commits to the same barrier, which completes when all eight have.
        if (gw < 4) {
            const uint32_t leader = tc::elect_one();
            if (narrow) {  // one product, all 64 rows i at once, row side Kg (a commit with nothing pending arrives at once)
                constexpr uint32_t id64 = tc::idesc_bf16(64, 64, 0, 0, 0);
                if (gw == 0)
#pragma unroll kIssue
                    for (int k0 = 0; k0 < DK; k0 += 16)
                        tc::mma_bf16_if(leader, tm + gcL, tc::desc_sw128_kmajor(gs + gKb, CH, k0), tc::desc_sw128_kmajor(gs + gK, CH, k0), id64, k0 > 0);
            } else {
                constexpr uint32_t id = tc::idesc_bf16(64, 16, 0, 0, 0);
                const int I = gw;
                const unsigned char* kct = gs + gKc + kc_tile(I);
#pragma unroll kIssue
                for (int k0 = 0; k0 < DK; k0 += 16)
                    tc::mma_bf16_if(leader, tm + gcL + 16 * I, tc::desc_sw128_kmajor(kct, 16 * (I + 1), k0), tc::desc_sw128_kmajor(gs + gKb + I * 2048, CH, k0), id, k0 > 0);
            }
            tc::mma_commit_if(leader, bar_lm);
            if (leader) atomicAdd(const_cast<uint32_t*>(ctx.progress), 1u);
            __syncwarp();
        }
        // ---- 3b. the block-wise form's tiles made from q, while L^T runs: row side Qgb = Q a (over Q); Qg = Q exp(G) out to the workspace
        if (!narrow) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int c = piece(t), J = block(t), r = row(t);
                const uint4 q8 = *reinterpret_cast<const uint4*>(gs + gQ + box_piece(r, c));
                const uint32_t qw[4] = {q8.x, q8.y, q8.z, q8.w};
                uint32_t qg[4], qgb[4];
                const float4 e0a = *reinterpret_cast<const float4*>(tabs + (tE0 + J) * 128 + c * 8), e0b = *reinterpret_cast<const float4*>(tabs + (tE0 + J) * 128 + c * 8 + 4);
                const float2 E0[4] = {{e0a.x, e0a.y}, {e0a.z, e0a.w}, {e0b.x, e0b.y}, {e0b.z, e0b.w}};
#pragma unroll
                for (int u2 = 0; u2 < 4; ++u2) {
                    const float2 qf = widen2<LAYER>(qw[u2]), av = {a[t * 8 + 2 * u2], a[t * 8 + 2 * u2 + 1]}, x = mul2(qf, av), y = mul2(qf, mul2(av, E0[u2]));
                    qgb[u2] = tc::bf16x2(x.x, x.y);
                    qg[u2] = tc::bf16x2(y.x, y.y);
                }
                *reinterpret_cast<uint4*>(gs + gQ + box_piece(r, c)) = make_uint4(qgb[0], qgb[1], qgb[2], qgb[3]);
                *reinterpret_cast<uint4*>(cell(slot + wQg, CH, c, r)) = make_uint4(qg[0], qg[1], qg[2], qg[3]);
            }
            publish();
        }
        // ---- 3c. M^T the same way, by the other four warps ------------------------------------------------------------------------
        if (gw >= 4) {
            const uint32_t leader = tc::elect_one();
            if (narrow) {
                constexpr uint32_t id64 = tc::idesc_bf16(64, 64, 0, 0, 0);
                if (gw == 4)
#pragma unroll kIssue
                    for (int k0 = 0; k0 < DK; k0 += 16)
                        tc::mma_bf16_if(leader, tm + gcM, tc::desc_sw128_kmajor(gs + gKb, CH, k0), tc::desc_sw128_kmajor(gs + gQ, CH, k0), id64, k0 > 0);
            } else {
                constexpr uint32_t id = tc::idesc_bf16(64, 16, 0, 0, 0);
                const int I = gw - 4;
                const unsigned char* kct = gs + gKc + kc_tile(I);
#pragma unroll kIssue
                for (int k0 = 0; k0 < DK; k0 += 16)
                    tc::mma_bf16_if(leader, tm + gcM + 16 * I, tc::desc_sw128_kmajor(kct, 16 * (I + 1), k0), tc::desc_sw128_kmajor(gs + gQ + I * 2048, CH, k0), id, k0 > 0);
            }
            tc::mma_commit_if(leader, bar_lm);
            if (leader) atomicAdd(const_cast<uint32_t*>(ctx.progress), 1u);
            __syncwarp();
        }
        if (!mma_wait(bar_lm, lm_phase)) break;
        if (gt == 0) mbar_arrive(bar_gfree);  // nothing is left over the log decays' place

        // ---- 4. from L^T and M^T (lane = column j, tensor-memory column = row i): L (FP32, strictly lower, times beta_i) into
        // the scratch; M (lower with the diagonal) out as bf16 cells of eight consecutive rows i, [8 cells][64 columns j] ----------
        {
            // In the fragment layout: columns j and j + 8, rows i = 16 x + 8 g + 2 (lane % 4) and the next.
            const int j = quad * 16 + (lane >> 2), i0 = 2 * (lane & 3);
            uint32_t f[4][8];
#pragma unroll
            for (int x = 0; x < 4; ++x) tc::tmem_ld_frag(tc::tmem_addr(tm, quad, (cg == 0 ? gcL : gcM) + 16 * x), f[x]);
            tc::tmem_ld_wait();
            if (cg == 0) {  // L stays transposed
                float* Lt = reinterpret_cast<float*>(gs + gL) + j * LS + i0;
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    const float2 b2 = *reinterpret_cast<const float2*>(betas + x * 8 + i0);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int i = x * 8 + i0, jh = j + 8 * h;
                        const float l0 = __uint_as_float(f[x >> 1][4 * (x & 1) + 2 * h]), l1 = __uint_as_float(f[x >> 1][4 * (x & 1) + 2 * h + 1]);
                        *reinterpret_cast<float2*>(Lt + h * 8 * LS + x * 8) = make_float2(i > jh ? b2.x * l0 : 0.0f, i + 1 > jh ? b2.y * l1 : 0.0f);
                    }
                }
            } else {  // four lanes' pairs are a cell
#pragma unroll
                for (int x = 0; x < 8; ++x)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int i = x * 8 + i0, jh = j + 8 * h;
                        const float m0 = __uint_as_float(f[x >> 1][4 * (x & 1) + 2 * h]), m1 = __uint_as_float(f[x >> 1][4 * (x & 1) + 2 * h + 1]);
                        *reinterpret_cast<uint32_t*>(cell(slot + wMm, CH, x, jh) + 2 * i0) = tc::bf16x2(i >= jh ? m0 : 0.0f, i + 1 >= jh ? m1 : 0.0f);
                    }
            }
        }
        tc::fence_before_sync();
        group_sync();

        // ---- 5. T = (I + L)^-1 in FP32, T' = T diag(beta) as bf16 hi + lo cells (over L, dead by then) -----------------------
        {
            const float* Lm = reinterpret_cast<const float*>(gs + gL);
            float* Tm = reinterpret_cast<float*>(gs + gT);
            float* Pm = reinterpret_cast<float*>(gs + gP);
            invert<kGroupThreads>(Lm, Tm, Pm, gt, BAR);
            const int i = gt & 63, cq = gt >> 6;
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                const int c = cq + cc * 4;
                uint32_t wh[4], wl[4];
#pragma unroll
                for (int j2 = 0; j2 < 2; ++j2) {
                    const float4 t4 = *reinterpret_cast<const float4*>(Tm + i * LS + c * 8 + 4 * j2), b4 = *reinterpret_cast<const float4*>(betas + c * 8 + 4 * j2);
                    tc::split_bf16x2(t4.x * b4.x, t4.y * b4.y, wh[2 * j2], wl[2 * j2]);
                    tc::split_bf16x2(t4.z * b4.z, t4.w * b4.w, wh[2 * j2 + 1], wl[2 * j2 + 1]);
                }
                *reinterpret_cast<uint4*>(gs + gTp + box_piece(i, c)) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
                if constexpr (WALK_U) {
                    if (cc == 0) {
                        *reinterpret_cast<uint4*>(cell(slot + wTp, CH, c, i)) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
                        *reinterpret_cast<uint4*>(cell(slot + wTp + kBox / 2, CH, c, i)) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
                    } else if (i >= CH / 2) {  // (above it there are only zeros)
                        *reinterpret_cast<uint4*>(cell(slot + wTp + kBox, CH / 2, c - 4, i - CH / 2)) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
                        *reinterpret_cast<uint4*>(cell(slot + wTp + kBox + kBox / 4, CH / 2, c - 4, i - CH / 2)) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
                    }
                } else {
                    *reinterpret_cast<uint4*>(gs + gTp + kBox + box_piece(i, c)) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
                }
            }
        }
        publish();

        // ---- 6. W^T = Kg^T T'^T (bf16 T'), U^T = V^T T'^T (T' hi + lo): 128 channels x 64 rows (as 64 rows x 128 channels the
        // products take the same instructions at half the rate) ------------------------------------------------------------
        mma_issue(bar_mma, [&](uint32_t leader) {
            constexpr uint32_t id = tc::idesc_bf16(128, 64, 1, 0, 0);
#pragma unroll kIssue
            for (int k0 = 0; k0 < CH; k0 += 16)
                tc::mma_bf16_if(leader, tm + gcW, tc::desc_sw128_mnmajor(gs + gK, CH, k0), tc::desc_sw128_kmajor(gs + gTp, CH, k0), id, k0 > 0);
            if constexpr (!WALK_U) {
#pragma unroll kIssue
                for (int k0 = 0; k0 < CH; k0 += 16)
                    tc::mma_bf16_if(leader, tm + gcU, tc::desc_sw128_mnmajor(gs + gV, CH, k0), tc::desc_sw128_kmajor(gs + gTp, CH, k0), id, k0 > 0);
#pragma unroll kIssue
                for (int k0 = 0; k0 < CH; k0 += 16)
                    tc::mma_bf16_if(leader, tm + gcU, tc::desc_sw128_mnmajor(gs + gV, CH, k0), tc::desc_sw128_kmajor(gs + gTp + kBox, CH, k0), id, true);
            }
        });
        report();
        // A walk that forms U reads V itself, a partial chunk's from the slot: zero past the sequence's end (the layer form's live rows lie there).
        if (WALK_U && live < CH) {
            const int h = at_item.chain % p.H;
            const long long row0 = LAYER ? 0 : p.cu[at_item.chain / p.H] + (long long)(p.intra_chunk0 + at_item.jj) * CH;
            uint4 v8[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int r = t * 16 + (gt >> 4);
                v8[t] = !LAYER && r < live ? *reinterpret_cast<const uint4*>(p.v + ((row0 + r) * p.H + h) * DK + (gt & 15) * 8) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int r = t * 16 + (gt >> 4);
                if (!LAYER || r >= live) *reinterpret_cast<uint4*>(slot + wV + box_piece(r, gt & 15)) = v8[t];
            }
        }
        const float egl_here = ONE && gt < DK ? reinterpret_cast<const float*>(gs + gGl)[gt] : 0.0f;
        if (!mma_wait(bar_mma, mma_phase)) break;
        // Nothing of this item is left in the group's shared memory: the loader may bring the next item in.
        if (gt == 0) mbar_arrive(bar_free);

        // ---- 7. W as bf16 cells and U as FP32 cells, from tensor memory (lane = channel, column = row) to the workspace ----------
        {
            const int ch = quad * 32 + lane;
            uint32_t r[32];
            tc::tmem_ld32(tc::tmem_addr(tm, quad, gcW + cg * 32), r);
            tc::tmem_ld_wait();
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) *reinterpret_cast<uint4*>(cell(slot + wW, DK, cg * 4 + cc, ch)) = pack8(r + cc * 8);
            if constexpr (!WALK_U) {
                tc::tmem_ld32(tc::tmem_addr(tm, quad, gcU + cg * 32), r);
                tc::tmem_ld_wait();
                if (ONE && !mbar_wait(one + o1OutEmpty, (uint32_t)(item + 1) & 1u, ctx, kStatusWaitPrefill)) break;  // its outputs have left U's place
#pragma unroll
                for (int j2 = 0; j2 < 8; ++j2)
                    *reinterpret_cast<uint4*>(slot + wU + u_cell(cg * 8 + j2, ch)) = make_uint4(r[j2 * 4], r[j2 * 4 + 1], r[j2 * 4 + 2], r[j2 * 4 + 3]);
            }
        }
        if (ONE) {
            if (gt < DK) reinterpret_cast<float*>(slot + wEgl)[gt] = egl_here;
            fence_proxy_async_smem();
        }
        if (FUSED) fence_proxy_async_global();  // another block's bulk copies read the slot
        tc::fence_before_sync();
        group_sync();
        tc::fence_after_sync();
        if (ONE && gt == 0) mbar_arrive(one + o1Full);
        unreported = at_item.group;
    }
    report();
}

// 16 bytes on their way from global to shared memory, or 16 zero bytes (nothing is read then).
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src, bool read) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem_dst)), "l"(gmem_src), "r"(read ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The loader warp of group G: takes items off the counter and brings each one's rows into the group's staging.  A full
// chunk arrives by eight or ten tiled tensor copies issued by one lane; a sequence's last, partial chunk by the warp's own
// 16-byte copies (rows past the sequence's end are not read, they become zero), so no copy ever reaches
// past the rows the caller's metadata names.  They are asynchronous, all in flight at once: as loads and stores, a row's after
// the other's, they were 8 to 12 us of a launch (33 rows x 64 heads by the chunked layer prefill: 59 us, 64 rows 52).
template <bool LAYER, bool FUSED, bool WALK_U, bool ONE = false>
__device__ __forceinline__ void intra_loader(const SpParams& p, unsigned char* smem, const WaitCtx& ctx, const int G, const int one_chain = 0) {
    unsigned char* gs = smem + G * kGroupBytes;
    uint64_t* bar_raw = reinterpret_cast<uint64_t*>(gs + gBars);
    uint64_t *bar_free = bar_raw + 3, *bar_g = bar_raw + 4, *bar_gfree = bar_raw + 5;
    volatile int* item_slot = reinterpret_cast<volatile int*>(gs + gItem);
    float* betas = reinterpret_cast<float*>(gs + gBeta);
    const int lane = threadIdx.x & 31;
    const int H = p.H, chains = p.batch * H;
    const long long items = (long long)chains * p.seg_chunks;  // item = jj * chains + chain: chunk-major
    uint32_t free_phase = 0;
    for (int it = 0;;) {
        long long item = ONE ? it : 0;
        if (!ONE && lane == 0) {
            unsigned int* taken = FUSED ? p.sets + p.ctr * kTailSet : p.counters + p.ctr;
            // (Only when every block has begun: those that stay run then, and a chain whose items they have may be waited for.)
            if (FUSED && (int)blockIdx.x < p.early_blocks && *reinterpret_cast<volatile unsigned int*>(taken) >= p.early_from &&
                *reinterpret_cast<volatile unsigned int*>(taken + kTailBegun) == gridDim.x)
                item = items;
            else
                item = atomicAdd(taken, 1u);
        }
        item = __shfl_sync(0xffffffffu, item, 0);
        bool last = !ONE && item >= items;
        int h = 0, n = 0;
        long long gr0 = 0;
        const unsigned char* in = nullptr;
        if (!last) {
            const Item at = ONE ? Item{one_chain, (int)item, 0} : item_of<FUSED>(p, (int)item);
            const int j = p.intra_chunk0 + at.jj, b = at.chain / H;
            h = at.chain % H;
            const int r0 = p.cu[b], T = p.cu[b + 1] - r0;
            if (ONE && (long long)j * CH >= T) {
                last = true;
            } else if ((long long)j * CH >= T) {  // the sequence has no such chunk
                if (FUSED && lane == 0) atomicAdd(p.sets + p.ctr * kTailSet + kTailDone + at.group, 1u);
                continue;
            }
            gr0 = (long long)r0 + (long long)j * CH;
            n = min(CH, T - j * CH);
            if constexpr (LAYER) in = slot_of(p.ws_intra, p.seg_chunks, at.chain, at.jj);
        }
        float b0 = 0.0f, b1 = 0.0f;
        if (lane < n) b0 = LAYER ? reinterpret_cast<const float*>(in + kSlotInBeta)[lane] : p.beta[(gr0 + lane) * H + h];
        if (lane + 32 < n) b1 = LAYER ? reinterpret_cast<const float*>(in + kSlotInBeta)[lane + 32] : p.beta[(gr0 + lane + 32) * H + h];
        if (!LAYER && !last && n == CH && lane == 0 && !(ONE && it == 0)) {  // on their way into L2 while the group is still busy with the item before
            const int row = (int)gr0;
            for (int x = 0; x < 4; ++x) tensor_prefetch_3d(&p.tm_g, x * 32, h, row);
            for (int x = 0; x < 2; ++x) tensor_prefetch_3d(&p.tm_k, x * 64, h, row);
            for (int x = 0; x < 2; ++x) tensor_prefetch_3d(&p.tm_q, x * 64, h, row);
            for (int x = 0; !WALK_U && x < 2; ++x) tensor_prefetch_3d(&p.tm_v, x * 64, h, row);
        }
        const int row = (int)gr0;
        // The log decays, as soon as the item before has formed its L and M; then the other rows, when it is through with its own.
        if (it > 0 && !mbar_wait(bar_gfree, free_phase, ctx, kStatusWaitPrefill)) break;
        if (lane == 0) {
            item_slot[0] = last ? -1 : (int)item;
            item_slot[1] = n;
        }
        if (last) {  // tell the compute warps that there is nothing more
            if (lane == 0) mbar_arrive(bar_g);
            break;
        }
        if (n == CH) {
            if (lane == 0) {
                mbar_arrive_expect_tx(bar_g, 4u * kBox);
                if constexpr (LAYER) bulk_load(gs + gG, in + kSlotInG, 4 * kBox, bar_g);
                else
                    for (int x = 0; x < 4; ++x) tensor_load_3d(gs + gG + x * kBox, &p.tm_g, x * 32, h, row, bar_g);
            }
        } else {
            for (int r = 0; r < CH; ++r) {
                const int live = min(r, n - 1);
                const void* src = LAYER ? (const void*)(in + kSlotInG + box_piece(live, lane)) : (const void*)(p.g + ((gr0 + live) * H + h) * DK + lane * 4);
                cp_async16(gs + gG + box_piece(r, lane), src, r < n);
            }
            cp_async_wait_all();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_g);
        }
        if (it > 0) {
            if (!mbar_wait(bar_free, free_phase, ctx, kStatusWaitPrefill)) break;
            free_phase ^= 1u;
        }
        ++it;
        betas[lane] = b0;
        betas[lane + 32] = b1;
        if (n == CH) {
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_expect_tx(bar_raw, (WALK_U ? 2u : 3u) * kTile);
                if constexpr (LAYER) {
                    bulk_load(gs + gK, in + kSlotInK, kTile, bar_raw);
                    bulk_load(gs + gQ, in + kSlotInQ, kTile, bar_raw);
                } else {
                    for (int x = 0; x < 2; ++x) tensor_load_3d(gs + gK + x * kBox, &p.tm_k, x * 64, h, row, bar_raw);
                    for (int x = 0; x < 2; ++x) tensor_load_3d(gs + gQ + x * kBox, &p.tm_q, x * 64, h, row, bar_raw);
                    for (int x = 0; !WALK_U && x < 2; ++x) tensor_load_3d(gs + gV + x * kBox, &p.tm_v, x * 64, h, row, bar_raw);
                }
            }
        } else {
            for (int r = lane >> 4; r < CH; r += 2) {
                const int c = lane & 15, live = min(r, n - 1), from = box_piece(live, c), to = box_piece(r, c);
                const long long at = ((gr0 + live) * H + h) * DK + c * 8;
                cp_async16(gs + gK + to, LAYER ? (const void*)(in + kSlotInK + from) : (const void*)(p.k + at), r < n);
                cp_async16(gs + gQ + to, LAYER ? (const void*)(in + kSlotInQ + from) : (const void*)(p.q + at), r < n);
                if (!WALK_U) cp_async16(gs + gV + to, p.v + at, r < n);
            }
            cp_async_wait_all();
            if (!WALK_U) fence_proxy_async_smem();  // V is read by the tensor core as it stands
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_raw);
        }
    }
}

template <bool LAYER, bool FUSED, bool WALK_U>
__device__ void intra_role(const SpParams& p, unsigned char* smem, const uint32_t tm) {
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + oCtl);
    const WaitCtx ctx{ctl, ctl + 1, p.status};
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        for (int g = 0; g < kGroups; ++g) {
            uint64_t* b = reinterpret_cast<uint64_t*>(smem + g * kGroupBytes + gBars);
            for (int i = 0; i < kGroupBars; ++i) mbar_init(b + i, i == 2 ? 8 : 1);  // raw, mma, L^T/M^T (eight issuers), free, log decays, their place free
        }
        mbar_init_fence();
    }
    __syncthreads();
    if (warp == kLoaderWarp || warp == kOutWarp) intra_loader<LAYER, FUSED, WALK_U>(p, smem, ctx, warp == kLoaderWarp ? 0 : 1);
    else if (warp != kMmaWarp) intra_group<LAYER, FUSED, WALK_U>(p, smem, tm, ctx, warp < kGroupThreads / 32 ? 0 : 1);
    tc::fence_before_sync();
    __syncthreads();
}

// =====================================================================================================================
// Pass 2: the state recurrence of one chain over the segment's chunks, from the workspace.
//
// The state lives transposed in tensor memory: lane = value channel, columns = key channels (FP32).  The walk is a chain of
// dependent steps per chunk, so nothing that can wait sits on it and no two roles meet at a block barrier (mbarriers only):
//   all 16 warps     S^T to bf16 pairs, in tensor memory; then, behind the first product, the decayed S^T back
//   MMA warp         (W S)^T = S^T W^T, 128 value channels x 64 rows, which D waits for; then (Qg S)^T, which it does not
//   all 16 warps     D^T = U^T - (W S)^T as bf16 hi + lo pairs, in tensor memory
//   MMA warp         S^T += D^T Kdec (hi hi + lo hi + hi lo), which the next chunk waits for; then O^T = (Qg S)^T + D^T M^T, and
//                    (WALK_U) the next chunk's U^T = V^T T'^T (T' hi + lo)
//   all 16 warps     the outputs of the chunk before, while the state's product runs
// Transposed, every product uses the tensor core's full height, every lane holds results, and the operands that change (S, D)
// are A operands that never leave tensor memory; what comes from the workspace is the B side, so shared memory has room for
// two chunks of it and a load has a whole chunk's time to arrive.
// Measured per chunk at 64 chains: 5,800 cycles with products of 64 rows, S and D through shared memory and block barriers
// around every step; 3,700 to 4,000 so; 3,500 with the single buffer's piece asked into L2 a chunk ahead (8 chains of 1,024 chunks: a whole call is 3,240 a chunk), 4,400
// with a chain on every SM, when the workspace comes at 5.9 TB/s.  With the gated norm 5,400: 16,384 exponentials and
// reciprocals a chunk are 1,000 cycles of the units that do them (before U and D instead of behind D they are as long, and cost registers).
// =====================================================================================================================
// Shared memory: two buffers of [Qg | W] and exp(G_last), two of [M | Kdec hi | Kdec lo], one of U, or T' hi | T' lo | V, each with a full / empty pair.
// Finished output rows (bf16) wait in one of two tiles for the output warp: two boxes of 64 rows x 128 bytes each (value
// channels 0-63, 64-127) in the 128-byte swizzle of box_piece(), which is what the tiled tensor stores read.
constexpr int kQW = 2 * kTile, kMKd = kTile / 2 + 2 * kTile, kOutTile = 2 * kBox;
constexpr int sQW = 0, sMKd = sQW + 2 * kQW, sU = sMKd + 2 * kMKd, sOut = sU + kUBytes, sRed = sOut + 2 * kOutTile, sE = sRed + 2 * 4 * CH * 4;
static_assert(sOut % 1024 == 0 && (sU + kTile) % 1024 == 0 && sE + 2 * 512 <= oCtl, "state role shared memory");
// Tensor memory columns: S^T; its bf16 pairs; (W S)^T; (Qg S)^T and O^T, two accumulators that alternate between chunks; D^T hi, lo; U^T.
constexpr uint32_t tS = 0, tS16 = 128, tWS = 192, tO = 256, tDhi = 384, tDlo = 416, tU = 448;

// The state role's barriers and their arrival counts.  Those of a buffer that alternates between chunks come in pairs, so that
// no barrier can complete a phase while somebody still has to see the one before.
enum : int { bFullQW = 0, bFullMKd = 2, bFullU = 4, bEmptyQW = 5, bEmptyMKd = 7, bEmptyU = 9, bWS = 10, bSNew = 11, bS16 = 12, bSDec = 13, bD = 14, bO = 15, bOFree = 17,
             bOutFull = 19, bOutEmpty = 21, bChainFull = 23, bChainEmpty = 25, bGate = 27, kStateBars = 29 };
__device__ __forceinline__ int state_bar_count(int i, bool walk_u) {
    // one arrival per compute warp, or one in all
    const bool warps = (i == bEmptyU && !walk_u) || i == bS16 || i == bSDec || i == bD || i == bOFree || i == bOFree + 1 || i == bOutFull || i == bOutFull + 1;
    return warps ? kCompute / 32 : i == bChainEmpty || i == bChainEmpty + 1 ? kCompute / 32 + 2 : 1;  // a chain is read by the MMA and the output warp too
}
static_assert(kStateBars * 8 <= oChain - oBarsState && oChain % 16 == 0, "state role barriers");

// Waits until a count in global memory has reached `want`; gives up when it has stood still for the waits' limit.  As long as it rises, the
// block's other warps, which wait for what follows, are told of progress, so that their limit is no shorter.
__device__ __forceinline__ bool count_wait(const unsigned int* at, unsigned want, const WaitCtx& ctx, int code) {
    unsigned seen = 0;
    uint64_t t0 = global_timer_ns();
    for (;;) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(at) : "memory");
        if (v >= want) return true;
        const uint64_t now = global_timer_ns();
        if (v != seen) {
            seen = v;
            t0 = now;
            atomicAdd(const_cast<uint32_t*>(ctx.progress), 1u);
        } else if (now - t0 > ctx.limit_ns) {
            atomicCAS(ctx.status, 0, code);
            return false;
        }
        __nanosleep(100);
    }
}

// What one walk of the state role covers: chunks [ja, jb) of its chain, where the state comes from and goes to, whether
// T'V takes part (not in the walk that yields a segment's transition) and whether outputs are produced.
struct Walk {
    int ja, jb;
    int init;          // 0: the state buffer (state_in for the first chunk of a sequence, else state_out); 1: zero; 2: identity; 3: FP32 `from`
    const float* from;
    int fin;           // where the end state goes: 0 state_out, 1 the FP32 buffer `to`, 2 nowhere
    float* to;
    bool use_u, emit;
};

// What the roles of a block need to know of a chain they walk: `count` chunks from row `row` of the whole batch on, of head h; `rows`
// rows are left of the sequence there.  The loader warp writes it; the others read it from shared memory whenever they want some of it.
struct Chain {
    int count, rows, h, start;  // count < 0: no more chains; start: the sequence begins here
    long long row, s_elem;
};
__device__ __forceinline__ Chain chain_of(const SpParams& p, const Walk& wk, int chain) {
    const int b = chain / p.H, h = chain % p.H, T = p.cu[b + 1] - p.cu[b];
    const int nch = (T + CH - 1) / CH, j0 = min(wk.ja, nch);
    return {max(min(nch, wk.jb) - j0, 0), T - j0 * CH, h, j0 == 0, p.cu[b] + (long long)j0 * CH, p.state_off[b] + (long long)h * DV * DK};
}
// A chain with no chunk in this range: only the first segment has anything to do (an empty sequence copies its state); a scan
// walk always delivers its end state.
__device__ __forceinline__ bool nothing_to_do(const SpParams& p, const Chain& c) {
    return p.scan_pass == 0 && c.count == 0 && !(c.start && p.state_out != p.state_in);
}

// A warp's 32 x 32 piece of the state between tensor memory and a state buffer on 16 bytes (rows of 128 elements).  A thread that moves
// its own row's 32 values touches a line of its own with every 16 bytes (2,000 cycles a state of bf16, 4,000 of FP32); from the fragment
// layout, in which four lanes hold a row's neighbouring columns, two or four lanes trade halves and a row's 64 bytes go at once.
__device__ __forceinline__ uint32_t trade(bool up, uint32_t lo, uint32_t hi, int lanes) { return __shfl_xor_sync(0xffffffffu, up ? lo : hi, lanes); }
__device__ __forceinline__ void state_from_tmem(uint32_t at, float* to, int lane) {  // to: row 0, column 0 of the piece
    const int q = lane & 3;
    const bool odd = q & 1;
    to += (lane >> 2) * DK + (odd ? 6 + 2 * q : 2 * q);
#pragma unroll
    for (int x = 0; x < 4; ++x) {  // sixteen rows (x / 2) and sixteen columns (x % 2)
        uint32_t f[8];
        tc::tmem_ld_frag(at + ((uint32_t)(x >> 1) << 20) + (x & 1) * 16, f);
        tc::tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // eight rows
            const uint32_t r0 = trade(odd, f[2 * h], f[4 + 2 * h], 1), r1 = trade(odd, f[2 * h + 1], f[5 + 2 * h], 1);
            *reinterpret_cast<uint4*>(to + ((x >> 1) * 16 + h * 8) * DK + (x & 1) * 16) = odd ? make_uint4(r0, r1, f[4 + 2 * h], f[5 + 2 * h]) : make_uint4(f[2 * h], f[2 * h + 1], r0, r1);
        }
    }
}
__device__ __forceinline__ void state_to_tmem(uint32_t at, const float* from, int lane) {
    const int q = lane & 3;
    const bool odd = q & 1;
    from += (lane >> 2) * DK + (odd ? 6 + 2 * q : 2 * q);
    uint4 w[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) w[x] = *reinterpret_cast<const uint4*>(from + ((x >> 2) * 16 + (x & 1) * 8) * DK + ((x >> 1) & 1) * 16);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        uint32_t f[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 v = w[2 * x + h];
            const uint32_t r0 = trade(odd, v.x, v.z, 1), r1 = trade(odd, v.y, v.w, 1);
            f[2 * h] = odd ? r0 : v.x; f[2 * h + 1] = odd ? r1 : v.y;
            f[4 + 2 * h] = odd ? v.z : r0; f[5 + 2 * h] = odd ? v.w : r1;
        }
        tc::tmem_st_frag(at + ((uint32_t)(x >> 1) << 20) + (x & 1) * 16, f);
    }
}
__device__ __forceinline__ void state_from_tmem(uint32_t at, uint16_t* to, int lane) {
    const int q = lane & 3;
    const bool odd = q & 1, up = q & 2;
    to += (lane >> 2) * DK + q * 8;
#pragma unroll
    for (int x = 0; x < 2; ++x) {  // sixteen rows
        uint32_t f[2][8];
        tc::tmem_ld_frag(at + ((uint32_t)x << 20), f[0]);
        tc::tmem_ld_frag(at + ((uint32_t)x << 20) + 16, f[1]);
        tc::tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t w[4], pr[2][2];  // w[g]: columns 8 g + 2 q and the next; pr: of g = 2 i + odd, those of lanes (q & 2) and (q & 2) + 1
#pragma unroll
            for (int g = 0; g < 4; ++g) w[g] = tc::bf16x2(__uint_as_float(f[g >> 1][4 * (g & 1) + 2 * h]), __uint_as_float(f[g >> 1][4 * (g & 1) + 2 * h + 1]));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t r = trade(odd, w[2 * i], w[2 * i + 1], 1);
                pr[i][0] = odd ? r : w[2 * i];
                pr[i][1] = odd ? w[2 * i + 1] : r;
            }
            const uint32_t r0 = trade(up, pr[0][0], pr[1][0], 2), r1 = trade(up, pr[0][1], pr[1][1], 2);
            *reinterpret_cast<uint4*>(to + (x * 16 + h * 8) * DK) = up ? make_uint4(r0, r1, pr[1][0], pr[1][1]) : make_uint4(pr[0][0], pr[0][1], r0, r1);
        }
    }
}
__device__ __forceinline__ void state_to_tmem(uint32_t at, const uint16_t* from, int lane) {
    const int q = lane & 3;
    const bool odd = q & 1, up = q & 2;
    from += (lane >> 2) * DK + q * 8;
    uint4 v[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) v[x] = *reinterpret_cast<const uint4*>(from + x * 8 * DK);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        uint32_t f[2][8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 y = v[2 * x + h];
            const uint32_t r0 = trade(up, y.x, y.z, 2), r1 = trade(up, y.y, y.w, 2);
            const uint32_t pr[2][2] = {{up ? r0 : y.x, up ? r1 : y.y}, {up ? y.z : r0, up ? y.w : r1}};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t r = trade(odd, pr[i][0], pr[i][1], 1), w0 = odd ? r : pr[i][0], w1 = odd ? pr[i][1] : r;
                f[i][2 * h] = w0 << 16; f[i][2 * h + 1] = w0 & 0xffff0000u;
                f[i][4 + 2 * h] = w1 << 16; f[i][5 + 2 * h] = w1 & 0xffff0000u;
            }
        }
        tc::tmem_st_frag(at + ((uint32_t)x << 20), f[0]);
        tc::tmem_st_frag(at + ((uint32_t)x << 20) + 16, f[1]);
    }
}

// The gated RMSNorm of sixteen output rows from i0 on by four warps, which have 32 channels each and meet at barrier `bar`; red: their sums, [4][64].  y2[g][q]:
// rows fi + 8 g and the next (fi = i0 + 2 (lane % 4)) of channel fv + 8 q as bf16, gt the gate's values alike, which `fetch` may bring behind the barrier.
// False on all four when one of them comes without `ok`.  The sigmoid is formed sixteenfold and a row's factor a sixteenth: below -87.3 the gate's sigmoid is not
// a normal number, which the reciprocal would flush, but leaves outputs that bf16 holds.
template <typename Fetch>
__device__ __forceinline__ bool gated_rows(float* red, float eps, int quad, int lane, int i0, const float (&nw)[4], uint32_t (&gt)[2][4], uint32_t (&y2)[2][4], int bar, bool ok, Fetch&& fetch) {
    float sq[4];  // [2 g + e]
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        float2 s2 = {0.0f, 0.0f};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 y = {__uint_as_float(y2[g][q] << 16), __uint_as_float(y2[g][q] & 0xffff0000u)};
            s2 = fma2(y, y, s2);
        }
        sq[2 * g] = s2.x;
        sq[2 * g + 1] = s2.y;
    }
    // The sum over the eight lanes of a row; at the first two steps a lane gives away the rows that it does not go on with.
    const bool up4 = lane & 4, up8 = lane & 8;
    const float a0 = (up4 ? sq[2] : sq[0]) + __shfl_xor_sync(0xffffffffu, up4 ? sq[0] : sq[2], 4);
    const float a1 = (up4 ? sq[3] : sq[1]) + __shfl_xor_sync(0xffffffffu, up4 ? sq[1] : sq[3], 4);
    float a = (up8 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up8 ? a0 : a1, 8);
    a += __shfl_xor_sync(0xffffffffu, a, 16);
    if (lane < 16) red[quad * CH + i0 + 2 * (lane & 3) + 8 * (up4 ? 1 : 0) + (up8 ? 1 : 0)] = a;
    ok = named_bar_all(bar, 128, ok);
    if (ok) fetch();
    // A row's factor is formed by one lane of each of the first two quarters (a square root and a division, both IEEE).
    const float* at = red + i0 + (lane & 15);
    const float rinv = 0.0625f * (1.0f / sqrtf((((at[0] + at[CH]) + at[2 * CH]) + at[3 * CH]) / (float)DV + eps));
    auto sigmoid16 = [](float x) { return rcp_approx(fmaf(ex2_ftz(-kLog2e * x), 0.0625f, 0.0625f)); };
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        const float2 rv = {__shfl_sync(0xffffffffu, rinv, 2 * (lane & 3) + 8 * g), __shfl_sync(0xffffffffu, rinv, 2 * (lane & 3) + 8 * g + 1)};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 sig = {sigmoid16(__uint_as_float(gt[g][q] << 16)), sigmoid16(__uint_as_float(gt[g][q] & 0xffff0000u))};
            const float2 y = mul2(mul2({nw[q], nw[q]}, mul2({__uint_as_float(y2[g][q] << 16), __uint_as_float(y2[g][q] & 0xffff0000u)}, rv)), sig);
            y2[g][q] = tc::bf16x2(y.x, y.y);
        }
    }
    return ok;
}

// Walks `chain`, or (MANY) the chains of a fused launch that this block's loader warp takes off the counter, until there are none.
// Nothing is set up or drained between two of these: the buffers, accumulators and barriers go on alternating with the chunks, whichever
// chain they belong to, the next chain's first chunks are loaded behind the last ones of the chain before, and the outputs of a chain's
// last chunk leave behind the next chain's first D.  A walk that began and ended by itself took 23 us for five chunks, 13 of them beside the
// chunks: counter, metadata, barriers and first loads one after another, the state a line per 16 bytes, the last chunk's gate.  Whole
// calls, us: chunked layer prefill of 4 x 2,048 rows 1,136 -> 1,043, of 3 x 700 342 -> 301; core prefill of 8,192 rows in 8 sequences 525 -> 504, with
// the norm in 3 sequences 663 -> 582; 8 chains of 1,024 chunks (one walk each) 1,968 -> 1,845.
template <bool MANY, bool GATED, bool WALK_U>
__device__ void state_role(const SpParams& p, unsigned char* smem, const uint32_t tm, const int chain, const Walk wk) {
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + oBarsState);
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + oCtl);
    volatile Chain* recs = reinterpret_cast<volatile Chain*>(smem + oChain);  // the chain that is walked, and the one before or after it
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quad = warp & 3, cg = warp >> 2;
    if (!MANY && nothing_to_do(p, chain_of(p, wk, chain))) return;
    const WaitCtx ctx{ctl, ctl + 1, p.status};
    auto wait = [&](int i, int phase) { return mbar_wait(&bars[i], (uint32_t)(phase & 1), ctx, kStatusWaitPrefill); };
    // This block's chain number n lies in record n & 1 until everyone has released it; its number of chunks, -1 where there are no more
    // chains, -2 where a wait gave up.
    auto chain_count = [&](int n) -> int { return wait(bChainFull + (n & 1), n >> 1) ? recs[n & 1].count : -2; };
    auto release = [&](int n) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[bChainEmpty + (n & 1)]);
    };
    // In every role C counts the chunks of all the block's chains: it selects the buffers and gives the phases.

    if (warp == kOutWarp) {
        // The output warp: each finished tile of rows goes to the shard-local `out` and, for a head-sharded launch, into
        // every rank's full buffer -- the all-gather, done here: a peer's buffer is reached over NVLink.  A full chunk
        // leaves by tiled tensor stores (two per destination), off the compute warps' path; a sequence's last, partial
        // chunk by the warp's own stores, so that no row beyond the sequence is touched.
        bool alive = wk.emit;
        for (int seq = 0, C = 0; alive; ++seq) {
            const int count = chain_count(seq);
            if (count < 0) break;
            const int rows = recs[seq & 1].rows, h = recs[seq & 1].h;
            const long long row = recs[seq & 1].row;
            release(seq);
            for (int c = 0; c < count; ++c, ++C) {
                const int n = min(CH, rows - c * CH);
                const long long gr0 = row + (long long)c * CH;
                if (!wait(bOutFull + (C & 1), C >> 1)) { alive = false; break; }
                const unsigned char* tile = smem + sOut + (C & 1) * kOutTile;
                if (n == CH) {
                    if (lane == 0) {
                        for (int x = 0; x < 2; ++x) {
                            if (p.out != nullptr) tensor_store_3d(&p.tm_out, x * 64, h, (int)gr0, tile + x * kBox);
                            for (int pe = 0; pe < p.ranks; ++pe) tensor_store_3d(&p.tm_full[pe], x * 64, p.head0 + h, (int)gr0, tile + x * kBox);
                        }
                        bulk_commit();
                        bulk_wait_read<0>();  // the tile has been read: the compute warps may refill it
                    }
                } else {
                    for (int e = lane; e < n * 16; e += 32) {
                        const int r = e >> 4, piece = e & 15;
                        const uint4 v4 = *reinterpret_cast<const uint4*>(tile + box_piece(r, piece));
                        if (p.out != nullptr) *reinterpret_cast<uint4*>(p.out + ((gr0 + r) * p.H + h) * DV + piece * 8) = v4;
                        const long long at_full = ((gr0 + r) * p.heads_total + p.head0 + h) * DV + piece * 8;
                        for (int pe = 0; pe < p.ranks; ++pe) *reinterpret_cast<uint4*>(p.full[pe] + at_full) = v4;
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[bOutEmpty + (C & 1)]);
            }
        }
        if (lane == 0) bulk_wait_all<0>();
        tc::fence_before_sync();
        __syncthreads();
        return;
    }
    if (warp == kLoaderWarp) {
        if (lane == 0) {
            unsigned int* set = p.sets + p.ctr * kTailSet;
            const int chains = p.batch * p.H;
            auto take = [&]() { return MANY ? (int)min(atomicAdd(set + 1, 1u), (unsigned)chains) : chain; };
            // Record number n; -1 chunks end the list.
            auto publish = [&](int n, const Chain& c) -> bool {
                if (!wait(bChainEmpty + (n & 1), (n >> 1) ^ 1)) return false;
                volatile Chain& to = recs[n & 1];
                to.count = c.count; to.rows = c.rows; to.h = c.h; to.start = c.start; to.row = c.row; to.s_elem = c.s_elem;
                mbar_arrive(&bars[bChainFull + (n & 1)]);
                return true;
            };
            // A chunk's gate values, for a chunk that the norm is fused into: into the tile that its outputs will take, when the chunk two before
            // has left it, and asked for behind the rows of the chunk after, so that nothing waits for that.
            bool gate_due = false;
            int gate_row = 0, gate_h = 0;
            auto load_gate = [&](int C) -> bool {  // of chunk C
                if (!wait(bOutEmpty + (C & 1), (C >> 1) ^ 1)) return false;
                if (gate_row < 0) {  // a partial chunk's are read by the threads that want them
                    mbar_arrive(&bars[bGate + (C & 1)]);
                    return true;
                }
                mbar_arrive_expect_tx(&bars[bGate + (C & 1)], kOutTile);
                for (int x = 0; x < 2; ++x) tensor_load_3d(smem + sOut + (C & 1) * kOutTile + x * kBox, &p.tm_gate, x * 64, gate_h, gate_row, &bars[bGate + (C & 1)]);
                return true;
            };
            int next = take(), C = 0;
            for (int seq = 0;;) {
                const int ch = next;
                if ((MANY && ch >= chains) || (!MANY && seq > 0)) {
                    publish(seq, Chain{-1, 0, 0, 0, 0, 0});
                    break;
                }
                const int real = MANY ? chain_at(p, ch) : ch;
                const Chain at = chain_of(p, wk, real);
                if constexpr (MANY) {
                    if (nothing_to_do(p, at)) {
                        next = take();
                        continue;
                    }
                    // Its state on the way into L2, and the chain's items, finished by whichever blocks took them: they lie in its group.
                    const int elem = p.state_bf16 ? 2 : 4;
                    const char* state = reinterpret_cast<const char*>(at.start ? p.state_in : p.state_out) + at.s_elem * elem;
                    if ((reinterpret_cast<uintptr_t>(state) & 15) == 0) bulk_prefetch(state, DV * DK * elem);
                    const int g = ch / p.group, want = min(p.group, chains - g * p.group) * p.seg_chunks;
                    if (!count_wait(set + kTailDone + g, (unsigned)want, ctx, kStatusWaitPrefill)) {
                        ctl[1] = 1u;
                        break;
                    }
                    fence_proxy_async_global();
                }
                if (!publish(seq, at)) break;
                ++seq;
                if (at.count == 0 && gate_due) {  // no rows behind which the gate of the chunk before would be asked for
                    if (!load_gate(C - 1)) break;
                    gate_due = false;
                }
                const int j0 = (wk.ja - p.state_chunk0);
                bool ok = true;
                for (int c = 0; ok && c < at.count; ++c, ++C) {
                    const unsigned char* slot = slot_of(p.ws_state, p.seg_chunks, real, j0 + c);
                    const int x = C & 1;
                    if (!(ok = wait(bEmptyQW + x, (C >> 1) ^ 1))) break;  // an empty barrier starts released
                    mbar_arrive_expect_tx(&bars[bFullQW + x], kQW + 512);
                    bulk_load(smem + sE + x * 512, slot + wEgl, 512, &bars[bFullQW + x]);
                    bulk_load(smem + sQW + x * kQW, slot + wQg, kQW, &bars[bFullQW + x]);
                    // U, or what it is made from, has one buffer: asked for before the chunk's other one, and from L2.
                    const bool walk_v = WALK_U && p.v != nullptr;  // else V lies in the slots
                    if (!WALK_U || wk.use_u) {
                        const bool whole = walk_v && at.rows - c * CH >= CH;
                        if (!(ok = wait(bEmptyU, C ^ 1))) break;
                        constexpr int skip = WALK_U ? wTp : 0;
                        mbar_arrive_expect_tx(&bars[bFullU], kUBytes - skip);
                        bulk_load(smem + sU + skip, slot + wU + skip, (whole ? kTile : kUBytes) - skip, &bars[bFullU]);
                        for (int y = 0; whole && y < 2; ++y) tensor_load_3d(smem + sU + kTile + y * kBox, &p.tm_v, y * 64, at.h, (int)at.row + c * CH, &bars[bFullU]);
                    }
                    if (!(ok = wait(bEmptyMKd + x, (C >> 1) ^ 1))) break;
                    mbar_arrive_expect_tx(&bars[bFullMKd + x], kMKd);
                    bulk_load(smem + sMKd + x * kMKd, slot + wMm, kMKd, &bars[bFullMKd + x]);
                    if (wk.use_u && c + 1 < at.count) {
                        const bool whole = walk_v && at.rows - (c + 1) * CH >= CH;
                        bulk_prefetch(slot + kSlotBytes + wU + (WALK_U ? wTp : 0), (whole ? kTile : kUBytes) - (WALK_U ? wTp : 0));
                        for (int y = 0; whole && y < 2; ++y) tensor_prefetch_3d(&p.tm_v, y * 64, at.h, (int)at.row + (c + 1) * CH);
                    }
                    if (gate_due && !(ok = load_gate(C - 1))) break;
                    gate_due = GATED && wk.emit && p.gate_boxes != 0;
                    gate_row = at.rows - c * CH >= CH ? (int)(at.row + c * CH) : -1;
                    gate_h = at.h;
                }
                if (!ok) break;
                next = take();  // a chunk and a half before it is wanted; any earlier, and blocks that come late find too few left
            }
            if (gate_due) load_gate(C - 1);
        }
        tc::fence_before_sync();
        __syncthreads();
        return;
    }
    if (warp == kMmaWarp) {
        const uint32_t leader = tc::elect_one();
        auto ready = [&](int i, int phase) { return tc::warp_all(wait(i, phase)); };
        constexpr uint32_t idw = tc::idesc_bf16(DV, CH, 0, 1, 0), idq = tc::idesc_bf16(DV, CH, 0, 0, 0), ids = tc::idesc_bf16(DV, DK, 0, 1, 0);
        constexpr uint32_t idv = tc::idesc_bf16(DV, CH, 1, 0, 0), idv2 = tc::idesc_bf16(DV, CH / 2, 1, 0, 0);
        bool alive = true;
        // U^T = V^T T'^T (T' hi, then lo; the rows of V behind the 31st are of the rows of U behind it only).  Behind the wait for the D of the chunk before:
        // the accumulator has been read.
        const bool walk_u = WALK_U && wk.use_u;
        bool have_u = false;  // the chunk to come's is on its way
        auto issue_u = [&]() {
            tc::fence_after_sync();
            const unsigned char* tp = smem + sU + wTp;
#pragma unroll
            for (int lo = 0; lo < 2; ++lo) {
#pragma unroll
                for (int k0 = 0; k0 < CH / 2; k0 += 16)
                    tc::mma_bf16_if(leader, tm + tU, tc::desc_sw128_mnmajor(smem + sU + kTile, CH, k0), tc::desc_kmajor_bf16(tp + lo * (kBox / 2), CH, 0, k0), idv, lo + k0 > 0);
#pragma unroll
                for (int k0 = 0; k0 < CH / 2; k0 += 16)
                    tc::mma_bf16_if(leader, tm + tU + CH / 2, tc::desc_sw128_mnmajor(smem + sU + kTile, CH, CH / 2 + k0),
                                    tc::desc_kmajor_bf16(tp + kBox + lo * (kBox / 4), CH / 2, 0, k0), idv2, true);
            }
            tc::mma_commit_if(leader, &bars[bEmptyU]);
        };
        int C = 0;
        for (int seq = 0; alive; ++seq) {
            const int count = chain_count(seq);
            if (!tc::warp_all(count >= 0)) break;
            release(seq);
            for (int c = 0; tc::warp_all(c < count); ++c, ++C) {
                alive = false;
                if (walk_u && !have_u) {
                    if (!ready(bFullU, C)) break;
                    issue_u();
                }
                const int x = C & 1;
                const uint32_t acc = tm + tO + (uint32_t)x * 64;
                const unsigned char *qw = smem + sQW + x * kQW, *mm = smem + sMKd + x * kMKd, *kdhi = mm + kTile / 2, *kdlo = kdhi + kTile;
                if (!ready(bFullQW + x, C >> 1) || !ready(bS16, C)) break;
                tc::fence_after_sync();
#pragma unroll
                for (int k0 = 0; k0 < DK; k0 += 16)
                    tc::mma_bf16_ts_if(leader, tm + tWS, tm + tS16 + k0 / 2, tc::desc_mnmajor_bf16(qw + kTile, DK, 0, k0), idw, k0 > 0);
                tc::mma_commit_if(leader, &bars[bWS]);
                if (wk.emit) {
                    if (C >= 2 && !ready(bOFree + x, (C >> 1) - 1)) break;  // chunk C - 2's outputs have left this accumulator
                    tc::fence_after_sync();
#pragma unroll
                    for (int k0 = 0; k0 < DK; k0 += 16)
                        tc::mma_bf16_ts_if(leader, acc, tm + tS16 + k0 / 2, tc::desc_kmajor_bf16(qw, CH, 0, k0), idq, k0 > 0);
                }
                if (!ready(bSDec, C)) break;  // the warps have read exp(G_last) too
                tc::mma_commit_if(leader, &bars[bEmptyQW + x]);
                if (!ready(bFullMKd + x, C >> 1) || !ready(bD, C)) break;
                tc::fence_after_sync();
#pragma unroll
                for (int k0 = 0; k0 < CH; k0 += 16) tc::mma_bf16_ts_if(leader, tm + tS, tm + tDhi + k0 / 2, tc::desc_mnmajor_bf16(kdhi, CH, 0, k0), ids, true);
#pragma unroll
                for (int k0 = 0; k0 < CH; k0 += 16) tc::mma_bf16_ts_if(leader, tm + tS, tm + tDlo + k0 / 2, tc::desc_mnmajor_bf16(kdhi, CH, 0, k0), ids, true);
#pragma unroll
                for (int k0 = 0; k0 < CH; k0 += 16) tc::mma_bf16_ts_if(leader, tm + tS, tm + tDhi + k0 / 2, tc::desc_mnmajor_bf16(kdlo, CH, 0, k0), ids, true);
                tc::mma_commit_if(leader, &bars[bSNew]);
                if (wk.emit) {
#pragma unroll
                    for (int k0 = 0; k0 < CH; k0 += 16) tc::mma_bf16_ts_if(leader, acc, tm + tDhi + k0 / 2, tc::desc_mnmajor_bf16(mm, CH, 0, k0), idw, true);
                    tc::mma_commit_if(leader, &bars[bO + x]);
                }
                tc::mma_commit_if(leader, &bars[bEmptyMKd + x]);
                have_u = walk_u && tc::warp_all(c + 1 < count) && tc::warp_all(mbar_test(&bars[bFullU], (uint32_t)((C + 1) & 1)));
                if (have_u) issue_u();
                if (leader) atomicAdd(const_cast<uint32_t*>(ctl), 1u);
                __syncwarp();
                alive = true;
            }
        }
        // Nobody else waits for the last two chunks' buffers.
        for (int c = max(C - 2, 0); c < C; ++c)
            if (!ready(bEmptyQW + (c & 1), c >> 1) || !ready(bEmptyMKd + (c & 1), c >> 1)) break;
        tc::fence_before_sync();
        __syncthreads();
        return;
    }

    bool alive = true;
    // What this warp wrote for the tensor core, or left in (or took out of) tensor memory, is there: one arrival a warp.
    auto arrive = [&](int i) {
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[i]);
    };
    // This thread's value channel (tensor-memory lane), 32 key channels of the state and 16 rows of the other accumulators.
    const int v = quad * 32 + lane, k_first = cg * 32, i0 = cg * 16;
    // S^T as bf16 pairs for chunk c's products, then the decayed S^T back.
    auto begin_chunk = [&](int c) -> bool {
        uint32_t r[32], pr[16];
        tc::tmem_ld32(tc::tmem_addr(tm, quad, tS + k_first), r);
        tc::tmem_ld_wait();
#pragma unroll
        for (int x = 0; x < 16; ++x) pr[x] = tc::bf16x2(__uint_as_float(r[2 * x]), __uint_as_float(r[2 * x + 1]));
        tc::tmem_st16(tc::tmem_addr(tm, quad, tS16 + k_first / 2), pr);
        tc::tmem_st_wait();
        arrive(bS16);
        if (p.state_bf16) {  // a bf16 state is rounded once per chunk
#pragma unroll
            for (int x = 0; x < 16; ++x) {
                r[2 * x] = pr[x] << 16;
                r[2 * x + 1] = pr[x] & 0xffff0000u;
            }
        }
        if (!wait(bFullQW + (c & 1), c >> 1)) return false;
        const float4* el = reinterpret_cast<const float4*>(smem + sE + (c & 1) * 512 + k_first * 4);
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const float4 e = el[x];
            r[4 * x] = __float_as_uint(__uint_as_float(r[4 * x]) * e.x);
            r[4 * x + 1] = __float_as_uint(__uint_as_float(r[4 * x + 1]) * e.y);
            r[4 * x + 2] = __float_as_uint(__uint_as_float(r[4 * x + 2]) * e.z);
            r[4 * x + 3] = __float_as_uint(__uint_as_float(r[4 * x + 3]) * e.w);
        }
        tc::tmem_st32(tc::tmem_addr(tm, quad, tS + k_first), r);
        tc::tmem_st_wait();
        arrive(bSDec);
        return true;
    };

    // ---- the incoming state into tensor memory; a thread's 32 key channels are consecutive in every state buffer ------------
    const int b_at = v * DK + k_first;
    auto piece_aligned = [](const void* at) { return (reinterpret_cast<uintptr_t>(at) & 15) == 0; };  // for all lanes or none
    auto state_in = [&](bool start, long long s_elem) {
        const void* src = start ? p.state_in : p.state_out;
        const long long s_at = s_elem + b_at;
        uint32_t r[32];
        if (wk.init == 1 || wk.init == 2) {
#pragma unroll
            for (int x = 0; x < 32; ++x) r[x] = wk.init == 2 && k_first + x == v ? __float_as_uint(1.0f) : 0u;
        } else if (wk.init == 0 && p.state_bf16) {
            const uint16_t* at = reinterpret_cast<const uint16_t*>(src) + s_at;
            if (piece_aligned(at)) {
                state_to_tmem(tc::tmem_addr(tm, quad, tS + k_first), at - lane * DK, lane);
                tc::tmem_st_wait();
                return;
            }
#pragma unroll
            for (int x = 0; x < 32; ++x) r[x] = (uint32_t)at[x] << 16;
        } else {
            const float* at = wk.init == 3 ? wk.from + b_at : reinterpret_cast<const float*>(src) + s_at;
            if (piece_aligned(at)) {
                state_to_tmem(tc::tmem_addr(tm, quad, tS + k_first), at - lane * DK, lane);
                tc::tmem_st_wait();
                return;
            }
#pragma unroll
            for (int x = 0; x < 32; ++x) r[x] = __float_as_uint(at[x]);
        }
        tc::tmem_st32(tc::tmem_addr(tm, quad, tS + k_first), r);
        tc::tmem_st_wait();
    };
    // The four warps that share output rows vote at a barrier in every chunk when the norm is fused, and before every chain of
    // several; one that gives up before it still takes part.
    const bool votes = GATED && wk.emit;
    auto leave = [&] {
        if (MANY || votes) named_bar_all(4 + cg, 128, false);
        alive = false;
    };

    // ---- a chunk's outputs: bf16(y), or the gated RMSNorm of bf16(y) ---------------------------------------------------
    // O^T is read in the fragment layout, from which a transposing matrix store puts rows of the output into the tile: this
    // thread's values are (channel fv + 8 q, row fi + 8 g + e), q < 4, g < 2, e < 2.
    const int fv = quad * 32 + (lane >> 2), fi = i0 + 2 * (lane & 3);
    float nw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (votes)
#pragma unroll
        for (int q = 0; q < 4; ++q) nw[q] = bf16_bits_to_f32(p.norm_w[fv + 8 * q]);
    // Into (and, with the gate, out of) the output tile: a lane names the row (lane % 8) of matrix lane / 8, the matrices being
    // (channels 8 (m % 2), rows 8 (m / 2)) of the two halves of the warp's channels.
    const int tile_row = i0 + (lane >> 4) * 8 + (lane & 7), tile_piece = quad * 4 + ((lane >> 3) & 1);
    // A chunk's gate values, laid out as y2 below.  They lie in the tile that the outputs go to (the loader's copy), or, in a partial chunk
    // or where the rows are not on 16 bytes, are fetched before D is formed, so that their latency is not in the walk.
    uint32_t gt[2][4];
    auto fetch_gate = [&](const volatile Chain& of, int c) {
        const int n = of.rows - c * CH;
        const uint16_t* at = p.gate + (of.row + c * CH + fi) * p.gate_stride + of.h * DV + fv;
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t lo = fi + 8 * g < n ? at[8 * g * p.gate_stride + 8 * q] : 0u, hi = fi + 8 * g + 1 < n ? at[(8 * g + 1) * p.gate_stride + 8 * q] : 0u;
                gt[g][q] = lo | hi << 16;
            }
    };
    auto emit = [&](int c, bool boxes) -> bool {  // boxes: the gate values come from the tile
        bool ok = wait(bO + (c & 1), c >> 1);
        tc::fence_after_sync();
        uint32_t ra[8], rb[8];
        const uint32_t at = tc::tmem_addr(tm, quad, tO + (uint32_t)(c & 1) * 64 + i0);
        tc::tmem_ld_frag(at, ra);
        tc::tmem_ld_frag(at + (16u << 16), rb);
        tc::tmem_ld_wait();
        arrive(bOFree + (c & 1));
        ok = ok && wait(bOutEmpty + (c & 1), (c >> 1) ^ 1);
        uint32_t y2[2][4];  // [g][q]: rows fi + 8 g and the next of channel fv + 8 q
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            y2[g][0] = tc::bf16x2(__uint_as_float(ra[4 * g]), __uint_as_float(ra[4 * g + 1]));
            y2[g][1] = tc::bf16x2(__uint_as_float(ra[4 * g + 2]), __uint_as_float(ra[4 * g + 3]));
            y2[g][2] = tc::bf16x2(__uint_as_float(rb[4 * g]), __uint_as_float(rb[4 * g + 1]));
            y2[g][3] = tc::bf16x2(__uint_as_float(rb[4 * g + 2]), __uint_as_float(rb[4 * g + 3]));
        }
        unsigned char* dst = smem + sOut + (c & 1) * kOutTile;
        if (votes) {
            if (boxes) ok = ok && wait(bGate + (c & 1), c >> 1);
            ok = gated_rows(reinterpret_cast<float*>(smem + sRed) + (c & 1) * 4 * CH, p.eps, quad, lane, i0, nw, gt, y2, 4 + cg, ok, [&] {
                if (boxes) {
                    tc::ldmatrix_t4(dst + box_piece(tile_row, tile_piece), gt[0][0], gt[0][1], gt[1][0], gt[1][1]);
                    tc::ldmatrix_t4(dst + box_piece(tile_row, tile_piece + 2), gt[0][2], gt[0][3], gt[1][2], gt[1][3]);
                }
            });
        }
        if (!ok) return false;  // else the output warp takes it from there
        tc::stmatrix_t4(dst + box_piece(tile_row, tile_piece), y2[0][0], y2[0][1], y2[1][0], y2[1][1]);
        tc::stmatrix_t4(dst + box_piece(tile_row, tile_piece + 2), y2[0][2], y2[0][3], y2[1][2], y2[1][3]);
        fence_proxy_async_smem();  // the tensor stores read the tile through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[bOutFull + (c & 1)]);
        return true;
    };

    // The outputs of a chunk leave behind the next chunk's D, be that chunk of the same chain or of the next; a chain's record is released
    // with its last outputs.
    int C = 0, due = -1, due_seq = 0;  // due: the chunk of chain due_seq whose outputs are still to leave
    int held = -1;                     // the chain before, while its record is
    auto out_boxes = [&] { return p.gate_boxes != 0 && recs[due_seq & 1].rows - due * CH >= CH; };
    auto emit_due = [&]() -> bool {
        const bool ok = emit(C - 1, votes && out_boxes());
        due = -1;
        if (ok) return true;
        if (votes) alive = false;  // it has voted
        else leave();
        return false;
    };
    auto emit_last = [&]() -> bool {  // where no D is on its way
        if (votes && !out_boxes()) fetch_gate(recs[due_seq & 1], due);
        return emit_due();
    };
    for (int seq = 0;; ++seq) {
        const int count = chain_count(seq);
        if (MANY) {
            if (!named_bar_all(4 + cg, 128, count != -2)) { alive = false; break; }
        } else if (count == -2) { leave(); break; }
        if (count < 0) break;
        state_in(recs[seq & 1].start, recs[seq & 1].s_elem);
        // A sequence of no rows has no D to wait for, and the output warp, which has to read its record too, may wait for these.
        if (count == 0 && held >= 0) {
            if (due >= 0 && !emit_last()) break;
            release(held);
            held = -1;
        }
        if (count > 0 && !begin_chunk(C)) { leave(); break; }
        for (int c = 0; c < count; ++c, ++C) {
            // ---- D^T = U^T - (W S)^T as bf16 hi + lo pairs of rows ------------------------------------------------------------
            if (votes && due >= 0 && !out_boxes()) fetch_gate(recs[due_seq & 1], due);
            uint32_t uu[16];
            if constexpr (!WALK_U) {
                if (!wait(bFullU, C)) { leave(); break; }
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const uint4 u4 = *reinterpret_cast<const uint4*>(smem + sU + u_cell(cg * 4 + x, v));
                    uu[4 * x] = u4.x; uu[4 * x + 1] = u4.y; uu[4 * x + 2] = u4.z; uu[4 * x + 3] = u4.w;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[bEmptyU]);  // U is consumed
            }
            if (!wait(bWS, C)) { leave(); break; }  // (U^T was issued before)
            tc::fence_after_sync();
            {
                uint32_t r[16], wh[8], wl[8];
                if constexpr (WALK_U) tc::tmem_ld16(tc::tmem_addr(tm, quad, tU + i0), uu);
                tc::tmem_ld16(tc::tmem_addr(tm, quad, tWS + i0), r);
                tc::tmem_ld_wait();
                if (!wk.use_u)
#pragma unroll
                    for (int x = 0; x < 16; ++x) uu[x] = 0u;
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    tc::split_bf16x2(__uint_as_float(uu[2 * x]) - __uint_as_float(r[2 * x]), __uint_as_float(uu[2 * x + 1]) - __uint_as_float(r[2 * x + 1]), wh[x], wl[x]);
                tc::tmem_st8(tc::tmem_addr(tm, quad, tDhi + i0 / 2), wh);
                tc::tmem_st8(tc::tmem_addr(tm, quad, tDlo + i0 / 2), wl);
                tc::tmem_st_wait();
                arrive(bD);
            }
            // The outputs of the chunk before leave while the state's product runs.
            if (due >= 0 && !emit_due()) break;
            if (held >= 0) release(held);
            held = -1;
            if (wk.emit) due = c;
            due_seq = seq;
            if (!wait(bSNew, C)) { leave(); break; }
            tc::fence_after_sync();
            if (c + 1 < count && !begin_chunk(C + 1)) { leave(); break; }
        }

        // ---- the outgoing state ---------------------------------------------------------------------------------------------
        if (!alive) break;
        const long long s_out = recs[seq & 1].s_elem + b_at;
        if (wk.fin != 2) {
            const uint32_t from = tc::tmem_addr(tm, quad, tS + k_first);
            uint16_t* to16 = reinterpret_cast<uint16_t*>(p.state_out) + s_out;
            float* to32 = wk.fin == 1 ? wk.to + b_at : reinterpret_cast<float*>(p.state_out) + s_out;
            const bool to_bf16 = wk.fin == 0 && p.state_bf16;
            if (piece_aligned(to_bf16 ? (const void*)to16 : (const void*)to32)) {
                if (to_bf16) state_from_tmem(from, to16 - lane * DK, lane);
                else state_from_tmem(from, to32 - lane * DK, lane);
            } else {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t r[16];
                    tc::tmem_ld16(from + half * 16, r);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int x = 0; x < 16; ++x) {
                        if (to_bf16) to16[half * 16 + x] = f32_to_bf16_bits(__uint_as_float(r[x]));
                        else to32[half * 16 + x] = __uint_as_float(r[x]);
                    }
                }
            }
        }
        if (count == 0) release(seq);
        else held = seq;
    }
    if (alive && due >= 0) emit_last();
    tc::fence_before_sync();
    __syncthreads();
}

// Both roles of a pass in one launch: every block takes items until there are none, then chains.  A block waits for other blocks'
// items only when every item has been handed out, that is to blocks that are running and wait for nobody; or when every block is running and
// those that still take items wait for nobody.
//
// With more chains than blocks some blocks walk one chain more than the others.  They stop taking items when as many are left as the others can do in
// that time (early_blocks, early_from), so that all end together: us, core prefill of
// 8,192 rows in 3 sequences (192 chains on 148 SMs) 499 -> 472, in 8 sequences 454 -> 446, of 20,000 rows x 32 heads in 5 with the norm 673 -> 640; chunked layer prefill of 3 x
// 700 rows 234 -> 215.
template <bool LAYER, bool GATED>
__device__ void fused_roles(const SpParams& p, unsigned char* smem, const uint32_t tm) {
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + oCtl);
    const int tid = threadIdx.x;
    intra_role<LAYER, true, true>(p, smem, tm);
    if (ctl[1] != 0u) return;
    if (tid < kGroupBars * kGroups) mbar_inval(reinterpret_cast<uint64_t*>(smem + tid / kGroupBars * kGroupBytes + gBars) + tid % kGroupBars);
    fence_proxy_async_smem();  // what the intra role left in shared memory is overwritten by bulk copies
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    state_role<true, GATED, true>(p, smem, tm, 0, Walk{p.state_chunk0, p.state_chunk0 + p.seg_chunks, 0, nullptr, 0, nullptr, true, true});
}

// One launch: the state role of one segment on the chain blocks, then the intra role of the next segment on all blocks.
// (An instance for each set of roles and for the norm: both roles are bound by their own instructions, and what an instance does not run costs
// it registers and room in the instruction caches.  Against one for all of the core form: 2 sequences of 10,000 rows x 32 heads 980 -> 865 us,
// 8 chains of 1,024 chunks 1,880 -> 1,680; 4 x 2,048 rows of the layer form 1,011 -> 985.)
template <bool LAYER, bool FUSED, bool GATED, bool WALK_U>
__global__ void __launch_bounds__(kThreadsSp, 1) prefill_sp_kernel(const __grid_constant__ SpParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + oCtl);
    uint32_t* tmem_slot = const_cast<uint32_t*>(ctl) + 2;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        uint64_t* bs = reinterpret_cast<uint64_t*>(smem + oBarsState);
        for (int i = 0; i < kStateBars; ++i) mbar_init(bs + i, state_bar_count(i, WALK_U));
        ctl[0] = 0u;
        ctl[1] = 0u;
        mbar_init_fence();
    }
    if (warp == 0) tc::tmem_alloc(tmem_slot, kTmemCols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = *tmem_slot;
    grid_ready();
    // the next launch's counters; nobody reads them during this launch.  (A scan pass leaves the counters alone: it may run
    // beside the next super-block's intra launch on another stream.)
    if (FUSED && blockIdx.x == 0 && tid < kTailSet) p.sets[(p.ctr ^ 1) * kTailSet + tid] = 0u;
    if (FUSED && tid == 0) atomicAdd(p.sets + p.ctr * kTailSet + kTailBegun, 1u);
    if (!FUSED && blockIdx.x == 0 && tid == 0 && p.scan_pass == 0) p.counters[p.ctr ^ 1] = 0u;
    if constexpr (FUSED) {
        fused_roles<LAYER, GATED>(p, smem, tm);
    } else if (p.has_state) {
        // Block (chain); (chain, segment s < scan_p1, kind) in scan pass 1: the segment's offset and transition; (chain, segment) in
        // scan pass 2: the walk with outputs from the segment's true incoming state, of which only the last delivers the sequence's
        // final state (the others end where the next one starts).
        const int pass = p.scan_pass, kind = blockIdx.x & 1, per = pass == 1 ? p.scan_p1 : pass == 2 ? p.scan_k : 1;
        const int at = pass == 1 ? blockIdx.x >> 1 : blockIdx.x, sg = at % per, chain = at / per;
        if (chain < p.batch * p.H) {
            const int hi = p.state_chunk0 + p.seg_chunks;  // the launch's chunk range ends here
            Walk wk{p.state_chunk0, hi, 0, nullptr, 0, nullptr, true, true};
            if (pass != 0) {
                const bool last = sg == p.scan_k - 1;
                wk.ja = min(p.state_chunk0 + sg * p.scan_chunks, hi);
                wk.jb = last ? (p.scan_open ? 0x7fffffff : hi) : min(p.state_chunk0 + (sg + 1) * p.scan_chunks, hi);
                if (pass == 1) {
                    wk.init = kind ? 2 : 1;
                    wk.fin = 1;
                    wk.to = p.scan_ab + (((size_t)chain * p.scan_p1 + sg) * 2 + kind) * DV * DK;
                    wk.use_u = kind == 0;
                    wk.emit = false;
                } else {
                    wk.init = 3;
                    wk.from = p.scan_start + ((size_t)chain * p.scan_k + sg) * DV * DK;
                    wk.fin = last ? 0 : 2;
                }
            }
            state_role<false, GATED, WALK_U>(p, smem, tm, chain, wk);
            tc::fence_after_sync();
        }
    }
    if (!FUSED && p.has_intra && ctl[1] == 0u) intra_role<LAYER, false, WALK_U>(p, smem, tm);
    if (ctl[1] != 0u) {  // after an abort copies into this block's shared memory may still be in flight: give them a bounded time
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 2000000ull) {
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tm, kTmemCols);
}

// =====================================================================================================================
// The prefill without a workspace: a block has a chain, one group of eight warps forms its chunks' items (intra_group) and eight warps walk them, the
// slot between them in shared memory.  The walk of a chunk runs beside the next one's item; the slot is one, and is free when the walk's last product of
// the chunk has read it, by which time the group has come to its operand tiles.  HBM sees the algorithm's bytes.
// Bound by a chunk's item, a chain of group-wide steps (scan 2,000 cycles, tiles 2,700, L and M 1,200, inverse 4,000, T' 800, products 1,000, results 1,200):
// 12,800 cycles a chunk.  One kernel of sixteen warps that did all of a chunk's steps one after the other took 22,900.  us, that / this: 64 rows x 64 heads
// 21.6 / 14.7, 1,000 rows 199 / 116, 8,192 rows in one sequence 1,558 / 861, in eight 774 / 444 (with the norm 788 / 517); 16,384 rows x 8 heads 3,052 / 1,682.
// =====================================================================================================================
constexpr int kOneThreads = 2 * kGroupThreads + 96, kOneLoader = 16, kOneOut = 17, kOneMma = 18;
constexpr uint32_t t1S = 128, t1S16 = 256, t1WS = 320, t1O = 384, t1Dhi = 448, t1Dlo = 480;  // behind the group's columns

template <bool GATED>
__device__ __forceinline__ void walk_one(const SpParams& p, unsigned char* smem, const uint32_t tm, const WaitCtx& ctx, const Chain& at) {
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + oBarsOne);
    const unsigned char* slot = smem + oSlotOne;
    unsigned char* tile = smem + oSlotOne + wU;  // the outputs of a chunk, boxes of 64 rows x 128 bytes
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3, half = (warp >> 2) & 1;
    auto wait = [&](int i, int phase) { return mbar_wait(&bars[i], (uint32_t)(phase & 1), ctx, kStatusWaitPrefill); };
    const int count = at.count;
    if (warp == kOneOut) {
        for (int c = 0; c < count; ++c) {
            const int n = min(CH, at.rows - c * CH);
            const long long gr0 = at.row + (long long)c * CH;
            if (GATED && n == CH) {  // the gate's values into the tile that the outputs will take, as soon as U has left it
                if (lane == 0)
                    for (int x = 0; x < 2; ++x) tensor_prefetch_3d(&p.tm_gate, x * 64, at.h, (int)gr0);
                if (!wait(o1D, c)) break;
                if (lane == 0) {
                    mbar_arrive_expect_tx(&bars[o1Gate], kTile);
                    for (int x = 0; x < 2; ++x) tensor_load_3d(tile + x * kBox, &p.tm_gate, x * 64, at.h, (int)gr0, &bars[o1Gate]);
                }
            }
            if (!wait(o1OutFull, c)) break;
            if (n == CH) {
                if (lane == 0) {
                    for (int x = 0; x < 2; ++x) tensor_store_3d(&p.tm_out, x * 64, at.h, (int)gr0, tile + x * kBox);
                    bulk_commit();
                    bulk_wait_read<0>();
                }
            } else {
                for (int e = lane; e < n * 16; e += 32)
                    *reinterpret_cast<uint4*>(p.out + ((gr0 + (e >> 4)) * p.H + at.h) * DV + (e & 15) * 8) = *reinterpret_cast<const uint4*>(tile + box_piece(e >> 4, e & 15));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[o1OutEmpty]);
        }
        if (lane == 0) bulk_wait_all<0>();
        return;
    }
    if (warp == kOneMma) {
        const uint32_t leader = tc::elect_one();
        auto ready = [&](int i, int phase) { return tc::warp_all(wait(i, phase)); };
        constexpr uint32_t idw = tc::idesc_bf16(DV, CH, 0, 1, 0), idq = tc::idesc_bf16(DV, CH, 0, 0, 0), ids = tc::idesc_bf16(DV, DK, 0, 1, 0);
        const unsigned char *mm = slot + wMm, *kdhi = slot + wKdHi, *kdlo = slot + wKdLo;
        for (int c = 0; tc::warp_all(c < count); ++c) {
            if (!ready(o1Full, c) || !ready(o1S16, c)) break;
            tc::fence_after_sync();
#pragma unroll
            for (int k0 = 0; k0 < DK; k0 += 16)
                tc::mma_bf16_ts_if(leader, tm + t1WS, tm + t1S16 + k0 / 2, tc::desc_mnmajor_bf16(slot + wW, DK, 0, k0), idw, k0 > 0);
            tc::mma_commit_if(leader, &bars[o1WS]);
            if (c > 0 && !ready(o1OFree, c - 1)) break;
            tc::fence_after_sync();
#pragma unroll
            for (int k0 = 0; k0 < DK; k0 += 16)
                tc::mma_bf16_ts_if(leader, tm + t1O, tm + t1S16 + k0 / 2, tc::desc_kmajor_bf16(slot + wQg, CH, 0, k0), idq, k0 > 0);
            if (!ready(o1SDec, c) || !ready(o1D, c)) break;
            tc::fence_after_sync();
#pragma unroll
            for (int k0 = 0; k0 < CH; k0 += 16) tc::mma_bf16_ts_if(leader, tm + t1S, tm + t1Dhi + k0 / 2, tc::desc_mnmajor_bf16(kdhi, CH, 0, k0), ids, true);
#pragma unroll
            for (int k0 = 0; k0 < CH; k0 += 16) tc::mma_bf16_ts_if(leader, tm + t1S, tm + t1Dlo + k0 / 2, tc::desc_mnmajor_bf16(kdhi, CH, 0, k0), ids, true);
#pragma unroll
            for (int k0 = 0; k0 < CH; k0 += 16) tc::mma_bf16_ts_if(leader, tm + t1S, tm + t1Dhi + k0 / 2, tc::desc_mnmajor_bf16(kdlo, CH, 0, k0), ids, true);
            tc::mma_commit_if(leader, &bars[o1SNew]);
#pragma unroll
            for (int k0 = 0; k0 < CH; k0 += 16) tc::mma_bf16_ts_if(leader, tm + t1O, tm + t1Dhi + k0 / 2, tc::desc_mnmajor_bf16(mm, CH, 0, k0), idw, true);
            tc::mma_commit_if(leader, &bars[o1O]);
            tc::mma_commit_if(leader, &bars[o1Free]);
            if (leader) atomicAdd(const_cast<uint32_t*>(ctx.progress), 1u);
            __syncwarp();
        }
        if (tc::warp_all(count > 0)) ready(o1Free, count - 1);  // nobody else waits for the last chunk's
        return;
    }
    // Eight warps: a thread has a value channel (tensor-memory lane) and two pieces of 32 key channels or 16 rows.
    auto arrive = [&](int i) {
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[i]);
    };
    const int v = quad * 32 + lane, piece0 = half * 2;
    const bool same = p.state_in == p.state_out;
    auto aligned = [](const void* a) { return (reinterpret_cast<uintptr_t>(a) & 15) == 0; };  // for all lanes or none
    // S^T as bf16 pairs for chunk c's products.
    auto operand = [&]() {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            uint32_t r[32], pr[16];
            tc::tmem_ld32(tc::tmem_addr(tm, quad, t1S + (piece0 + s) * 32), r);
            tc::tmem_ld_wait();
#pragma unroll
            for (int x = 0; x < 16; ++x) pr[x] = tc::bf16x2(__uint_as_float(r[2 * x]), __uint_as_float(r[2 * x + 1]));
            tc::tmem_st16(tc::tmem_addr(tm, quad, t1S16 + (piece0 + s) * 16), pr);
        }
        tc::tmem_st_wait();
        arrive(o1S16);
    };
#pragma unroll
    for (int s = 0; s < 2; ++s) {  // the incoming state
        const int k_first = (piece0 + s) * 32;
        const uint32_t to = tc::tmem_addr(tm, quad, t1S + k_first);
        const long long from = at.s_elem + v * DK + k_first;
        const uint16_t* a16 = reinterpret_cast<const uint16_t*>(p.state_in) + from;
        const float* a32 = reinterpret_cast<const float*>(p.state_in) + from;
        if (p.state_bf16 ? aligned(a16) : aligned(a32)) {
            if (p.state_bf16) state_to_tmem(to, a16 - lane * DK, lane);
            else state_to_tmem(to, a32 - lane * DK, lane);
        } else {
            uint32_t r[32];
#pragma unroll
            for (int x = 0; x < 32; ++x) r[x] = p.state_bf16 ? (uint32_t)a16[x] << 16 : __float_as_uint(a32[x]);
            tc::tmem_st32(to, r);
        }
    }
    tc::tmem_st_wait();
    __syncwarp();
    const int fv = quad * 32 + (lane >> 2), tile_piece = quad * 4 + ((lane >> 3) & 1);
    float nw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (GATED)
#pragma unroll
        for (int q = 0; q < 4; ++q) nw[q] = bf16_bits_to_f32(p.norm_w[fv + 8 * q]);
    bool alive = true;
    auto leave = [&] {  // the four warps that share output rows vote at a barrier when the norm is fused
        if (GATED) named_bar_all(4 + half, 128, false);
        alive = false;
    };
    if (count > 0) operand();
    for (int c = 0; c < count; ++c) {
        if (!wait(o1Full, c)) { leave(); break; }
#pragma unroll
        for (int s = 0; s < 2; ++s) {  // the decayed S^T
            const int k_first = (piece0 + s) * 32;
            uint32_t r[32];
            tc::tmem_ld32(tc::tmem_addr(tm, quad, t1S + k_first), r);
            tc::tmem_ld_wait();
            const float4* el = reinterpret_cast<const float4*>(slot + wEgl + k_first * 4);
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                const float4 e = el[x];
                const float ee[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
                for (int y = 0; y < 4; y += 2) {
                    float s0 = __uint_as_float(r[4 * x + y]), s1 = __uint_as_float(r[4 * x + y + 1]);
                    if (p.state_bf16) {  // a bf16 state is rounded once per chunk
                        const uint32_t two = tc::bf16x2(s0, s1);
                        s0 = __uint_as_float(two << 16);
                        s1 = __uint_as_float(two & 0xffff0000u);
                    }
                    r[4 * x + y] = __float_as_uint(s0 * ee[y]);
                    r[4 * x + y + 1] = __float_as_uint(s1 * ee[y + 1]);
                }
            }
            tc::tmem_st32(tc::tmem_addr(tm, quad, t1S + k_first), r);
        }
        tc::tmem_st_wait();
        arrive(o1SDec);
        uint32_t gt[2][2][4];
        const int n = at.rows - c * CH;
        const bool boxes = n >= CH;  // else the threads read the gate's values that they want
        if (GATED && !boxes) {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int fi = (piece0 + s) * 16 + 2 * (lane & 3);
                const uint16_t* g = p.gate + (at.row + c * CH + fi) * p.gate_stride + at.h * DV + fv;
#pragma unroll
                for (int y = 0; y < 2; ++y)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t lo = fi + 8 * y < n ? g[8 * y * p.gate_stride + 8 * q] : 0u, hi = fi + 8 * y + 1 < n ? g[(8 * y + 1) * p.gate_stride + 8 * q] : 0u;
                        gt[s][y][q] = lo | hi << 16;
                    }
            }
        }
        if (!wait(o1WS, c)) { leave(); break; }
        tc::fence_after_sync();
#pragma unroll
        for (int s = 0; s < 2; ++s) {  // D^T = U^T - (W S)^T as bf16 hi + lo pairs of rows
            const int cg = piece0 + s;
            uint32_t r[16], wh[8], wl[8];
            tc::tmem_ld16(tc::tmem_addr(tm, quad, t1WS + cg * 16), r);
            float uu[16];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const float4 u4 = *reinterpret_cast<const float4*>(slot + wU + u_cell(cg * 4 + x, v));
                uu[4 * x] = u4.x; uu[4 * x + 1] = u4.y; uu[4 * x + 2] = u4.z; uu[4 * x + 3] = u4.w;
            }
            tc::tmem_ld_wait();
#pragma unroll
            for (int x = 0; x < 8; ++x) tc::split_bf16x2(uu[2 * x] - __uint_as_float(r[2 * x]), uu[2 * x + 1] - __uint_as_float(r[2 * x + 1]), wh[x], wl[x]);
            tc::tmem_st8(tc::tmem_addr(tm, quad, t1Dhi + cg * 8), wh);
            tc::tmem_st8(tc::tmem_addr(tm, quad, t1Dlo + cg * 8), wl);
        }
        tc::tmem_st_wait();
        arrive(o1D);
        if (!wait(o1SNew, c)) { leave(); break; }
        tc::fence_after_sync();
        if (c + 1 < count) operand();
        // ---- the chunk's outputs: bf16(y), or the gated RMSNorm of bf16(y); U has been consumed by all --------------------------------
        if (!wait(o1O, c)) { leave(); break; }
        tc::fence_after_sync();
        uint32_t y2[2][2][4];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            uint32_t ra[8], rb[8];
            const uint32_t from = tc::tmem_addr(tm, quad, t1O + (piece0 + s) * 16);
            tc::tmem_ld_frag(from, ra);
            tc::tmem_ld_frag(from + (16u << 16), rb);
            tc::tmem_ld_wait();
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                y2[s][g][0] = tc::bf16x2(__uint_as_float(ra[4 * g]), __uint_as_float(ra[4 * g + 1]));
                y2[s][g][1] = tc::bf16x2(__uint_as_float(ra[4 * g + 2]), __uint_as_float(ra[4 * g + 3]));
                y2[s][g][2] = tc::bf16x2(__uint_as_float(rb[4 * g]), __uint_as_float(rb[4 * g + 1]));
                y2[s][g][3] = tc::bf16x2(__uint_as_float(rb[4 * g + 2]), __uint_as_float(rb[4 * g + 3]));
            }
        }
        arrive(o1OFree);
        const bool ok = !GATED || !boxes || wait(o1Gate, c);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int i0 = (piece0 + s) * 16, tile_row = i0 + (lane >> 4) * 8 + (lane & 7);
            if (GATED && !gated_rows(reinterpret_cast<float*>(smem + oRedOne), p.eps, quad, lane, i0, nw, gt[s], y2[s], 4 + half, ok, [&] {
                    if (boxes) {
                        tc::ldmatrix_t4(tile + box_piece(tile_row, tile_piece), gt[s][0][0], gt[s][0][1], gt[s][1][0], gt[s][1][1]);
                        tc::ldmatrix_t4(tile + box_piece(tile_row, tile_piece + 2), gt[s][0][2], gt[s][0][3], gt[s][1][2], gt[s][1][3]);
                    }
                })) {
                alive = false;
                break;
            }
            tc::stmatrix_t4(tile + box_piece(tile_row, tile_piece), y2[s][0][0], y2[s][0][1], y2[s][1][0], y2[s][1][1]);
            tc::stmatrix_t4(tile + box_piece(tile_row, tile_piece + 2), y2[s][0][2], y2[s][0][3], y2[s][1][2], y2[s][1][3]);
        }
        if (!alive) break;
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[o1OutFull]);
    }
    if (!alive || (count == 0 && (same || !at.start))) return;
#pragma unroll
    for (int s = 0; s < 2; ++s) {  // the outgoing state
        const int k_first = (piece0 + s) * 32;
        const uint32_t from = tc::tmem_addr(tm, quad, t1S + k_first);
        const long long to = at.s_elem + v * DK + k_first;
        uint16_t* to16 = reinterpret_cast<uint16_t*>(p.state_out) + to;
        float* to32 = reinterpret_cast<float*>(p.state_out) + to;
        if (p.state_bf16 ? aligned(to16) : aligned(to32)) {
            if (p.state_bf16) state_from_tmem(from, to16 - lane * DK, lane);
            else state_from_tmem(from, to32 - lane * DK, lane);
        } else {
            uint32_t r[32];
            tc::tmem_ld32(from, r);
            tc::tmem_ld_wait();
#pragma unroll
            for (int x = 0; x < 32; ++x) {
                if (p.state_bf16) to16[x] = f32_to_bf16_bits(__uint_as_float(r[x]));
                else to32[x] = __uint_as_float(r[x]);
            }
        }
    }
}

// The sequence that comes n-th when the longest come first (by each warp; up to kOrderSeqs of them).  Blocks of more chains than SMs are handed out in order, and a
// long chain begun when the others end runs alone.  us, as they come / so: 16,384 rows x 32 heads in 8 sequences 621 / 446, 50,000 rows in 7 1,698 / 1,317; 64 heads,
// 8,192 rows in 3 619 / 515, in 16 465 / 451, 12,000 in 6 678 / 643; where neither order fills the last round, 8,192 rows in 8 443 / 457, 3,000 in 3 245 / 249.  (The
// fused launches' blocks take items as they go: there 1 to 2 % slower.)
constexpr int kOrderSeqs = 32;
__device__ __forceinline__ int nth_longest(const SpParams& p, int n) {
    const int lane = threadIdx.x & 31, chunks = lane < p.batch ? (p.cu[lane + 1] - p.cu[lane] + CH - 1) / CH : -1;
    int rank = 0;
    for (int i = 0; i < p.batch; ++i) {
        const int other = __shfl_sync(0xffffffffu, chunks, i);
        rank += other > chunks || (other == chunks && i < lane) ? 1 : 0;
    }
    return __ffs(__ballot_sync(0xffffffffu, lane < p.batch && rank == n)) - 1;
}

template <bool GATED>
__global__ void __launch_bounds__(kOneThreads, 1) prefill_one_kernel(const __grid_constant__ SpParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + oCtlOne);
    uint32_t* tmem_slot = const_cast<uint32_t*>(ctl) + 2;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        uint64_t* b = reinterpret_cast<uint64_t*>(smem + gBars);
        for (int i = 0; i < kGroupBars; ++i) mbar_init(b + i, i == 2 ? 8 : 1);  // as in intra_role()
        uint64_t* one = reinterpret_cast<uint64_t*>(smem + oBarsOne);
        for (int i = 0; i < kOneBars; ++i) mbar_init(one + i, i == o1S16 || i == o1SDec || i == o1D || i == o1OFree || i == o1OutFull ? 8 : 1);
        ctl[0] = 0u;
        ctl[1] = 0u;
        mbar_init_fence();
    }
    if (warp == 0) tc::tmem_alloc(tmem_slot, kTmemCols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = *tmem_slot;
    grid_ready();
    const WaitCtx ctx{ctl, ctl + 1, p.status};
    int chain = blockIdx.x;
    if (p.longest_first) chain = nth_longest(p, chain / p.H) * p.H + chain % p.H;
    const Chain at = chain_of(p, Walk{0, 0x7fffffff, 0, nullptr, 0, nullptr, true, true}, chain);
    if (warp < kGroupThreads / 32) intra_group<false, false, false, true>(p, smem, tm, ctx, 0);
    else if (warp == kOneLoader) intra_loader<false, false, false, true>(p, smem, ctx, 0, chain);
    else walk_one<GATED>(p, smem, tm, ctx, at);
    if (ctl[1] != 0u) {  // after an abort copies into this block's shared memory may still be in flight: give them a bounded time
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 2000000ull) {
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tm, kTmemCols);
}

// Between the two scan passes: the state before every segment, S_start[s + 1] = A_s S_start[s] + B_s in FP32, from the
// caller's state.  A state's value columns never mix, so a block owns two of them (held in shared memory across the
// segments) and a thread one key channel: acc[v] += A_s[k][k'] S[k'][v] with A_s read along k (coalesced; A_s lies in
// the state's layout, entry [k'][k]).
constexpr int kComposeCols = 2;  // value columns per block: 64 blocks a chain (with eight columns, 16 blocks, a launch took 0.3 ms)
__global__ void __launch_bounds__(128) scan_compose_kernel(const __grid_constant__ SpParams p) {
    constexpr int kCols = kComposeCols;
    __shared__ float S[kCols][DK];
    const int chain = blockIdx.x / (DV / kCols), v0 = (blockIdx.x % (DV / kCols)) * kCols, k = threadIdx.x;
    const int b = chain / p.H, h = chain % p.H;
    const float* s0 = p.scan_carry_in != nullptr ? p.scan_carry_in + (size_t)chain * DV * DK
                                                 : reinterpret_cast<const float*>(p.state_in) + p.state_off[b] + (long long)h * DV * DK;
    // Segment 0 starts from a copy: in place, the last segment of a sequence that ends early writes the final state over the
    // caller's before segment 0 may have read it.
#pragma unroll
    for (int vi = 0; vi < kCols; ++vi) {
        S[vi][k] = s0[(v0 + vi) * DK + k];
        p.scan_start[(size_t)chain * p.scan_k * DV * DK + (v0 + vi) * DK + k] = S[vi][k];
    }
    __syncthreads();
    for (int sg = 0; sg < p.scan_p1; ++sg) {
        const float* B = p.scan_ab + ((size_t)chain * p.scan_p1 + sg) * 2 * DV * DK;
        const float* A = B + DV * DK;
        float acc[kCols];
#pragma unroll
        for (int vi = 0; vi < kCols; ++vi) acc[vi] = B[(v0 + vi) * DK + k];
#pragma unroll 8
        for (int kp = 0; kp < DK; ++kp) {
            const float a = A[kp * DK + k];
#pragma unroll
            for (int vi = 0; vi < kCols; ++vi) acc[vi] = fmaf(a, S[vi][kp], acc[vi]);
        }
        __syncthreads();
        // the state before segment sg + 1, or, after the last segment (scan_p1 == K), the state after the launch's range
        float* out = sg + 1 < p.scan_k ? p.scan_start + ((size_t)chain * p.scan_k + sg + 1) * DV * DK : p.scan_carry_out + (size_t)chain * DV * DK;
#pragma unroll
        for (int vi = 0; vi < kCols; ++vi) {
            S[vi][k] = acc[vi];
            out[(v0 + vi) * DK + k] = acc[vi];
        }
        __syncthreads();
    }
}

}  // namespace

// A [rows][H][128] tensor of `elem`-byte elements, its rows row_bytes apart (0: dense), as (128, H, rows) with boxes of 64 rows of one
// head, 128 bytes wide.
static bool row_tensor_map(CUtensorMap* tm, const void* base, int elem, int H, long long rows, long long row_bytes = 0) {
    EncodeTiled enc = encode_tiled();
    if (enc == nullptr) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)DK, (cuuint64_t)H, (cuuint64_t)rows};
    const cuuint64_t strides[2] = {(cuuint64_t)DK * elem, row_bytes != 0 ? (cuuint64_t)row_bytes : (cuuint64_t)H * DK * elem};
    const cuuint32_t box[3] = {(cuuint32_t)(128 / elem), 1u, (cuuint32_t)CH};
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    return enc(tm, elem == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The gate rows' map, where they are on 16 bytes; else the walk reads them value by value.
static void gate_tensor_map(SpParams& p, long long rows) {
    const long long bytes = p.gate_stride * 2;
    p.gate_boxes = p.gate != nullptr && ((reinterpret_cast<uintptr_t>(p.gate) | (uintptr_t)bytes) & 15) == 0 && bytes >= (long long)p.H * DV * 2 &&
                   row_tensor_map(&p.tm_gate, p.gate, 2, p.H, rows, bytes);
}

constexpr long long kCounterBytes = kPrefillTailBytes;  // tail of the workspace: the launches' counters (kda_internal.h)

int64_t core_prefill_workspace_bytes(int32_t heads, int32_t batch, int32_t chunks_per_pass) {
    if (heads < 1 || batch < 1 || chunks_per_pass < 1) return 0;
    return (int64_t)heads * batch * chunks_per_pass * kSlotBytes + kCounterBytes;
}

// A fused launch over chunks [chunk0, chunk0 + chunks) of every sequence; pass = its number in the call.
template <bool LAYER>
static int fused_launch(SpParams& p, unsigned char* slots, unsigned int* tail, int pass, int chunks, int chunk0, cudaStream_t stream) {
    const long long chains = (long long)p.H * p.batch, items = chains * chunks, sms = sm_count(), most = items > chains ? items : chains;
    p.seg_chunks = chunks;
    p.intra_chunk0 = p.state_chunk0 = chunk0;
    p.ws_intra = p.ws_state = slots;
    p.counters = tail;
    p.sets = tail + kTailSets;
    p.ctr = pass & 1;
    p.group = (int)((chains + kTailGroups - 1) / kTailGroups);
    // A chunk of a walk takes about 0.45 of an item of a block (0.3 to 0.7 measured alike to 1 %); below four chunks a chain the blocks that stay are too
    // few items from the end of theirs to gain (4 requests x 130 rows 84.8 -> 85.9 us).
    const long long more = (chains - 1) % sms + 1;  // blocks with a chain more than the others
    const bool early = chains > sms && more < sms && chunks >= 4;
    p.early_blocks = early ? (int)more : 0;
    p.early_from = early ? items - (sms - more) * chunks * 45 / 100 : 0;
    // (The prologue in front is a plain launch: begun early too, its blocks crowd onto the SMs that come free first, 952 against
    // 921 us for 4 requests x 2,048 rows.)
    return launch_early(LAYER || p.gate != nullptr ? prefill_sp_kernel<LAYER, true, true, true> : prefill_sp_kernel<LAYER, true, LAYER, true>, (unsigned)(most < sms ? most : sms), kThreadsSp, kSmemSp, stream, p);
}

// The launches over every segment of the longest sequence, in stream order.  A workspace of two or more chunks per
// chain is split into halves so that the state role of one segment runs beside the intra role of the next; a
// workspace of one chunk per chain alternates intra-only and state-only launches.
// Two side streams and their events per device, made on the first head-sharded scan (host objects only; no device memory).
constexpr int kMaxSuperBlocks = 16;
struct SideStreams {
    cudaStream_t a = nullptr, b = nullptr;
    cudaEvent_t fork = nullptr, join_a = nullptr, join_b = nullptr, ready[kMaxSuperBlocks] = {};
};
static SideStreams* side_streams() {
    constexpr int kMaxDevices = 64;
    static SideStreams table[kMaxDevices];
    static bool made[kMaxDevices] = {};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    SideStreams& t = table[dev];
    if (!made[dev]) {
        int lo = 0, hi = 0;
        cudaDeviceGetStreamPriorityRange(&lo, &hi);  // hi is the numerically lowest = the most urgent
        bool ok = cudaStreamCreateWithPriority(&t.a, cudaStreamNonBlocking, lo) == cudaSuccess &&
                  cudaStreamCreateWithPriority(&t.b, cudaStreamNonBlocking, hi) == cudaSuccess;  // the stores go first
        ok = ok && cudaEventCreateWithFlags(&t.fork, cudaEventDisableTiming) == cudaSuccess &&
             cudaEventCreateWithFlags(&t.join_a, cudaEventDisableTiming) == cudaSuccess &&
             cudaEventCreateWithFlags(&t.join_b, cudaEventDisableTiming) == cudaSuccess;
        for (int i = 0; ok && i < kMaxSuperBlocks; ++i) ok = cudaEventCreateWithFlags(&t.ready[i], cudaEventDisableTiming) == cudaSuccess;
        if (!ok) {
            cudaGetLastError();
            return nullptr;
        }
        made[dev] = true;
    }
    return &t;
}

int core_prefill_sp_launch(int32_t heads, int32_t batch, const int32_t* cu_seqlens, int32_t max_len, const glm53f_bf16* q,
                           const glm53f_bf16* k, const glm53f_bf16* v, const float* g, const float* beta, const void* state_in,
                           void* state_out, const int64_t* state_off, bool bf16_state, const glm53f_bf16* gate,
                           const glm53f_bf16* norm_w, float eps, glm53f_bf16* out, void* workspace, int64_t workspace_bytes,
                           cudaStream_t stream, const PrefillScatter* scatter) {
    static int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        cudaError_t e = cudaSuccess;
        for (auto kernel : {prefill_sp_kernel<false, false, false, false>, prefill_sp_kernel<false, false, true, false>, prefill_sp_kernel<false, false, false, true>,
                            prefill_sp_kernel<false, false, true, true>, prefill_sp_kernel<false, true, false, true>, prefill_sp_kernel<false, true, true, true>})
            if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemSp);
        if (e != cudaSuccess) return (int)e;
        configured_dev = dev;
    }
    const long long chains = (long long)heads * batch;
    if ((reinterpret_cast<uintptr_t>(workspace) & 15) != 0 || workspace_bytes < kCounterBytes) return kInvalid;
    const long long usable = (workspace_bytes - kCounterBytes) & ~15ll;
    const long long whole = usable / (chains * kSlotBytes);
    if (whole < 1) return kInvalid;
    const bool overlap = whole >= 2;
    long long seg = overlap ? whole / 2 : whole;
    const long long need = ((long long)max_len + CH - 1) / CH;
    if (seg > need) seg = need > 0 ? need : 1;
    // One block a chain, without the workspace, where the chains have few chunks.  The lengths are not known here, and a long sequence among short ones has only its
    // own chains' blocks at work where the two roles would spread its items, so the line is where that call, too, is no slower.  us, over a workspace of 32
    // chunks / so, inputs not in L2:
    //  - every chain has an SM: up to three chunks (1 chain x 192 rows 42 / 38, with the norm 52 / 44; 64 chains + 64 of one row 47 / 38; 128 alike 61 / 40);
    //  - of more than three quarters of the SMs: four (4 chains x 256 rows + 136 of one row 45 / 42), and where one sequence's chains are more than a quarter of the
    //    SMs, five and six (39 heads, 3 sequences, one of 320 rows 50 / 50, of 384 61 / 58; 48 heads 61 / 52 and 64 / 59; 112 chains x 384 rows 78 / 60; but 4 heads, one
    //    of 35 sequences of 320 rows 46 / 48, 14 heads, one of 8 of 384 rows 45 / 53);
    //  - in a second round of more than half of the SMs: two, without the norm (256 chains x 64 rows 45 / 42, x 128 rows 60 / 58, one sequence of four that long
    //    52 / 46, 8 heads and one of 30 45 / 45; x 192 rows 69 / 73; with the norm x 128 rows 65 / 66, 192 rows 77 / 85); 192 chains x 128 rows 47 / 47, 320 65 / 66.
    const long long at_once = sm_count(), nearly_all = heads * 4ll > at_once ? 6 : 4;
    const long long chunks_alone = chains <= at_once ? (chains * 4 > 3 * at_once ? nearly_all : 3) : chains <= 2 * at_once && chains * 2 > 3 * at_once && gate == nullptr ? 2 : 0;
    if (scatter == nullptr && out != nullptr && max_len <= chunks_alone * CH)
        return core_prefill_one_launch(heads, batch, cu_seqlens, q, k, v, g, beta, state_in, state_out, state_off, bf16_state, gate, norm_w, eps, out, stream);
    SpParams p{};
    p.H = heads; p.batch = batch; p.cu = cu_seqlens;
    p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta;
    p.state_in = state_in; p.state_out = state_out;
    p.state_off = reinterpret_cast<const long long*>(state_off);
    p.state_bf16 = bf16_state ? 1 : 0;
    p.gate = gate; p.gate_stride = (long long)heads * DV; p.norm_w = norm_w; p.eps = eps; p.out = out;
    if (scatter != nullptr) {
        if (scatter->ranks < 1 || scatter->ranks > 8 || scatter->head0 < 0 || scatter->head0 + heads > scatter->heads_total) return kInvalid;
        for (int r = 0; r < scatter->ranks; ++r) {
            if (scatter->full[r] == nullptr || (reinterpret_cast<uintptr_t>(scatter->full[r]) & 15) != 0) return kInvalid;
            p.full[r] = scatter->full[r];
        }
        p.ranks = scatter->ranks; p.heads_total = scatter->heads_total; p.head0 = scatter->head0;
    } else if (out == nullptr) {
        return kInvalid;
    }
    p.seg_chunks = (int)seg;
    unsigned char* base = reinterpret_cast<unsigned char*>(workspace);
    unsigned char* half[2] = {base, overlap ? base + chains * seg * kSlotBytes : base};
    p.counters = reinterpret_cast<unsigned int*>(base + usable);
    p.status = status_word();
    if (p.status == nullptr) return (int)cudaErrorUnknown;
    // Tensor copies fetch full chunks only, whose rows the caller's metadata vouches for; the extent written into the
    // maps is the most rows the batch can hold.
    long long rows_cap = (long long)batch * max_len;
    rows_cap = rows_cap < CH ? CH : (rows_cap > 0x7fffffffll ? 0x7fffffffll : rows_cap);
    if (!row_tensor_map(&p.tm_q, q, 2, heads, rows_cap) || !row_tensor_map(&p.tm_k, k, 2, heads, rows_cap) ||
        !row_tensor_map(&p.tm_v, v, 2, heads, rows_cap) || !row_tensor_map(&p.tm_g, g, 4, heads, rows_cap))
        return (int)cudaErrorNotSupported;
    if (out != nullptr && !row_tensor_map(&p.tm_out, out, 2, heads, rows_cap)) return (int)cudaErrorNotSupported;
    gate_tensor_map(p, rows_cap);
    for (int r = 0; r < p.ranks; ++r)
        if (!row_tensor_map(&p.tm_full[r], p.full[r], 2, p.heads_total, rows_cap)) return (int)cudaErrorNotSupported;
    // U in the walk (WALK_U) from a chain on every fourth SM on: below that the walks wait for one another's products, not for memory, and SMs without a
    // chain form U for nothing.  us, 30,000 rows, workspaces of 128 chunks, U in the items / in the walk: 16 heads 876 / 957, 32 heads 1,040 / 1,080 (with the
    // norm 1,350 / 1,358), 48 heads 1,322 / 1,302 (1,541 / 1,521), 64 heads 1,753 / 1,603 (1,925 / 1,836); 64 heads x 1,000 rows 120 / 115.
    const bool walk_u = chains * 4 > sm_count();
    const auto kernel = gate != nullptr ? (walk_u ? prefill_sp_kernel<false, false, true, true> : prefill_sp_kernel<false, false, true, false>)
                                        : (walk_u ? prefill_sp_kernel<false, false, false, true> : prefill_sp_kernel<false, false, false, false>);
    cudaError_t e = cudaMemsetAsync(p.counters, 0, kCounterBytes, stream);
    if (e != cudaSuccess) return (int)e;
    const long long sms = sm_count();
    // Few chains and a long sequence: the serial walk over a chain's chunks is the critical path whatever the number of
    // idle SMs.  The recurrence is affine in the state (S_end = A S_start + B over any run of chunks), so the sequence is
    // cut into K segments that are walked at the same time: once from the zero state and once from the identity without
    // U (their end states are B and A), then, after the K - 1 compositions, once more from the true incoming states with
    // the outputs.  Needs FP32 states (a bf16 state is rounded every chunk, which is not affine) and a workspace that
    // holds every chunk of the call plus (3K - 2) states per chain.  K follows from the number of chains, the SM count and
    // the length (or GLM53F_KDA_PREFILL_SEGMENTS); the results depend on K, not otherwise on the workspace size.
    {
        long long K = 1;
        if (const char* env = getenv("GLM53F_KDA_PREFILL_SEGMENTS")) K = atoll(env);
        else if (chains <= 16) {  // measured, 2^18 tokens: 8 chains 7.5 -> 2.7 ms, 16 chains 8.4 -> 5.6, 24 (four segments) 9.2 -> 8.2, 32 (three) 10.1 -> 10.8
            const long long ka = sms / (2 * chains) + 1, kc = sms / chains;
            K = ka < kc ? ka : kc;
            if (K > 16) K = 16;
            if (K > need / 32) K = need / 32;  // a segment of fewer than 32 chunks is not worth three walks
        }
        if (K > need) K = need;
        // A head-sharded launch sends every output row to every rank, and the scan emits all outputs in its last pass: the
        // NVLink time (15 GB per GPU at 8 ranks) would follow the compute instead of running beside it.  So there the
        // sequence is cut into super-blocks, each scanned on its own: the intra role and pass 1 of super-block b + 1 run on
        // one side stream while the composition and pass 2 of super-block b -- the stores -- run on another.  Pass 2 then
        // holds SMs while it waits for the links, so it gets fewer, longer segments (K <= 48 / chains).
        // GLM53F_KDA_PREFILL_SUPERBLOCKS overrides the count (1 = off).
        long long SB = (scatter != nullptr && scatter->ranks > 1) ? 8 : 1;
        long long min_seg = 32;  // a segment of fewer than 32 chunks is not worth three walks (an override may ask for any)
        if (const char* env = getenv("GLM53F_KDA_PREFILL_SUPERBLOCKS")) {
            SB = atoll(env);
            min_seg = 1;
        }
        if (SB > kMaxSuperBlocks) SB = kMaxSuperBlocks;
        if (SB > 1 && K >= 2 && !bf16_state) {
            long long Ks = K;
            if (getenv("GLM53F_KDA_PREFILL_SEGMENTS") == nullptr && Ks > 48 / chains) Ks = 48 / chains > 2 ? 48 / chains : 2;
            while (SB > 1 && need / (SB * Ks) < min_seg) --SB;
            const long long sb = (need + SB - 1) / SB;
            // per super-block: K transitions and offsets, K incoming states, and the state after the super-block
            const long long scratch_sb = chains * (3 * Ks + 1) * (long long)(DV * DK * sizeof(float));
            SideStreams* side = SB > 1 && chains * SB * sb * kSlotBytes + SB * scratch_sb <= usable ? side_streams() : nullptr;
            if (side != nullptr) {
                if ((e = cudaEventRecord(side->fork, stream)) != cudaSuccess) return (int)e;
                cudaStreamWaitEvent(side->a, side->fork, 0);
                cudaStreamWaitEvent(side->b, side->fork, 0);
                unsigned char* scratch0 = base + chains * SB * sb * kSlotBytes;
                const float* carry = nullptr;
                for (long long b = 0; b < SB; ++b) {
                    const long long c0 = b * sb, cnt = (need - c0) < sb ? (need - c0) : sb;
                    if (cnt <= 0) break;
                    const long long Kb = cnt >= min_seg * Ks ? Ks : (cnt / min_seg > 1 ? cnt / min_seg : 1);
                    p.seg_chunks = (int)cnt;
                    p.intra_chunk0 = p.state_chunk0 = (int)c0;
                    p.ws_intra = p.ws_state = base + b * chains * sb * kSlotBytes;
                    p.ctr = (int)(b & 1);
                    p.scan_k = (int)Kb;
                    p.scan_p1 = (int)Kb;  // every segment: the state after the super-block is composed, not walked for
                    p.scan_chunks = (int)((cnt + Kb - 1) / Kb);
                    p.scan_open = (c0 + cnt >= need) ? 1 : 0;
                    p.scan_ab = reinterpret_cast<float*>(scratch0 + b * scratch_sb);
                    p.scan_start = p.scan_ab + chains * Kb * 2 * DV * DK;
                    p.scan_carry_in = carry;
                    p.scan_carry_out = p.scan_start + chains * Kb * DV * DK;
                    // one stream: everything up to the states before this super-block's segments and after it -- the intra
                    // role, both walks of every segment, the composition (which needs the previous super-block's, not its
                    // pass 2)
                    p.has_intra = 1; p.has_state = 0; p.scan_pass = 0;
                    // The intra blocks are persistent: on every SM they would keep the previous super-block's output pass,
                    // which is ready about now, off the machine until they are done, and the links idle.  From the second
                    // super-block on they leave that pass its SMs (measured on 8 GPUs, 2^20 tokens: 28.6 -> 26.1 ms).
                    const long long items = chains * cnt, room = b == 0 ? sms : (sms - Kb * chains > sms / 2 ? sms - Kb * chains : sms / 2);
                    kernel<<<(unsigned)(items < room ? items : room), kThreadsSp, kSmemSp, side->a>>>(p);
                    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
                    p.has_intra = 0; p.has_state = 1; p.scan_pass = 1;
                    kernel<<<(unsigned)(2 * Kb * chains), kThreadsSp, kSmemSp, side->a>>>(p);
                    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
                    scan_compose_kernel<<<(unsigned)(chains * (DV / kComposeCols)), 128, 0, side->a>>>(p);
                    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
                    cudaEventRecord(side->ready[b], side->a);
                    // the other: the walks with the outputs (and the stores to the peers), super-block after super-block
                    cudaStreamWaitEvent(side->b, side->ready[b], 0);
                    p.scan_pass = 2;
                    kernel<<<(unsigned)(Kb * chains), kThreadsSp, kSmemSp, side->b>>>(p);
                    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
                    carry = p.scan_carry_out;
                }
                cudaEventRecord(side->join_a, side->a);
                cudaEventRecord(side->join_b, side->b);
                cudaStreamWaitEvent(stream, side->join_a, 0);
                if ((e = cudaStreamWaitEvent(stream, side->join_b, 0)) != cudaSuccess) return (int)e;
                return 0;
            }
        }
        const long long scratch = chains * (3 * K - 2) * (long long)(DV * DK * sizeof(float));
        if (K >= 2 && !bf16_state && chains * need * kSlotBytes + scratch <= usable) {
            p.seg_chunks = (int)need;
            p.ws_intra = p.ws_state = base;
            p.intra_chunk0 = p.state_chunk0 = 0;
            p.ctr = 0;
            p.scan_k = (int)K;
            p.scan_chunks = (int)((need + K - 1) / K);
            p.scan_ab = reinterpret_cast<float*>(base + chains * need * kSlotBytes);
            p.scan_start = p.scan_ab + chains * (K - 1) * 2 * DV * DK;
            p.scan_open = 1;
            p.scan_p1 = (int)K - 1;
            p.scan_carry_in = nullptr; p.scan_carry_out = nullptr;
            p.has_intra = 1; p.has_state = 0; p.scan_pass = 0;
            const long long items = chains * need;
            kernel<<<(unsigned)(items < sms ? items : sms), kThreadsSp, kSmemSp, stream>>>(p);
            if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
            p.has_intra = 0; p.has_state = 1; p.scan_pass = 1;
            kernel<<<(unsigned)(2 * (K - 1) * chains), kThreadsSp, kSmemSp, stream>>>(p);
            if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
            scan_compose_kernel<<<(unsigned)(chains * (DV / kComposeCols)), 128, 0, stream>>>(p);
            if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
            p.scan_pass = 2;
            kernel<<<(unsigned)(K * chains), kThreadsSp, kSmemSp, stream>>>(p);
            return (int)cudaGetLastError();
        }
    }
    // More chains than SMs: the state role fills the machine by itself, there is nothing to run beside it, and a fused launch over
    // all the slots needs half as many launches as two halves that swap.  Workspaces of 32 chunks a chain: 150 chains (3 x 1,365
    // rows) 309 -> 233 us, 192 (3 x 2,731 rows) 674 -> 567, 512 (8 x 1,024 rows) 608 -> 540.
    if (chains > sms && need > 0) {
        const long long passes = (need + whole - 1) / whole, n = (need + passes - 1) / passes;
        for (long long c = 0; c < need; c += n) {
            const int rc = fused_launch<false>(p, base, p.counters, (int)(c / n), (int)n, (int)c, stream);
            if (rc != 0) return rc;
        }
        return 0;
    }
    // A workspace that holds everything is not reason enough for one segment, whose items and walks would run one after the other: from 64 chunks on two, from
    // 128 on three, where there are items enough to wait for and SMs without a chain to form the next ones.  us, one / two / three segments: 64 heads, 2,048 rows 139 / 148 / 160,
    // 4,096 rows 249 / 247 / 254, 8,192 rows 468 / 453 / 453 (with the norm 574 / 533 / 530); 32 heads, 8,192 rows 350 / 326 / 322, 12,288 rows 511 / 468 / 458;
    // 20 heads, 8,192 rows 296 / 284 / 278; 16 heads, bf16 states, 4,096 rows 156 / 151; but 72 chains of as many 275 / 277, 96 with the norm 371 / 381 / 398,
    // 8 heads, bf16 states, 8,192 rows with the norm 358 / - / 362, 4 heads, 4,096 rows 121 / 127.
    if (scatter == nullptr && chains >= 16 && chains * 9 <= 4 * sms && need >= 64) {
        const long long parts = need >= 128 ? 3 : 2, most = (need + parts - 1) / parts;
        if (seg > most) {
            seg = most;
            p.seg_chunks = (int)seg;
            half[1] = base + chains * seg * kSlotBytes;  // (a workspace of one chunk a chain has no halves, and its segments are below `most`)
        }
    }
    const long long segs = need > 0 ? (need + seg - 1) / seg : 0;
    int launch_no = 0;
    auto launch = [&](long long intra_seg, long long state_seg) -> int {
        p.has_intra = intra_seg >= 0 ? 1 : 0;
        p.has_state = state_seg >= 0 ? 1 : 0;
        p.intra_chunk0 = (int)(intra_seg * seg);
        p.state_chunk0 = (int)(state_seg * seg);
        p.ws_intra = half[intra_seg & 1];
        p.ws_state = half[state_seg & 1];
        p.ctr = launch_no++ & 1;
        long long grid = p.has_state ? chains : 0;
        if (p.has_intra) {
            const long long items = chains * seg, want = items < sms ? items : sms;
            if (grid < want) grid = want;
        }
        return launch_early(kernel, (unsigned)grid, kThreadsSp, kSmemSp, stream, p);
    };
    if (segs == 0) return launch(-1, 0);  // nothing but empty sequences: their states are copied
    if (overlap) {
        for (long long s = 0; s <= segs; ++s) {
            const int rc = launch(s < segs ? s : -1, s - 1);
            if (rc != 0) return rc;
        }
    } else {
        for (long long s = 0; s < segs; ++s) {
            int rc = launch(s, -1);
            if (rc == 0) rc = launch(-1, s);
            if (rc != 0) return rc;
        }
    }
    return 0;
}

// A pass of a layer prefill.  No halves that swap: a slot's inputs and results share its bytes, so a pass takes all the chunks
// that the workspace has slots for, both roles in one launch.
int layer_pass_launch(int32_t heads, int32_t batch, const int32_t* cu_rows, int32_t chunks, int32_t chunk0, unsigned char* slots,
                      unsigned int* tail, const void* state_in, void* state_out, const int64_t* state_off, bool bf16_state,
                      const glm53f_bf16* gate, int64_t gate_stride, const glm53f_bf16* norm_w, float eps, glm53f_bf16* out, cudaStream_t stream) {
    static int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(prefill_sp_kernel<true, true, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemSp);
        if (e != cudaSuccess) return (int)e;
        configured_dev = dev;
    }
    SpParams p{};
    p.H = heads; p.batch = batch; p.cu = cu_rows;
    p.state_in = state_in; p.state_out = state_out;
    p.state_off = reinterpret_cast<const long long*>(state_off);
    p.state_bf16 = bf16_state ? 1 : 0;
    p.gate = gate; p.gate_stride = gate_stride; p.norm_w = norm_w; p.eps = eps; p.out = out;
    p.status = status_word();
    if (p.status == nullptr) return (int)cudaErrorUnknown;
    // Only full chunks leave by tensor stores, and the metadata vouches for their rows: the map's extent bounds nothing.
    if (!row_tensor_map(&p.tm_out, out, 2, heads, 0x7fffffffll)) return (int)cudaErrorNotSupported;
    gate_tensor_map(p, 0x7fffffffll);
    return fused_launch<true>(p, slots, tail, chunk0 / chunks, chunks, chunk0, stream);
}

// ---------------------------------------------------------------------------------------------------------------------
// The same two-pass prefill for callers that may not allocate device memory at all.
//
// Some hosts of this library run inside a memory plan that is fixed before the first request: an inference engine
// whose planner has handed every byte of HBM to weights, KV pages and state arenas, or a component called from a
// region of its host where allocation is forbidden (an allocator lock held, a latency-critical loop), where cudaMalloc
// would fail, fragment the plan or stall.  Such a caller cannot produce the workspace
// glm53f_kda_core_prefill_varlen_ws asks for.  For them the library carries its own scratch: a fixed array in the
// library's device image (held by every GPU that has loaded the image until the process exits; with the runtime's
// default lazy loading the image is placed in device memory at the first call below, which is why a host makes one
// small set-up call per device before its memory plan is final), big enough for 64 workspace slots and the item counters.  Nothing in it has to start at zero: the
// intra role writes every byte of a slot that the state role reads, and each call clears the counters itself.  All calls share the one array, so two calls in flight at once (two
// streams, two threads) overwrite each other's slots; the caller serialises them.
constexpr int kStaticSlots = 64;
constexpr long long kStaticScratchBytes = (long long)kStaticSlots * kSlotBytes + kCounterBytes;  // 6,848,768 bytes
static __device__ __align__(256) unsigned char g_prefill_scratch[kStaticScratchBytes];

// The array's name is a host-side handle here, not a device address: the address a kernel can use is asked for once
// per device (with that device current) and remembered.
int core_prefill_static_launch(int32_t heads, int32_t batch, const int32_t* cu_seqlens, int32_t max_len, const glm53f_bf16* q,
                               const glm53f_bf16* k, const glm53f_bf16* v, const float* g, const float* beta, const void* state_in,
                               void* state_out, const int64_t* state_off, bool bf16_state, const glm53f_bf16* gate,
                               const glm53f_bf16* norm_w, float eps, glm53f_bf16* out, cudaStream_t stream) {
    constexpr int kMaxDevices = 64;
    static void* scratch_of[kMaxDevices] = {};
    if ((long long)heads * batch > kStaticSlots) return kInvalid;  // not even one chunk per chain would fit
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= kMaxDevices) return kInvalid;
    if (scratch_of[dev] == nullptr) {
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_prefill_scratch);
        if (e != cudaSuccess) return (int)e;
        scratch_of[dev] = ptr;
    }
    return core_prefill_sp_launch(heads, batch, cu_seqlens, max_len, q, k, v, g, beta, state_in, state_out, state_off, bf16_state,
                                  gate, norm_w, eps, out, scratch_of[dev], kStaticScratchBytes, stream);
}

int core_prefill_one_launch(int32_t heads, int32_t batch, const int32_t* cu_seqlens, const glm53f_bf16* q, const glm53f_bf16* k,
                            const glm53f_bf16* v, const float* g, const float* beta, const void* state_in, void* state_out,
                            const int64_t* state_off, bool bf16_state, const glm53f_bf16* gate, const glm53f_bf16* norm_w,
                            float eps, glm53f_bf16* out, cudaStream_t stream) {
    static int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        cudaError_t e = cudaFuncSetAttribute(prefill_one_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemOne);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(prefill_one_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemOne);
        if (e != cudaSuccess) return (int)e;
        configured_dev = dev;
    }
    SpParams p{};
    p.H = heads; p.batch = batch; p.cu = cu_seqlens;
    p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta;
    p.state_in = state_in; p.state_out = state_out;
    p.state_off = reinterpret_cast<const long long*>(state_off);
    p.state_bf16 = bf16_state ? 1 : 0;
    p.gate = gate; p.gate_stride = (long long)heads * DV; p.norm_w = norm_w; p.eps = eps; p.out = out;
    p.status = status_word();
    if (p.status == nullptr) return (int)cudaErrorUnknown;
    p.longest_first = batch > 1 && batch <= kOrderSeqs && (long long)heads * batch > sm_count() ? 1 : 0;
    constexpr long long rows_cap = 0x7fffffffll;  // only whole chunks go by the maps, and max_len is not asked for here
    if (!row_tensor_map(&p.tm_q, q, 2, heads, rows_cap) || !row_tensor_map(&p.tm_k, k, 2, heads, rows_cap) ||
        !row_tensor_map(&p.tm_v, v, 2, heads, rows_cap) || !row_tensor_map(&p.tm_g, g, 4, heads, rows_cap) || !row_tensor_map(&p.tm_out, out, 2, heads, rows_cap) ||
        (gate != nullptr && !row_tensor_map(&p.tm_gate, gate, 2, heads, rows_cap)))
        return (int)cudaErrorNotSupported;
    return launch_early(gate != nullptr ? prefill_one_kernel<true> : prefill_one_kernel<false>, (unsigned)(heads * batch), kOneThreads, kSmemOne, stream, p);
}

}  // namespace kda
