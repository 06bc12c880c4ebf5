// The projections either side of the KDA core as a tcgen05 GEMM: out[g][r][o] = sum_k x[g][r][k] * w[g][o][k], bf16
// operands, f32 accumulation in tensor memory, bf16 or f32 results.
//
// What it stands in for: the reference's Gemm::bf16 (crates/glm53f-forward/src/gemm.rs:212-235), which sends up to 8
// rows to its CUDA-core GEMV (kernels/glm53f_forward.h:19-40) and more rows to cuBLAS, at the call sites of a KDA
// layer (crates/glm53f-forward/src/forward.rs:3494-3542: the fused [q|k|v|b] projection 4096 -> 24,640 and the
// low-rank gate pair 4096 -> 256 -> 2 x 8192; 3772-3790: o_proj 8192 -> 4096).
//
// Shape of the kernel.  The weight is the M operand: a tile is 128 output features x NR activation rows, NR in
// {16, 32, 64, 96} chosen from the row count (more rows: proj_gemm_pair.cu), so a decode step's 16 rows waste nothing and the weight -- which
// dominates the traffic at few rows (202 MB for the fused projection) -- streams through once.  Both operands are
// K-major in global memory ([o][k] and [r][k]), so tiled tensor copies in the 128-byte swizzle feed tcgen05.mma
// in place: a stage is 64 k of the weight tile (16 KiB) and of the row tile (NR x 128 bytes).  Roles per block:
//   warp 0  producer: tensor copies into a ring of stages, each completing a stage's mbarrier;
//   warp 1  issues 4 MMAs (K = 16) per stage, the warp converged and one lane elected (tc::mma_bf16_if), and commits the stage
//           back to the producer, and the tile's accumulator to the epilogue when its last stage is in; owns the TMEM allocation;
//   warps 2-5  epilogue: tcgen05.ld of the finished accumulator (lane = feature, column = row), convert, store.
// Two accumulators alternate, so the epilogue of a tile overlaps the MMAs of the next; blocks walk the tile list with
// the row tile fastest (blocks that run together share a weight tile in L2).  A block stays under
// 113 KiB of shared memory so that two fit an SM and every tile of a decode-size launch is in flight at once
// (measured for the fused projection at 16 rows, 193 tiles: 38 us so, 48 us with one deeper-ringed block per SM).
//
// A row's result depends on that row's inputs and on (n, k) only -- the accumulation order over k is fixed by the
// stage loop -- never on how many rows the launch has or which NR it picked (tests hold this bitwise).
//
// Few tiles (o_proj at decode: 32 feature tiles of k = 8192) would leave most SMs idle: there the k range of a tile is
// split over the blocks of a thread-block cluster, each with its own accumulator, and the blocks add the partial tiles,
// each for some of the rows, in rank order through distributed shared memory (no scratch in global memory, the same bits every run).
//
// Two GEMMs that do not depend on one another share a launch without clusters where that is the shorter way (share_launch): a tile list for both, and a
// split k is summed part after part by the tile's one block, the sums in tensor memory behind the two accumulators.  The same bits.
//
// Every wait is bounded (codes 130-135 in the device status word); TMEM is freed on every path; every block of a
// cluster reaches the closing cluster barrier on every path.

#include <cuda.h>


#include "common.cuh"
#include "glm53f_proj.h"
#include "kda_internal.h"
#include "proj_gemm.cuh"
#include "tc.cuh"
#include "tensor_map.cuh"

namespace kda {
namespace {

constexpr int kBM = 128;            // output features per tile (UMMA M)
constexpr int kBK = 64;             // k per stage: one 128-byte swizzle row of bf16
constexpr int kGemmThreads = 192;   // producer, MMA, 4 epilogue warps
constexpr int kEpiThreads = 128;
constexpr int kABytes = kBM * 128;  // a stage's weight tile
constexpr int kBlocksPerSm = 2;     // of any tile

enum : int { kStatusGemmEmpty = 130, kStatusGemmFull = 131, kStatusGemmAccFull = 132, kStatusGemmAccEmpty = 133, kStatusGemmRedFull = 134, kStatusGemmRedEmpty = 135 };

template <int NR, bool SPLIT, bool TWO = false>
struct Cfg {
    static constexpr int kBBytes = NR * 128;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kStages = SPLIT ? (NR == 16 ? 5 : NR == 32 ? 4 : 3) : (NR == 16 ? 6 : NR == 32 ? 5 : NR <= 64 ? 4 : 3);
    // Tensor memory columns: two accumulators kAcc apart and (TWO) the sums of a split k.  With tiles of more than 64 rows there are no columns left for those where
    // two blocks share an SM: the parts then come one after the other in one accumulator, the sums lie in the other.
    static constexpr int kAcc = NR <= 64 ? NR : 128;
    static constexpr bool kApart = NR <= 64;
    static constexpr int kTmemCols = TWO && kApart ? 4 * kAcc : 2 * kAcc;
    static constexpr int kRedBytes = SPLIT ? kBM * NR * 4 : 0;  // this block's partial tile, f32 [NR][128]
    static constexpr int oRed = kStages * kStageBytes;
    static constexpr int oBars = oRed + kRedBytes;  // full[S], empty[S], acc_full[2], acc_empty[2], red_full, red_empty
    static constexpr int oCtl = oBars + (2 * kStages + 6) * 8;
    static constexpr int kBytes = oCtl + 16 + 1024;      // + slack to align the stages to 1024 bytes
};

struct GemmProblem {
    CUtensorMap tm_w, tm_x;
    void* out;
    long long ldo, o_gstride;
    int rows, n, kblocks, out_f32;
    int segments;              // without a cluster: k runs in so many equal parts, each a sum of its own
    int n_tiles, r_tiles;
    int w_swapped, x_swapped;  // the map's coordinates are (k, group, row) instead of (k, row, group)
};
struct GemmParams {
    GemmProblem problem[2];    // the second: none, or (without clusters) another GEMM's tiles behind the first's
    long long tiles0, tiles;
    int overlap;  // 0: alone; 1: the first of two independent launches; 2: the second (see glm53f_kda_proj_bf16_many)
    int* status;
};

// ---- thread-block clusters: the K splits of a tile are the blocks of one cluster --------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void prefetch_tensormap(const void* tmap) { asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory"); }
// Programmatic dependent launch: the next kernel of the stream may be scheduled once every block has said so, and a
// block touches nothing an earlier kernel may still write (or read, where this kernel writes) before grid_dependency_wait.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of this block's shared-memory location `local` in block `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_smem(const void* local, uint32_t rank) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(local)), "r"(rank));
    return ra;
}
__device__ __forceinline__ void peer_mbar_arrive(uint32_t remote_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
__device__ __forceinline__ void fence_cluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }

__device__ __forceinline__ float peer_load(uint32_t remote_addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote_addr) : "memory");
    return v;
}

// Tile t of the launch: its problem and its place there, the row tile fastest.
struct GemmTile {
    const GemmProblem& q;
    int rt, nt, g;
};
template <bool TWO>
__device__ __forceinline__ GemmTile gemm_tile(const GemmParams& p, long long t) {
    const bool second = TWO && t >= p.tiles0;
    const GemmProblem& q = p.problem[second ? 1 : 0];
    const long long i = second ? t - p.tiles0 : t, u = i / q.r_tiles;
    return {q, (int)(i % q.r_tiles), (int)(u % q.n_tiles), (int)(u / q.n_tiles)};
}

// KS = blocks per cluster = K splits of a tile (1: no cluster).  TWO: two problems, KS = 1 (an instance to itself: reading the parameters by a tile's problem
// and the sums of a split k cost a launch of one 1 to 3 us).
template <int NR, int KS, bool TWO>
__global__ void __launch_bounds__(kGemmThreads, kBlocksPerSm) proj_gemm_kernel(const __grid_constant__ GemmParams p) {
    constexpr bool SPLIT = KS > 1;
    static_assert(!SPLIT || !TWO, "");
    using C = Cfg<NR, SPLIT, TWO>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::oBars);
    uint64_t* empty = full + C::kStages;
    uint64_t* acc_full = empty + C::kStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* red_full = acc_empty + 2;   // every block's partial of this tile is in its buffer
    uint64_t* red_empty = red_full + 1;   // every block has read this block's partial
    constexpr uint32_t ks = KS;
    const uint32_t kr = SPLIT ? cluster_rank() : 0u;
    const long long tile0 = blockIdx.x / ks, tile_step = gridDim.x / ks;
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + C::oCtl);
    uint32_t* tmem_slot = const_cast<uint32_t*>(ctl) + 2;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < C::kStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], kEpiThreads / 32);
        }
        mbar_init(red_full, ks * (kEpiThreads / 32));
        mbar_init(red_empty, ks * (kEpiThreads / 32));
        ctl[0] = 0u;
        ctl[1] = 0u;
        mbar_init_fence();
    }
    if (warp == 1) tc::tmem_alloc(tmem_slot, C::kTmemCols);
    if (tid == 0) {
        const GemmProblem& q = gemm_tile<TWO>(p, tile0).q;
        prefetch_tensormap(&q.tm_w);
        prefetch_tensormap(&q.tm_x);
    }
    tc::fence_before_sync();
    __syncthreads();
    // Every block's barriers exist before a peer arrives on one: the blocks say so here and check it only before their
    // first remote arrival (the end of their first tile), so nobody stands still at the start.
    if (SPLIT) cluster_arrive();
    tc::fence_after_sync();
    const uint32_t tm = *tmem_slot;
    const WaitCtx ctx{ctl, ctl + 1, p.status};
    bool opened = !SPLIT;  // whether this thread has completed the opening cluster barrier
    // Before the first global access: an earlier kernel may be writing the weight or the rows.  Of two independent launches the
    // first lets the second in only once the kernels before both have finished, and the second does not wait for the first
    // until its own end, where whatever follows it expects both to be done.
    if (p.overlap == 0) launch_dependents();
    if (p.overlap != 2) grid_dependency_wait();
    if (p.overlap != 0) launch_dependents();

    if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            for (long long t = tile0; t < p.tiles; t += tile_step) {
                const GemmTile x = gemm_tile<TWO>(p, t);
                const int kb_n = x.q.kblocks / (int)ks, kb0 = (int)kr * kb_n;
                const void *mw = &x.q.tm_w, *mx = &x.q.tm_x;
                const bool ws = x.q.w_swapped != 0, xs = x.q.x_swapped != 0;
                for (int kb = kb0; kb < kb0 + kb_n; ++kb) {
                    if (!mbar_wait(&empty[s], ph ^ 1u, ctx, kStatusGemmEmpty)) goto done;
                    unsigned char* st = smem + s * C::kStageBytes;
                    mbar_arrive_expect_tx(&full[s], C::kStageBytes);
                    tensor_load_3d(st, mw, kb * kBK, ws ? x.g : x.nt * kBM, ws ? x.nt * kBM : x.g, &full[s]);
                    tensor_load_3d(st + kABytes, mx, kb * kBK, xs ? x.g : x.rt * NR, xs ? x.rt * NR : x.g, &full[s]);
                    if (++s == C::kStages) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // The whole warp runs this loop and one lane issues (tc::mma_bf16_if): operands stay in uniform registers.
        constexpr uint32_t idesc = tc::idesc_bf16(kBM, NR, 0, 0, 0);
        const uint32_t leader = tc::elect_one();
        int s = 0, buf = 0;
        uint32_t ph = 0, acc_ph[2] = {0, 0};
        for (long long t = tile0; t < p.tiles; t += tile_step) {
            const GemmProblem& q = gemm_tile<TWO>(p, t).q;
            const int segments = TWO ? q.segments : 1, kb_n = q.kblocks / (SPLIT ? (int)ks : segments);
            for (int seg = 0; seg < segments; ++seg) {
                if (!tc::warp_all(mbar_wait(&acc_empty[buf], acc_ph[buf] ^ 1u, ctx, kStatusGemmAccEmpty))) goto done;
                tc::fence_after_sync();
                const uint32_t d = tm + (uint32_t)(buf * C::kAcc);
                for (int kb = 0; kb < kb_n; ++kb) {
                    if (!tc::warp_all(mbar_wait(&full[s], ph, ctx, kStatusGemmFull))) goto done;
                    tc::fence_after_sync();
                    const unsigned char* st = smem + s * C::kStageBytes;
#pragma unroll
                    for (int i = 0; i < kBK / 16; ++i)
                        tc::mma_bf16_if(leader, d, tc::desc_sw128_kmajor(st, kBM, 16 * i), tc::desc_sw128_kmajor(st + kABytes, NR, 16 * i), idesc, kb > 0 || i > 0);
                    tc::mma_commit_if(leader, &empty[s]);
                    if (++s == C::kStages) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                tc::mma_commit_if(leader, &acc_full[buf]);
                acc_ph[buf] ^= 1u;
                if (C::kApart || segments == 1) buf ^= 1;
                if (leader) ctl[0] = ctl[0] + 1u;
            }
        }
    } else {
        const int q = warp & 3;  // the TMEM lane quarter this warp may read
        int buf = 0;
        uint32_t acc_ph[2] = {0, 0}, red_ph = 0;
        for (long long t = tile0; t < p.tiles; t += tile_step) {
            const GemmTile tile = gemm_tile<TWO>(p, t);
            const GemmProblem& x = tile.q;
            if (!mbar_wait(&acc_full[buf], acc_ph[buf], ctx, kStatusGemmAccFull)) goto done;
            acc_ph[buf] ^= 1u;
            tc::fence_after_sync();
            const int fl = q * 32 + lane, f = tile.nt * kBM + fl;
            const bool f_ok = f < x.n;
            const long long row0 = (long long)tile.rt * NR;
            const long long ldo = x.ldo;
            const int rows = x.rows, out_f32 = x.out_f32;
            unsigned char* base = reinterpret_cast<unsigned char*>(x.out) + ((long long)tile.g * x.o_gstride + f) * (out_f32 ? 4 : 2);
            auto store = [&](int c, float v) {
                const long long row = row0 + c;
                if (f_ok && row < rows) {
                    if (out_f32) *reinterpret_cast<float*>(base + row * ldo * 4) = v;
                    else *reinterpret_cast<uint16_t*>(base + row * ldo * 2) = f32_to_bf16_bits(v);
                }
            };
            auto release = [&] {
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[buf]);
            };
            if constexpr (!SPLIT) {
                if (!TWO || x.segments == 1) {
#pragma unroll 1
                    for (int c0 = 0; c0 < NR; c0 += 16) {
                        uint32_t r[16];
                        tc::tmem_ld16(tc::tmem_addr(tm, q, buf * C::kAcc + c0), r);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) store(c0 + j, __uint_as_float(r[j]));
                    }
                    release();
                } else {  // the parts of k, added in their order
                    for (int seg = 0; seg < x.segments; ++seg) {
                        if (seg > 0) {
                            if (C::kApart) buf ^= 1;
                            if (!mbar_wait(&acc_full[buf], acc_ph[buf], ctx, kStatusGemmAccFull)) goto done;
                            acc_ph[buf] ^= 1u;
                            tc::fence_after_sync();
                        }
                        const int sums = C::kApart ? 2 * C::kAcc : (buf ^ 1) * C::kAcc;
#pragma unroll 1
                        for (int c0 = 0; c0 < NR; c0 += 16) {
                            uint32_t r[16], sum[16];
                            tc::tmem_ld16(tc::tmem_addr(tm, q, buf * C::kAcc + c0), r);
                            if (seg > 0) tc::tmem_ld16(tc::tmem_addr(tm, q, sums + c0), sum);
                            tc::tmem_ld_wait();
                            if (seg > 0)
#pragma unroll
                                for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(sum[j]) + __uint_as_float(r[j]));
                            if (seg + 1 < x.segments) {
                                tc::tmem_st16(tc::tmem_addr(tm, q, sums + c0), r);
                            } else {
#pragma unroll
                                for (int j = 0; j < 16; ++j) store(c0 + j, __uint_as_float(r[j]));
                            }
                        }
                        tc::tmem_st_wait();
                        release();
                    }
                    if (!C::kApart) buf ^= 1;  // (back at the end: the next tile takes the same accumulator)
                }
            } else {
                // The tile's K splits live in the blocks of this cluster.  Every block parks its partial tile in its own shared
                // memory and then finishes NR / KS of the tile's rows: it adds the blocks' partials in rank order (a fixed order:
                // the same bits every time) through distributed shared memory, and stores.  (With rank 0 alone adding everything
                // a launch of 64 rows of the 4096 -> 256 factor took 25 us.)
                constexpr int CW = NR / KS;
                float* red = reinterpret_cast<float*>(smem + C::oRed) + fl;  // [NR rows][128 features]
                if (!opened) {  // the opening cluster barrier: every peer's barriers and buffers exist
                    cluster_wait();
                    opened = true;
                }
                if (!mbar_wait(red_empty, red_ph ^ 1u, ctx, kStatusGemmRedEmpty)) goto done;  // the last tile's partial has been read
                fence_cluster();
#pragma unroll 1
                for (int c0 = 0; c0 < NR; c0 += 16) {
                    uint32_t r[16];
                    tc::tmem_ld16(tc::tmem_addr(tm, q, buf * C::kAcc + c0), r);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) red[(c0 + j) * kBM] = __uint_as_float(r[j]);
                }
                tc::fence_before_sync();
                fence_cluster();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[buf]);
                if (lane < KS) peer_mbar_arrive(peer_smem(red_full, lane));
                if (!mbar_wait(red_full, red_ph, ctx, kStatusGemmRedFull)) goto done;
                fence_cluster();
                float v[CW][KS];
#pragma unroll
                for (uint32_t r = 0; r < ks; ++r) {
                    const uint32_t remote = peer_smem(red + kr * CW * kBM, r);
#pragma unroll
                    for (int c = 0; c < CW; ++c) v[c][r] = peer_load(remote + (uint32_t)(c * kBM * 4));
                }
#pragma unroll
                for (int c = 0; c < CW; ++c) {
                    float sum = v[c][0];
#pragma unroll
                    for (uint32_t r = 1; r < ks; ++r) sum = sum + v[c][r];
                    store((int)kr * CW + c, sum);
                }
                fence_cluster();
                __syncwarp();
                if (lane < KS) peer_mbar_arrive(peer_smem(red_empty, lane));
                red_ph ^= 1u;
            }
            buf ^= 1;
        }
    }
done:
    // After an abort, copies into this block's shared memory may still be in flight: give them a bounded time.
    if (ctl[1]) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 2000000ull) {
        }
    }
    if (p.overlap == 2) grid_dependency_wait();
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tm, C::kTmemCols);
    // No block leaves while a peer may still read its partial tile or arrive on its barriers.
    if (SPLIT) {
        if (!opened) cluster_wait();  // the threads that never needed the opening barrier complete it here
        cluster_sync_all();
    }
}

constexpr int kFewRows = 96;        // launches of up to this many rows run here, larger ones on SM pairs (a layer's four at 80 rows 75.4 us, on pairs 77.9; at 128 with tiles
                                    // of 128 rows, which leave the sums of a split k no columns of their own, 80.0 and 79.5)
// ... and a K-split shape by itself up to here: its splits run side by side on a cluster, on a pair one after another (o_proj at
// 128 rows: 36 us on pairs, 24 so)
constexpr int kFewRowsSplit = 128;
constexpr int kSplitRowsMax = 512;  // ... and every launch of up to this many keeps the K split's summation order (see k_segments)

// A [groups][rows][k] bf16 matrix (row stride ld, group stride gstride, in elements) as a 3-D map with boxes of
// 64 k x box_rows rows in the 128-byte swizzle; rows past the extent read as zero.  The dimensions are ordered by
// stride -- (k, rows, groups), or (k, groups, rows) when the groups interleave inside a row (`swapped`).
bool matrix_map(CUtensorMap* tm, int* swapped, const void* base, long long k, long long rows, long long groups, long long ld, long long gstride,
                int box_rows, int box_k = kBK) {
    EncodeTiled enc = encode_tiled();
    if (enc == nullptr) return false;
    const long long gs = groups > 1 ? gstride : rows * ld;
    *swapped = groups > 1 && gs < ld;
    if (groups > 1 && !*swapped && gs < rows * ld) return false;  // neither nesting: not a layout the callers have
    const cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)(*swapped ? groups : rows), (cuuint64_t)(*swapped ? rows : groups)};
    const cuuint64_t strides[2] = {(cuuint64_t)(*swapped ? gs : ld) * 2, (cuuint64_t)(*swapped ? ld : gs) * 2};
    const cuuint32_t box[3] = {(cuuint32_t)box_k, *swapped ? 1u : (cuuint32_t)box_rows, *swapped ? (cuuint32_t)box_rows : 1u};
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// K splits for a launch of few tiles (little n, deep k: o_proj at decode): the largest of 8, 4, 2 that divides the
// k blocks into runs of at least four and still leaves every block of a one-row-tile launch resident at once.  It is
// a function of (n, k, groups) alone in all launches of up to 512 rows (beyond 96 rows, 128 for a split k by itself, the same parts of k are summed
// in the same order on SM pairs), so a row's bits do not depend on `rows` there.  Measured for
// o_proj at 16 rows (32 tiles): no split 40.7 us, 2 splits 27.1, 4 splits 20.9, 8 splits (two waves of clusters) 24.7.
int pick_ksplit(long long tiles, int kblocks, long long resident) {
    for (int s = 8; s >= 2; s >>= 1)
        if (kblocks % s == 0 && kblocks / s >= 4 && tiles * s <= resident) return s;
    return 1;
}

template <int NR, int KS, bool TWO = false>
int launch_one(GemmParams& p, long long clusters, cudaStream_t stream) {
    using C = Cfg<NR, (KS > 1), TWO>;
    static int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(proj_gemm_kernel<NR, KS, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kBytes);
        if (e != cudaSuccess) return (int)e;
        configured_dev = dev;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(clusters * KS));
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = C::kBytes;
    cfg.stream = stream;
    // Programmatic stream serialization: the kernel waits for its predecessors itself (grid_dependency_wait) before its
    // first global access, so its blocks' set-up (barriers, tensor memory, descriptor fetch) overlaps their tail.
    cudaLaunchAttribute attr[2];
    unsigned na = early_attribute(attr[0]);
    if (KS > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)KS;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return (int)cudaLaunchKernelEx(&cfg, proj_gemm_kernel<NR, KS, TWO>, p);
}

// The GEMM `j` as a launch's problem with tiles of nr rows; its tiles, 0 where it has no such form.
long long few_rows_problem(GemmProblem& q, const glm53f_proj_job& j, int nr) {
    q.out = j.out;
    q.ldo = j.ldo;
    q.o_gstride = j.groups > 1 ? j.o_gstride : 0;
    q.rows = j.rows;
    q.n = j.n;
    q.kblocks = j.k / kBK;
    q.out_f32 = j.out_f32 != 0;
    // The split is chosen for ONE row tile, whatever the launch's row count: a row's bits then depend on (groups, n, k) only.
    q.n_tiles = (j.n + kBM - 1) / kBM;
    q.r_tiles = (j.rows + nr - 1) / nr;
    q.segments = pick_ksplit((long long)j.groups * q.n_tiles, q.kblocks, sm_count());  // clusters were measured at one block per SM
    if (!matrix_map(&q.tm_w, &q.w_swapped, j.w, j.k, j.n, j.groups, j.ldw, j.w_gstride, kBM) ||
        !matrix_map(&q.tm_x, &q.x_swapped, j.x, j.k, j.rows, j.groups, j.ldx, j.x_gstride, nr))
        return 0;
    return (long long)j.groups * q.n_tiles * q.r_tiles;
}

// One GEMM, or (b) two that share a launch without clusters.
template <int NR>
int launch_gemm(GemmParams& p, const glm53f_proj_job& a, const glm53f_proj_job* b, cudaStream_t stream) {
    p.tiles = p.tiles0 = few_rows_problem(p.problem[0], a, NR);
    if (p.tiles0 == 0) return (int)cudaErrorNotSupported;
    const long long cap = (long long)sm_count() * kBlocksPerSm;
    if (b != nullptr) {
        const long long more = few_rows_problem(p.problem[1], *b, NR);
        if (more == 0) return (int)cudaErrorNotSupported;
        p.tiles += more;
        return launch_one<NR, 1, true>(p, p.tiles < cap ? p.tiles : cap, stream);
    }
    const int ks = p.problem[0].segments;
    const long long fit = cap / ks;
    const long long clusters = p.tiles < fit ? p.tiles : fit;
    if constexpr (NR <= 64) {
        if (ks == 8) return launch_one<NR, 8>(p, clusters, stream);
        if (ks == 4) return launch_one<NR, 4>(p, clusters, stream);
        if (ks == 2) return launch_one<NR, 2>(p, clusters, stream);
    }
    return launch_one<NR, 1>(p, clusters, stream);
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Rows per tile of a launch on SM pairs: the multiple of 16 with the least time by the counts of the machine.  A stage of 64 k
// takes a pair 2 NR cycles of tensor pipe and 16 KiB + 64 NR bytes per block through a port of about 60 bytes a cycle; a tile
// costs about 1,500 cycles beside its stages, or its epilogue (500 cycles for 64 rows) where that is longer; pairs take
// tiles in rounds.  (At 333 rows of the fused projection: two tiles of 176 rows, 194 of them in three rounds.)
int pick_row_tile(long long feature_tiles, int rows, int kblocks, int most) {
    const long long pairs = sm_count() / 2;
    int best = most;
    double least = 1e30;
    for (int nr = 16; nr <= most; nr += 16) {
        const long long r_tiles = (rows + nr - 1) / nr, rounds = (feature_tiles * r_tiles + pairs - 1) / pairs;
        const double load = (16384.0 + 64.0 * nr) / 60.0, mma = 2.0 * nr, stages = kblocks * (load > mma ? load : mma), out = (nr + 63) / 64 * 500.0;
        const double time = (double)rounds * ((stages > out ? stages : out) + 1500.0);
        if (time < least * 0.999) {
            least = time;
            best = nr;
        }
        if (r_tiles == 1) break;
    }
    return best;
}

// The parts k is summed in.  Above 512 rows a launch whose tiles of 128 features x 256 rows fill the GPU runs k in one go; the others
// keep the parts of a small launch, and with them its bits (the 4096 -> 256 factor at any row count, o_proj up to 1,024 rows: 41 to
// 44 us for 513 to 768 rows and 64 us for 1,024, against 38 to 41 and 50 in one go).
int k_segments(const glm53f_proj_job& j) {
    const long long feature_tiles = (long long)j.groups * ((j.n + kBM - 1) / kBM);
    if (j.rows > kSplitRowsMax && feature_tiles * ((j.rows + 255) / 256) >= sm_count()) return 1;
    return pick_ksplit(feature_tiles, j.k / kBK, sm_count());
}

bool pair_problem(PairProblem& q, const glm53f_proj_job& j) {
    q = PairProblem{};
    q.out = j.out;
    q.ldo = j.ldo;
    q.o_gstride = j.groups > 1 ? j.o_gstride : 0;
    q.rows = j.rows;
    q.n = j.n;
    q.kblocks = j.k / kBK;
    q.out_f32 = j.out_f32 != 0;
    q.segments = k_segments(j);
    q.n_tiles = (j.n + 2 * kBM - 1) / (2 * kBM);
    // Segmented tiles of more than 128 rows have a slower instance of the kernel: only where one round of them replaces two or more.
    q.row_tile = pick_row_tile((long long)j.groups * q.n_tiles, j.rows, q.kblocks, q.segments == 1 ? 256 : j.rows > kSplitRowsMax ? kPairSplitRows : 128);
    q.r_tiles = (j.rows + q.row_tile - 1) / q.row_tile;
    q.tiles = (long long)j.groups * q.n_tiles * q.r_tiles;
    if (q.tiles > 0x3fffffff) return false;
    if (!matrix_map(&q.tm_w, &q.w_swapped, j.w, j.k, j.n, j.groups, j.ldw, j.w_gstride, kBM) ||
        !matrix_map(&q.tm_x, &q.x_swapped, j.x, j.k, j.rows, j.groups, j.ldx, j.x_gstride, q.row_tile / 2))
        return false;
    // bf16 rows that start on 16 bytes leave as tensor stores (boxes of 64 features x 16 rows).
    q.tensor_out = !q.out_f32 && aligned16(j.out) && j.ldo % 8 == 0 && (j.groups == 1 || (j.o_gstride % 8 == 0 && j.o_gstride > 0)) &&
                   matrix_map(&q.tm_out, &q.out_swapped, j.out, j.n, j.rows, j.groups, j.ldo, j.o_gstride, 16, 64);
    return true;
}

// Whether the arguments are those of a GEMM the kernels take (kInvalid otherwise); rows == 0 needs no pointers.
int check_job(const glm53f_proj_job& j) {
    if (j.groups < 1 || j.rows < 0 || j.n < 1 || j.k < kBK || j.k % kBK || j.n % 8 || j.ldx % 8 || j.ldw % 8 || j.ldx < j.k || j.ldw < j.k || j.ldo < j.n)
        return kInvalid;
    if (j.groups > 1 && (j.x_gstride % 8 || j.w_gstride % 8 || j.x_gstride < 0 || j.w_gstride < 0 || j.o_gstride < 0)) return kInvalid;
    if (j.rows == 0) return 0;
    if (!j.x || !j.w || !j.out || !aligned16(j.x) || !aligned16(j.w) || (reinterpret_cast<uintptr_t>(j.out) & (j.out_f32 ? 3 : 1))) return kInvalid;
    return 0;
}

int few_rows(const glm53f_proj_job& a, const glm53f_proj_job* b, int overlap, int* status, cudaStream_t stream) {
    GemmParams p{};
    p.overlap = overlap;
    p.status = status;
    const int rows = b != nullptr && b->rows > a.rows ? b->rows : a.rows;
    if (rows <= 16) return launch_gemm<16>(p, a, b, stream);
    if (rows <= 32) return launch_gemm<32>(p, a, b, stream);
    if (rows <= 64 || (b == nullptr && k_segments(a) > 1)) return launch_gemm<64>(p, a, b, stream);
    return launch_gemm<96>(p, a, b, stream);
}

// Whether two GEMMs of few rows are one launch, the parts of a split k one after another in one block each: where one of them has tiles enough by itself
// and the other one's are no longer than its.  (As two launches side by side, the second not waiting for the first, the 4096 -> 256 factor cost nearly all of
// its own time beside the fused projection: both and the second factor 45.5 us at 16 rows, 41.2 so; 58.5 and 46.6 at 64.)
bool share_launch(const glm53f_proj_job& a, const glm53f_proj_job& b) {
    const int ka = k_segments(a), kb = k_segments(b);
    return (ka == 1 && b.k <= a.k) || (kb == 1 && a.k <= b.k);
}

}  // namespace
}  // namespace kda

extern "C" int32_t glm53f_kda_proj_bf16_many(const glm53f_proj_job* jobs, int32_t count, glm53f_stream_t stream) {
    using namespace kda;
    if (!jobs || count < 0) return kInvalid;
    for (int i = 0; i < count; ++i)
        if (check_job(jobs[i]) != 0) return kInvalid;
    int* status = status_word();
    if (status == nullptr) return (int)cudaErrorUnknown;
    for (int i = 0; i < count; ++i) {
        const glm53f_proj_job& j = jobs[i];
        if (j.rows == 0) continue;
        const bool two = i + 1 < count && jobs[i + 1].rows > 0 && (jobs[i + 1].rows <= kFewRows) == (j.rows <= kFewRows);
        int rc = 0;
        if (j.rows <= kFewRows || (!two && j.rows <= kFewRowsSplit && k_segments(j) > 1)) {
            const bool share = two && share_launch(j, jobs[i + 1]);
            rc = few_rows(j, share ? &jobs[i + 1] : nullptr, two && !share ? 1 : 0, status, stream);
            if (rc == 0 && two && !share) rc = few_rows(jobs[i + 1], nullptr, 2, status, stream);
            i += two ? 1 : 0;
        } else {
            PairProblem q[kPairProblems];
            if (!pair_problem(q[0], j) || (two && !pair_problem(q[1], jobs[i + 1]))) return (int)cudaErrorNotSupported;
            rc = proj_gemm_pair_launch(q, two ? 2 : 1, status, stream);
            i += two ? 1 : 0;
        }
        if (rc != 0) return rc;
    }
    return 0;
}

extern "C" int32_t glm53f_kda_proj_bf16(const uint16_t* x, int64_t ldx, int64_t x_gstride, const uint16_t* w, int64_t ldw, int64_t w_gstride,
                                        int32_t groups, int32_t rows, int32_t n, int32_t k, void* out, int32_t out_f32, int64_t ldo,
                                        int64_t o_gstride, glm53f_stream_t stream) {
    const glm53f_proj_job job{x, ldx, x_gstride, w, ldw, w_gstride, groups, rows, n, k, out, out_f32, ldo, o_gstride};
    const int rc = kda::check_job(job);
    return rc != 0 || rows == 0 ? rc : glm53f_kda_proj_bf16_many(&job, 1, stream);
}
