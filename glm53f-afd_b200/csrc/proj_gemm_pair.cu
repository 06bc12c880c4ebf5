// The projection GEMM for many rows on SM pairs: out[g][r][o] = sum_k x[g][r][k] * w[g][o][k] with tiles of 256 features x NR
// rows computed by tcgen05.mma.cta_group::2, NR a multiple of 16 up to 256 chosen per launch.
//
// Why a pair.  With one block per tile (proj_gemm.cu) a 128 x 256 tile reads 48 KiB of operands from L2 per 4.2 MFLOP;
// the tensor pipe then waits on the copies a quarter of the time.  Two blocks of a cluster that share a 256 x 256 tile
// read 32 KiB each for the same work: each loads its own 128 weight rows and HALF of the activation rows, and the
// pair's MMA reads the activation halves from both blocks' shared memory.
//
// Protocol (block 0 of the pair leads):
//   producer (warp 0, both blocks)  tensor copies of the block's weight tile and its half of the rows into its own
//                                   ring; the copies of BOTH blocks complete the LEADER's stage barrier;
//   MMA (warp 1 of the leader)      one thread issues the pair's MMAs (M = 256, N = NR, K = 16) and commits each stage
//                                   to both blocks' `empty` barriers, each finished accumulator to both `acc_full` barriers;
//   epilogue (warps 2-9, both)      each block drains its own 128 features x NR rows from its tensor memory, through
//                                   shared memory (transposing matrix stores; rows of 64 features leave as
//                                   tiled tensor stores), and arrives on the leader's `acc_empty`.
// The epilogue's way out was what bounded wide launches: with two-byte stores straight from the registers a 256 x 256 tile
// took 17 us to leave, as long as a k of 4,096 takes to compute, and the k = 128 gate factor (67 MB of results at 2,048 rows)
// ran at 0.5 TB/s.
//
// A launch carries up to two independent problems (their tiles in one list): the 4096 -> 256 first gate factor has one feature
// tile and is all latency by itself (114 us at 2,048 rows as its own K-split launch); beside the fused [q|k|v|b] projection
// of the same rows it is one tile column more.
//
// K segments.  A shape whose small launches split k over a cluster (proj_gemm.cu) adds its partial sums in f32 in split order;
// a row's bits must not depend on the launch's row count, so here such a shape's tile runs its k in the same segments, each
// into a fresh accumulator, and the epilogue adds them in the same order (kept in registers: NR <= kPairSplitRows then;
// the sums of more than 128 rows do not quite fit, so launches with such tiles have an instance of the kernel to themselves).
//
// Tensor memory is allocated by both blocks together (512 columns: two accumulators).  Every wait is bounded (codes
// 140-143); both blocks reach the collective TMEM release and the closing cluster barrier on every path.

#include <cuda.h>

#include "common.cuh"
#include "glm53f_proj.h"
#include "kda_internal.h"
#include "proj_gemm.cuh"
#include "tc.cuh"

namespace kda {
namespace {

constexpr int kPM = 128;           // features per block (256 per pair)
constexpr int kPN = 256;           // rows per tile at most (half of them loaded by each block)
constexpr int kPK = 64;
constexpr int kPairThreads = 320;  // producer, MMA, eight epilogue warps
constexpr int kPairStages = 6;
constexpr int kPairABytes = kPM * 128, kPairBBytes = (kPN / 2) * 128;
constexpr int kPairStageBytes = kPairABytes + kPairBBytes;  // 32 KiB
constexpr int kPairTmemCols = 512;
// Output staging: two buffers per pair of epilogue warps, each two boxes of 16 rows x 64 features in the 128-byte swizzle.
// (NR is a multiple of 16, not of 32; a fence and two barriers per sixteen rows were most of the epilogue's time.)
constexpr int kBoxRows = 16, kChunk = 2 * kBoxRows, kOutBuf = kChunk * 128;
constexpr int oPairOut = kPairStages * kPairStageBytes;
constexpr int oPairBars = oPairOut + 8 * kOutBuf;
constexpr int oPairCtl = oPairBars + (2 * kPairStages + 4) * 8;
constexpr int kPairSmem = oPairCtl + 16 + 1024;
static_assert(kPairSmem <= 232448, "shared memory budget");

enum : int { kStatusPairEmpty = 140, kStatusPairFull = 141, kStatusPairAccFull = 142, kStatusPairAccEmpty = 143 };

__device__ __forceinline__ uint32_t pair_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void pair_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t pair_addr(const void* local, uint32_t rank) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(local)), "r"(rank));
    return ra;
}
__device__ __forceinline__ void pair_mbar_arrive(uint32_t remote_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
// A tiled tensor copy into this block's shared memory whose completion is counted on `bar_addr`, a barrier of this
// block or of its pair (a shared::cluster address).
__device__ __forceinline__ void pair_tensor_load(void* smem_dst, const void* tmap, int x, int y, int z, uint32_t bar_addr) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_addr), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void pair_tmem_alloc(uint32_t* smem_result, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// Issued by the whole warp with `leader` set in one lane: the operands then stay in uniform registers.  (Inside an `if` of one
// lane the compiler moves every operand of every MMA over from the lane's registers: about 90 cycles an instruction, 360 of
// the 590 cycles a stage took.)
__device__ __forceinline__ void pair_mma(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate), "r"(leader)
        : "memory");
}
// The barrier at this shared-memory offset in BOTH blocks completes once the pair's MMAs issued so far by this thread have
// (one commit with a block mask instead of one per block).
__device__ __forceinline__ void pair_commit(uint32_t leader, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
        "h"((uint16_t)3), "r"(leader)
        : "memory");
}

struct PairParams {
    PairProblem problem[kPairProblems];
    long long tiles0, tiles;  // the first problem's tiles, all tiles
    int* status;
};

// Tile t of the launch: its problem and its place there (row tiles fastest: pairs that run together share a weight tile in L2).
struct PairTile {
    const PairProblem& q;
    int rt, nt, g;
};
__device__ __forceinline__ PairTile pair_tile(const PairParams& p, long long t) {
    const bool second = t >= p.tiles0;
    const PairProblem& q = p.problem[second ? 1 : 0];
    const int i = (int)(second ? t - p.tiles0 : t), u = i / q.r_tiles;
    return {q, i - u * q.r_tiles, u % q.n_tiles, u / q.n_tiles};
}

// SPLIT_ROWS: rows per tile at most where k runs in segments.
template <int SPLIT_ROWS>
__global__ void __launch_bounds__(kPairThreads, 1) proj_gemm_pair_kernel(const __grid_constant__ PairParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + oPairBars);   // used in the leader: both blocks' copies
    uint64_t* empty = full + kPairStages;                            // in each block: the pair's MMAs are done with the stage
    uint64_t* acc_full = empty + kPairStages;                        // in each block
    uint64_t* acc_empty = acc_full + 2;                              // used in the leader: both blocks' epilogues
    volatile uint32_t* ctl = reinterpret_cast<volatile uint32_t*>(smem + oPairCtl);
    uint32_t* tmem_slot = const_cast<uint32_t*>(ctl) + 2;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = pair_rank();
    const long long tile0 = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
    if (tid == 0) {
        for (int i = 0; i < kPairStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 16);  // eight epilogue warps of each block
        }
        ctl[0] = 0u;
        ctl[1] = 0u;
        mbar_init_fence();
    }
    __syncthreads();
    pair_sync_all();  // the pair's barriers exist before either block touches the other's
    if (warp == 1) pair_tmem_alloc(tmem_slot, kPairTmemCols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = *tmem_slot;
    const WaitCtx ctx{ctl, ctl + 1, p.status};
    // Programmatic dependent launch: nothing global is touched before the kernels ahead have finished.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            for (long long t = tile0; t < p.tiles; t += tile_step) {
                const PairTile x = pair_tile(p, t);
                const int half = x.q.row_tile / 2;
                const int f0 = x.nt * 2 * kPM + (int)rank * kPM, r0 = x.rt * x.q.row_tile + (int)rank * half;
                const void *mw = &x.q.tm_w, *mx = &x.q.tm_x; const int nkb = x.q.kblocks; const uint32_t tx = 2u * (uint32_t)(kPairABytes + half * 128);
                const int wy = x.q.w_swapped ? x.g : f0, wz = x.q.w_swapped ? f0 : x.g, xy = x.q.x_swapped ? x.g : r0, xz = x.q.x_swapped ? r0 : x.g;
                const uint32_t bar0 = pair_addr(&full[0], 0);
                for (int kb = 0; kb < nkb; ++kb) {
                    if (!mbar_wait(&empty[s], ph ^ 1u, ctx, kStatusPairEmpty)) goto done;
                    unsigned char* st = smem + s * kPairStageBytes;
                    if (rank == 0) mbar_arrive_expect_tx(&full[s], tx);
                    pair_tensor_load(st, mw, kb * kPK, wy, wz, bar0 + 8 * s);
                    pair_tensor_load(st + kPairABytes, mx, kb * kPK, xy, xz, bar0 + 8 * s);
                    if (++s == kPairStages) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t leader = tc::elect_one();
            int s = 0, buf = 0;
            uint32_t ph = 0, acc_ph[2] = {0, 0};
            for (long long t = tile0; t < p.tiles; t += tile_step) {
                const PairTile x = pair_tile(p, t);
                const uint32_t idesc = tc::idesc_bf16(2 * kPM, 0, 0, 0, 0) | ((uint32_t)(x.q.row_tile >> 3) << 17);
                const int segments = x.q.segments, seg_kb = x.q.kblocks / segments;
                for (int seg = 0; seg < segments; ++seg) {
                    if (!tc::warp_all(mbar_wait(&acc_empty[buf], acc_ph[buf] ^ 1u, ctx, kStatusPairAccEmpty))) goto done;
                    tc::fence_after_sync();
                    const uint32_t d = tm + (uint32_t)(buf * kPN);
                    for (int kb = 0; kb < seg_kb; ++kb) {
                        if (!tc::warp_all(mbar_wait(&full[s], ph, ctx, kStatusPairFull))) goto done;
                        tc::fence_after_sync();
                        const unsigned char* st = smem + s * kPairStageBytes;
#pragma unroll
                        for (int i = 0; i < kPK / 16; ++i)
                            pair_mma(leader, d, tc::desc_sw128_kmajor(st, kPM, 16 * i), tc::desc_sw128_kmajor(st + kPairABytes, kPN / 2, 16 * i), idesc, kb > 0 || i > 0);
                        pair_commit(leader, &empty[s]);
                        if (++s == kPairStages) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                    pair_commit(leader, &acc_full[buf]);
                    acc_ph[buf] ^= 1u;
                    buf ^= 1;
                    if (leader) ctl[0] = ctl[0] + 1u;
                }
            }
        }
    } else {
        const int q = warp & 3;                             // the TMEM lane quarter this warp may read
        const int set = (warp - 2) >> 2;                    // two sets of four warps share a tile's rows, 32 at a time in turn
        const int side = q >> 1, fl = (q & 1) * 32 + lane;  // feature fl of the block's 64-feature box `side`
        const int bar = 1 + set * 2 + side;                 // the two warps that fill a box together
        unsigned char* boxes = smem + oPairOut + (set * 2 + side) * 2 * kOutBuf;
        const bool issuer = (q & 1) == 0 && lane == 0;      // issues the boxes' tensor stores
        int buf = 0, out_buf = 0;
        uint32_t acc_ph[2] = {0, 0};
        // Sixteen rows of the accumulator from c0 on.  For tensor stores in the fragment layout, from which transposing matrix stores put rows of eight
        // features into the boxes: v[8 h + 4 g + 2 p + e] = feature 16 h + 8 p + lane / 4 of the warp, row c0 + 8 g + 2 (lane % 4) + e.  (With lane = feature, 32
        // two-byte stores where four are enough now: the k = 128 gate factor at 512 rows
        // 13.8 -> 12.5 us, at 1,024 24.5 -> 21.3.)  Else lane = feature, v[j] = row c0 + j; and so in the instance that keeps the sums of more than 128 rows,
        // whose registers are full (o_proj at 513, 660 and 768 rows 40.6, 43.4 and 44.6 us, from fragments 45.9, 48.8 to 52.4 and 51.0 to 56.9).
        constexpr bool kFragments = SPLIT_ROWS <= 128;
        auto load = [&](const PairTile& x, int c0, float* v) {
            uint32_t r[16];
            if (x.q.tensor_out) {
                uint32_t a[8], b[8];
                tc::tmem_ld_frag(tc::tmem_addr(tm, q, buf * kPN + c0), a);
                tc::tmem_ld_frag(tc::tmem_addr(tm, q, buf * kPN + c0) + (16u << 16), b);
                tc::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) r[j] = a[j], r[8 + j] = b[j];
            } else {
                tc::tmem_ld16(tc::tmem_addr(tm, q, buf * kPN + c0), r);
                tc::tmem_ld_wait();
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
        };
        // The tile's rows c0 .. c0 + 31 (those below row_tile) out, as load() gave them.
        auto emit = [&](const PairTile& x, int c0, const float (&v)[kChunk]) {
            const long long row0 = (long long)x.rt * x.q.row_tile + c0;
            const int f0 = x.nt * 2 * kPM + (int)rank * kPM + side * 64;
            if (row0 >= x.q.rows) return;  // the whole chunk is past the last row (the same for every thread)
            if (x.q.tensor_out) {
                unsigned char* box = boxes + out_buf * kOutBuf;
                out_buf ^= 1;
                if (issuer) bulk_wait_read<1>();  // this buffer's last stores have been read
                named_bar_sync(bar, 64);
                if constexpr (kFragments) {
                    // A lane names row lane % 8 of matrix lane / 8: features 8 ((lane / 8) % 2), rows 8 (lane / 16) of the sixteen by sixteen.
                    const int row = (lane >> 4) * 8 + (lane & 7), piece = (q & 1) * 4 + ((lane >> 3) & 1);
#pragma unroll
                    for (int c = 0; c < 2; ++c)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float* w = v + 16 * c + 8 * h;
                            tc::stmatrix_t4(box + (16 * c + row) * 128 + (((piece + 2 * h) ^ (row & 7)) << 4), tc::bf16x2(w[0], w[1]), tc::bf16x2(w[2], w[3]),
                                            tc::bf16x2(w[4], w[5]), tc::bf16x2(w[6], w[7]));
                        }
                } else {
#pragma unroll
                    for (int j = 0; j < kChunk; j += 2) {
                        const uint32_t two = tc::bf16x2(v[j], v[j + 1]);
                        *reinterpret_cast<uint16_t*>(box + j * 128 + (((fl >> 3) ^ (j & 7)) << 4) + (fl & 7) * 2) = (uint16_t)two;
                        *reinterpret_cast<uint16_t*>(box + (j + 1) * 128 + (((fl >> 3) ^ ((j + 1) & 7)) << 4) + (fl & 7) * 2) = (uint16_t)(two >> 16);
                    }
                }
                fence_proxy_async_smem();
                named_bar_sync(bar, 64);
                if (issuer) {
                    if (f0 < x.q.n)  // features and rows past the extents are clipped by the copy
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            if (c0 + half * kBoxRows >= x.q.row_tile || row0 + half * kBoxRows >= x.q.rows) break;
                            const void* src = box + half * kBoxRows * 128;
                            if (x.q.out_swapped) tensor_store_3d(&x.q.tm_out, f0, x.g, (int)row0 + half * kBoxRows, src);
                            else tensor_store_3d(&x.q.tm_out, f0, (int)row0 + half * kBoxRows, x.g, src);
                        }
                    bulk_commit();
                }
            } else if (f0 + fl < x.q.n) {
                unsigned char* base = reinterpret_cast<unsigned char*>(x.q.out) + ((long long)x.g * x.q.o_gstride + f0 + fl) * (x.q.out_f32 ? 4 : 2);
#pragma unroll
                for (int j = 0; j < kChunk; ++j) {
                    const long long row = row0 + j;
                    if (row < x.q.rows && c0 + j < x.q.row_tile) {
                        if (x.q.out_f32) *reinterpret_cast<float*>(base + row * x.q.ldo * 4) = v[j];
                        else *reinterpret_cast<uint16_t*>(base + row * x.q.ldo * 2) = f32_to_bf16_bits(v[j]);
                    }
                }
            }
        };
        auto release = [&] {
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                if (rank == 0) mbar_arrive(&acc_empty[buf]);
                else pair_mbar_arrive(pair_addr(&acc_empty[buf], 0));
                ctl[0] = ctl[0] + 1u;
            }
            buf ^= 1;
        };
        for (long long t = tile0; t < p.tiles; t += tile_step) {
            const PairTile x = pair_tile(p, t);
            // The warps of a box meet at its barrier: they decide together whether an accumulator came.
            auto arrived = [&] {
                const bool ok = mbar_wait(&acc_full[buf], acc_ph[buf], ctx, kStatusPairAccFull);
                acc_ph[buf] ^= 1u;
                const bool all = named_bar_all(bar, 64, ok);
                tc::fence_after_sync();
                return all;
            };
            if (x.q.segments == 1) {
                if (!arrived()) goto done;
                for (int c0 = set * kChunk; c0 < x.q.row_tile; c0 += 2 * kChunk) {
                    float v[kChunk];
                    if constexpr (kFragments) {
                        load(x, c0, v);
                        load(x, c0 + 16, v + 16);
                    } else {
                        uint32_t r[kChunk];
                        tc::tmem_ld32(tc::tmem_addr(tm, q, buf * kPN + c0), r);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < kChunk; ++j) v[j] = __uint_as_float(r[j]);
                    }
                    emit(x, c0, v);
                }
                release();
            } else {
                float sum[SPLIT_ROWS / kChunk / 2][kChunk];
                for (int seg = 0; seg < x.q.segments; ++seg) {
                    if (!arrived()) goto done;
#pragma unroll
                    for (int c = 0; c < SPLIT_ROWS / kChunk / 2; ++c) {
                        const int c0 = (2 * c + set) * kChunk;
                        if (c0 >= x.q.row_tile) break;
#pragma unroll
                        for (int j0 = 0; j0 < kChunk; j0 += 16) {
                            if constexpr (kFragments) {
                                float r[16];
                                load(x, c0 + j0, r);
#pragma unroll
                                for (int j = 0; j < 16; ++j) sum[c][j0 + j] = seg == 0 ? r[j] : sum[c][j0 + j] + r[j];
                            } else {
                                uint32_t r[16];
                                tc::tmem_ld16(tc::tmem_addr(tm, q, buf * kPN + c0 + j0), r);
                                tc::tmem_ld_wait();
#pragma unroll
                                for (int j = 0; j < 16; ++j) sum[c][j0 + j] = seg == 0 ? __uint_as_float(r[j]) : sum[c][j0 + j] + __uint_as_float(r[j]);
                            }
                        }
                    }
                    release();
                }
#pragma unroll
                for (int c = 0; c < SPLIT_ROWS / kChunk / 2; ++c) {
                    const int c0 = (2 * c + set) * kChunk;
                    if (c0 >= x.q.row_tile) break;
                    emit(x, c0, sum[c]);
                }
            }
        }
        if (issuer) bulk_wait_all<0>();
    }
done:
    // After an abort, copies into this block's shared memory may still be in flight: give them a bounded time.
    if (ctl[1]) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 2000000ull) {
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    pair_sync_all();  // neither block releases tensor memory or leaves while the pair's MMAs or arrivals may still touch it
    if (warp == 1) pair_tmem_dealloc(tm, kPairTmemCols);
    pair_sync_all();
}

}  // namespace

int proj_gemm_pair_launch(const PairProblem* problems, int n, int* status, cudaStream_t stream) {
    bool wide = false;  // tiles of more than 128 rows in segments: 7 % slower a tile than the narrow instance
    for (int i = 0; i < n; ++i) wide = wide || (problems[i].segments > 1 && problems[i].row_tile > 128);
    auto* kernel = wide ? proj_gemm_pair_kernel<kPairSplitRows> : proj_gemm_pair_kernel<128>;
    static int configured_dev[2] = {-1, -1};
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev[wide] != dev) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem);
        if (e != cudaSuccess) return (int)e;
        configured_dev[wide] = dev;
    }
    PairParams p{};
    for (int i = 0; i < n; ++i) p.problem[i] = problems[i];
    p.tiles0 = problems[0].tiles;
    p.tiles = p.tiles0 + (n > 1 ? problems[1].tiles : 0);
    p.status = status;
    const long long pairs_cap = sm_count() / 2;
    const long long pairs = p.tiles < pairs_cap ? p.tiles : pairs_cap;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(pairs * 2));
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = kPairSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1 + early_attribute(attr[1]);
    return (int)cudaLaunchKernelEx(&cfg, kernel, p);
}

}  // namespace kda
