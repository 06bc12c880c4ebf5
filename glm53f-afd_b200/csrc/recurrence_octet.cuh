// The exact recurrence step of recurrence.cuh with EIGHT lanes to a value row, for kernels in which many warps of several units share an
// SM (the core entry points' exact verify, the commit replay of many units, the exact prefill of several prompts).
//
// The reference forms a sum over the 128 key channels as a warp does: a lane adds its four consecutive channels (a leaf) in order
// from zero, then the xor butterfly 16, 8, 4, 2, 1 adds the 32 leaves.  Here lane 8g + j holds leaves j, j + 8, j + 16 and j + 24 of R
// rows, so that the butterfly's first two levels are additions within the thread and only three cross lanes.  Same additions,
// same pairing, hence the same bits.  A warp owns 4R consecutive value rows, rows gR .. gR + R - 1 of them with lane group g.
//
// What bounds it: no unit is full.  Seven separately rounded operations a state element and row are 896 cycles of an SM's 128 lanes, and
// two-wide instructions halve the issue slots, not the pipe's time; with four warps a scheduler the FP32 pipe is 59 % active, issue 69 to
// 74 %, and warps wait for the pipe, for their turn and for fixed latencies about equally.  With a row's 32 leaves in 32 lanes a unit
// and row cost 1,340 issue slots a scheduler: 18 shuffles and 8 broadcasts for eight rows, and 24 moves that double k, decay and q.  Here 8 shuffles
// and 4 broadcasts for sixteen rows (R = 4), and k, decay and q are used in the pairs in which they lie, for four times the
// shared-memory reads.  Exact verify and replay of 48 slots x up to 16 rows x 34 layers: 11.16 -> 10.04 ms.  With few warps an SM the
// reads' latency shows instead (one prompt of 701 rows: 405 against 417 us; the replay of few units, launch_replay_small), so the
// others keep the layout of recurrence.cuh.
#pragma once

#include "recurrence.cuh"

namespace kda {
namespace {
namespace oct {

constexpr int kLeaves = 4, kRowPairs = 2 * kLeaves;  // of a row in a thread: pair 2b + i holds channels 4(j + 8b) + 2i and the next

__device__ __forceinline__ f32x2 widen2(uint32_t w) { return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }

// Four leaves of a row of 128 floats (k, decay, q), 16-byte aligned.
__device__ __forceinline__ void load_leaves(const float* row, int lane, f32x2 (&x)[kRowPairs]) {
#pragma unroll
    for (int b = 0; b < kLeaves; ++b) {
        const ulonglong2 v = reinterpret_cast<const ulonglong2*>(row)[(lane & 7) + 8 * b];
        x[2 * b] = v.x;
        x[2 * b + 1] = v.y;
    }
}

// Asynchronous copies of a thread's piece of a row into shared memory, in groups.
__device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---- state registers <-> global memory -------------------------------------------------------------------------
// `head` is the unit's [128][128] state, `warp` counts warps of 4R rows.  A leaf is 16 (f32) or 8 (bf16) contiguous bytes, a
// lane group's eight a run of 128 or 64.
template <typename S, int R>
__device__ __forceinline__ void load_rows(const S* head, int warp, int lane, f32x2 (&s)[R][kRowPairs]) {
    const bool vec = (reinterpret_cast<uintptr_t>(head) & (4 * sizeof(S) - 1)) == 0;
    const S* at = head + (size_t)(warp * 4 * R + (lane >> 3) * R) * DK + (lane & 7) * 4;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int b = 0; b < kLeaves; ++b) {
            const S* src = at + r * DK + 32 * b;
            if constexpr (sizeof(S) == 4) {
                if (vec) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src);
                    s[r][2 * b] = v.x;
                    s[r][2 * b + 1] = v.y;
                } else {
                    s[r][2 * b] = pack2(src[0], src[1]);
                    s[r][2 * b + 1] = pack2(src[2], src[3]);
                }
            } else {
                uint2 v;
                if (vec) {
                    v = *reinterpret_cast<const uint2*>(src);
                } else {
                    const uint16_t* u = reinterpret_cast<const uint16_t*>(src);
                    v = make_uint2((uint32_t)u[0] | ((uint32_t)u[1] << 16), (uint32_t)u[2] | ((uint32_t)u[3] << 16));
                }
                s[r][2 * b] = widen2(v.x);
                s[r][2 * b + 1] = widen2(v.y);
            }
        }
}

// A pair rounded to bf16 (nearest even) in one instruction: lo in the low half.
__device__ __forceinline__ uint32_t round2(f32x2 x) {
    float lo, hi;
    unpack2(x, lo, hi);
    return pack_bf16x2(lo, hi);
}

template <typename S, int R>
__device__ __forceinline__ void store_rows(S* head, int warp, int lane, const f32x2 (&s)[R][kRowPairs]) {
    const bool vec = (reinterpret_cast<uintptr_t>(head) & (4 * sizeof(S) - 1)) == 0;
    S* at = head + (size_t)(warp * 4 * R + (lane >> 3) * R) * DK + (lane & 7) * 4;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int b = 0; b < kLeaves; ++b) {
            S* dst = at + r * DK + 32 * b;
            if constexpr (sizeof(S) == 4) {
                if (vec) {
                    *reinterpret_cast<ulonglong2*>(dst) = make_ulonglong2(s[r][2 * b], s[r][2 * b + 1]);
                } else {
                    float x[4];
                    unpack2(s[r][2 * b], x[0], x[1]);
                    unpack2(s[r][2 * b + 1], x[2], x[3]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) dst[i] = x[i];
                }
            } else {
                const uint32_t lo = round2(s[r][2 * b]), hi = round2(s[r][2 * b + 1]);
                if (vec) {
                    *reinterpret_cast<uint2*>(dst) = make_uint2(lo, hi);
                } else {
                    uint16_t* d = reinterpret_cast<uint16_t*>(dst);
                    d[0] = (uint16_t)lo; d[1] = (uint16_t)(lo >> 16); d[2] = (uint16_t)hi; d[3] = (uint16_t)(hi >> 16);
                }
            }
        }
}

// A bf16 state's rounding between two rows of a window: every element to bf16 and back.
template <int R>
__device__ __forceinline__ void round_rows(f32x2 (&s)[R][kRowPairs]) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < kRowPairs; ++i) s[r][i] = widen2(round2(s[r][i]));
}

// ---- the step ------------------------------------------------------------------------------------------------------
// A thread's share of the dot products of its rows with x: each leaf in order from zero (the first product takes the zero
// along as its addend, so that a negative zero becomes the sum's positive one), then the butterfly's levels 16 and 8.
template <int R>
__device__ __forceinline__ void rows_partial(const f32x2 (&s)[R][kRowPairs], const f32x2 (&x)[kRowPairs], float* part, f32x2 nz) {
    float z, negative;
    unpack2(nz, z, negative);
    const f32x2 from_zero = pack2(0.0f, negative);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        float leaf[kLeaves];
#pragma unroll
        for (int b = 0; b < kLeaves; ++b) {
            float p0, p1, p2, p3;
            unpack2(mul2(s[r][2 * b], x[2 * b], from_zero), p0, p1);
            unpack2(mul2(s[r][2 * b + 1], x[2 * b + 1], nz), p2, p3);
            leaf[b] = ((p0 + p1) + p2) + p3;
        }
        part[r] = (leaf[0] + leaf[2]) + (leaf[1] + leaf[3]);
    }
}
// The warp's value row whose sums a lane receives (8 / R neighbouring lanes to a row).
template <int R>
__device__ __forceinline__ int row_of_lane(int lane) { return lane / (8 / R); }
template <int R>
__device__ __forceinline__ bool first_of_row(int lane) { return (lane & (8 / R - 1)) == 0; }
template <int R>
__device__ __forceinline__ float rows_dot(const f32x2 (&s)[R][kRowPairs], const f32x2 (&x)[kRowPairs], int lane, f32x2 nz) {
    float part[R];
    rows_partial(s, x, part, nz);
    return butterfly_of<R>(part, lane, 4);
}
template <int R>
__device__ __forceinline__ void decay_rows(f32x2 (&s)[R][kRowPairs], const f32x2 (&gg)[kRowPairs], f32x2 nz) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < kRowPairs; ++i) s[r][i] = mul2(s[r][i], gg[i], nz);
}
// `d` is (v - k-product) * beta of the lane's group's row r in its lane r * STEP.
template <int R, int STEP>
__device__ __forceinline__ void update_rows(f32x2 (&s)[R][kRowPairs], const f32x2 (&kk)[kRowPairs], float d, int lane, f32x2 nz) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float x = __shfl_sync(FULL, d, (lane & 24) + r * STEP);
        const f32x2 delta = pack2(x, x);
#pragma unroll
        for (int i = 0; i < kRowPairs; ++i) s[r][i] = add2(s[r][i], mul2(kk[i], delta, nz));
    }
}
// Reference kda.cu:38-53: decay, read with k, correct toward v.  `v_mine` is v at the value row whose sums the lane receives.
template <int R>
__device__ __forceinline__ void delta_rule(f32x2 (&s)[R][kRowPairs], const f32x2 (&kk)[kRowPairs], const f32x2 (&gg)[kRowPairs], float v_mine,
                                           int lane, float beta, f32x2 nz) {
    decay_rows(s, gg, nz);
    update_rows<R, 8 / R>(s, kk, (v_mine - rows_dot(s, kk, lane, nz)) * beta, lane, nz);
}

}  // namespace oct
}  // namespace
}  // namespace kda
