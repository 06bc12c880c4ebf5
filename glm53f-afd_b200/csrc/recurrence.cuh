// The exact recurrence step as device code: a unit's 128 x 128 state spread over sixteen warps, the delta rule, the
// read-out, and the state's way in and out of registers.  Shared by every kernel that returns the reference kernels' bits
// (files compiled with --fmad=false --ftz=false --prec-div=true --prec-sqrt=true).
//
// Warp w of a unit owns value rows 8w .. 8w+7, which never interact with the others; lane l key columns 4l .. 4l+3.
#pragma once

#include "common.cuh"

namespace kda {
namespace {

constexpr int kRecWarps = 16;                 // warps that share a unit's state
constexpr int kRowsPerLane = DV / kRecWarps;  // 8
constexpr unsigned FULL = 0xffffffffu;

// ---- packed FP32 pairs -----------------------------------------------------------------------------------------
// sm_100 has two-wide FP32 instructions (mul.f32x2, add.f32x2): each half is an IEEE round-to-nearest operation,
// so a pair gives the bits of two scalar instructions for half the issue slots (the pipe's time stays).  The state is
// held as pairs: pair jp of a lane holds value rows 2jp and 2jp+1 of its warp at one key column.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
// The product of two pairs, each half rounded once.  It is written as fma(a, b, -0) with the -0 pair read from the
// kernel's parameters: ptxas contracts a dependent mul.rn.f32x2 / add.rn.f32x2 pair into one FFMA2 even when
// contraction is off (measured: 1-ulp differences against the scalar sequence), which would break the bitwise
// contract; a product that comes out of an FMA with an addend the compiler cannot see through is left alone, and
// x*y + (-0) is x*y for every x*y, signed zeros included.
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b, f32x2 nz) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(nz));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

constexpr int kPairs = kRowsPerLane / 2;  // 4 row pairs per lane

// ---- state registers <-> shared memory -----------------------------------------------------------------------
template <typename S>
__device__ __forceinline__ void load_row(const unsigned char* slot, int row, int lane, float (&x)[4]) {
    if constexpr (sizeof(S) == 4) {
        const float4 v = *reinterpret_cast<const float4*>(slot + ((size_t)row * DK + lane * 4) * 4);
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    } else {
        const uint2 v = *reinterpret_cast<const uint2*>(slot + ((size_t)row * DK + lane * 4) * 2);
        x[0] = __uint_as_float(v.x << 16);
        x[1] = __uint_as_float(v.x & 0xffff0000u);
        x[2] = __uint_as_float(v.y << 16);
        x[3] = __uint_as_float(v.y & 0xffff0000u);
    }
}

template <typename S>
__device__ __forceinline__ void load_rows(const unsigned char* slot, int warp, int lane, f32x2 (&s)[kPairs][4]) {
#pragma unroll
    for (int jp = 0; jp < kPairs; ++jp) {
        float a[4], b[4];
        load_row<S>(slot, warp * kRowsPerLane + 2 * jp, lane, a);
        load_row<S>(slot, warp * kRowsPerLane + 2 * jp + 1, lane, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) s[jp][i] = pack2(a[i], b[i]);
    }
}

// Two floats rounded to bf16 (nearest even) in one instruction: lo in the low half.
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// P row pairs a lane: 2P value rows a warp, `warp` counting warps of that many rows.
template <typename S, int P>
__device__ __forceinline__ void store_rows_global(S* head, int warp, int lane, const f32x2 (&s)[P][4]) {
    const bool vec = (reinterpret_cast<uintptr_t>(head) & (4 * sizeof(S) - 1)) == 0;
#pragma unroll
    for (int jp = 0; jp < P; ++jp) {
        float x[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) unpack2(s[jp][i], x[0][i], x[1][i]);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            S* dst = head + (size_t)(warp * 2 * P + 2 * jp + half) * DK + lane * 4;
            if constexpr (sizeof(S) == 4) {
                if (vec) *reinterpret_cast<float4*>(dst) = make_float4(x[half][0], x[half][1], x[half][2], x[half][3]);
                else
#pragma unroll
                    for (int i = 0; i < 4; ++i) dst[i] = x[half][i];
            } else {
                const uint32_t lo = pack_bf16x2(x[half][0], x[half][1]), hi = pack_bf16x2(x[half][2], x[half][3]);
                if (vec) *reinterpret_cast<uint2*>(dst) = make_uint2(lo, hi);
                else {
                    uint16_t* d = reinterpret_cast<uint16_t*>(dst);
                    d[0] = (uint16_t)lo; d[1] = (uint16_t)(lo >> 16); d[2] = (uint16_t)hi; d[3] = (uint16_t)(hi >> 16);
                }
            }
        }
    }
}

// A bf16 state's rounding between two rows of a window: every element to bf16 and back.
template <int P>
__device__ __forceinline__ void round_rows(f32x2 (&s)[P][4]) {
#pragma unroll
    for (int jp = 0; jp < P; ++jp)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float a, b;
            unpack2(s[jp][i], a, b);
            const uint32_t r = pack_bf16x2(a, b);
            s[jp][i] = pack2(__uint_as_float(r << 16), __uint_as_float(r & 0xffff0000u));
        }
}

// The 32-lane xor butterfly (offsets 16, 8, 4, 2, 1) of eight independent values per lane, evaluated as a
// reduce-scatter.  Lane l returns the butterfly's result for value (l >> 2); the additions and their pairing are
// those of `x += shfl_xor(x, o)` applied to each value, so the bits are the same.
__device__ __forceinline__ float butterfly8(const float (&p)[kRowsPerLane], int lane) {
    float r[4], t[2];
    {
        const bool up = (lane & 16) != 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float mine = up ? p[4 + j] : p[j];
            const float give = up ? p[j] : p[4 + j];
            r[j] = mine + __shfl_xor_sync(FULL, give, 16);
        }
    }
    {
        const bool up = (lane & 8) != 0;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float mine = up ? r[2 + j] : r[j];
            const float give = up ? r[j] : r[2 + j];
            t[j] = mine + __shfl_xor_sync(FULL, give, 8);
        }
    }
    const bool up = (lane & 4) != 0;
    float x = (up ? t[1] : t[0]) + __shfl_xor_sync(FULL, up ? t[0] : t[1], 4);
    x = x + __shfl_xor_sync(FULL, x, 2);
    x = x + __shfl_xor_sync(FULL, x, 1);
    return x;
}

// The same for N values (2 ... 32): lane l returns the butterfly's result for value l / (32 / N).
template <int N>
__device__ __forceinline__ float butterfly_of(const float (&v)[N], int lane, int offset = 16) {
    if constexpr (N == 1) {
        float x = v[0];
        for (; offset; offset >>= 1) x = x + __shfl_xor_sync(FULL, x, offset);
        return x;
    } else {
        const bool up = (lane & offset) != 0;
        float r[N / 2];
#pragma unroll
        for (int j = 0; j < N / 2; ++j) r[j] = (up ? v[N / 2 + j] : v[j]) + __shfl_xor_sync(FULL, up ? v[j] : v[N / 2 + j], offset);
        return butterfly_of<N / 2>(r, lane, offset >> 1);
    }
}

// Dot products of the lane's eight rows with a key-channel vector x (both halves of x2[i] hold x[i]): per row the
// lane's four channels added in order from zero, then the butterfly.  Lane l gets row (l >> 2).
template <int P>
__device__ __forceinline__ void rows_partial(const f32x2 (&s)[P][4], const f32x2 (&x2)[4], float* part, f32x2 nz) {
#pragma unroll
    for (int jp = 0; jp < P; ++jp) {
        f32x2 acc = mul2(s[jp][0], x2[0], pack2(0.0f, 0.0f));  // the product plus the sum's starting zero, in one instruction
#pragma unroll
        for (int i = 1; i < 4; ++i) acc = add2(acc, mul2(s[jp][i], x2[i], nz));
        unpack2(acc, part[2 * jp], part[2 * jp + 1]);
    }
}
__device__ __forceinline__ float rows_dot(const f32x2 (&s)[kPairs][4], const f32x2 (&x2)[4], int lane, f32x2 nz) {
    float part[kRowsPerLane];
    rows_partial(s, x2, part, nz);
    return butterfly8(part, lane);
}

// The plain butterfly for one value per lane (norms).
__device__ __forceinline__ float butterfly1(float x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x = x + __shfl_xor_sync(FULL, x, o);
    return x;
}

// One delta-rule step on a lane's 8 x 4 tile (reference kda.cu:38-53): decay, read with k, correct toward v.
// `v_mine` is v at the value row lane l reduces: row (l >> 2) of the warp's eight.
__device__ __forceinline__ void delta_rule_v(f32x2 (&s)[kPairs][4], const f32x2 (&kk)[4], const f32x2 (&gg)[4], float v_mine, int lane,
                                             float beta, f32x2 nz) {
#pragma unroll
    for (int jp = 0; jp < kPairs; ++jp)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[jp][i] = mul2(s[jp][i], gg[i], nz);
    const float kv = rows_dot(s, kk, lane, nz);
    const float mine = (v_mine - kv) * beta;
#pragma unroll
    for (int jp = 0; jp < kPairs; ++jp) {
        const f32x2 delta = pack2(__shfl_sync(FULL, mine, 8 * jp), __shfl_sync(FULL, mine, 8 * jp + 4));
#pragma unroll
        for (int i = 0; i < 4; ++i) s[jp][i] = add2(s[jp][i], mul2(kk[i], delta, nz));
    }
}
__device__ __forceinline__ void delta_rule(f32x2 (&s)[kPairs][4], const f32x2 (&kk)[4], const f32x2 (&gg)[4],
                                           const float* vrow, int warp, int lane, float beta, f32x2 nz) {
    delta_rule_v(s, kk, gg, vrow[warp * kRowsPerLane + (lane >> 2)], lane, beta, nz);
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

template <typename S, int P>
__device__ __forceinline__ void load_rows_global(const S* head, int warp, int lane, f32x2 (&s)[P][4]) {
    const bool vec = (reinterpret_cast<uintptr_t>(head) & (4 * sizeof(S) - 1)) == 0;
#pragma unroll
    for (int jp = 0; jp < P; ++jp) {
        float x[2][4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const S* src = head + (size_t)(warp * 2 * P + 2 * jp + half) * DK + lane * 4;
            if constexpr (sizeof(S) == 4) {
                if (vec) {
                    const float4 v = *reinterpret_cast<const float4*>(src);
                    x[half][0] = v.x; x[half][1] = v.y; x[half][2] = v.z; x[half][3] = v.w;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[half][i] = src[i];
                }
            } else {
                uint32_t lo, hi;
                if (vec) {
                    const uint2 v = *reinterpret_cast<const uint2*>(src);
                    lo = v.x; hi = v.y;
                } else {
                    const uint16_t* u = reinterpret_cast<const uint16_t*>(src);
                    lo = (uint32_t)u[0] | ((uint32_t)u[1] << 16);
                    hi = (uint32_t)u[2] | ((uint32_t)u[3] << 16);
                }
                x[half][0] = __uint_as_float(lo << 16);
                x[half][1] = __uint_as_float(lo & 0xffff0000u);
                x[half][2] = __uint_as_float(hi << 16);
                x[half][3] = __uint_as_float(hi & 0xffff0000u);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) s[jp][i] = pack2(x[0][i], x[1][i]);
    }
}

}  // namespace
}  // namespace kda
