// Pieces of the chunk-64 tensor-core prefill kernels: the chunk geometry, the cell helpers and the FP32 triangular inverse.
#pragma once

#include "common.cuh"
#include "tc.cuh"

namespace kda {
namespace pf {

constexpr int CH = 64;            // rows per chunk
constexpr int kCompute = 512;     // 16 compute warps: warp w reaches TMEM lanes 32*(w%4).., and takes columns 32*(w/4)..
constexpr int kTile = CH * 16 * 16;  // 16 KiB: 64 rows x 128 bf16
// The column sides of L and M, one tile per row block I (rows 0 .. 16 I + 15, 256 bytes a row); the per-block decay factor tables (14 x 128
// floats: E0[4], EL[4], F[6]).
constexpr int kTabs = 14, tE0 = 0, tEL = 4, tF = 8;
__device__ __forceinline__ int kc_tile(int I) { return 2048 * I * (I + 1); }
// FP32 scratch of the inversion: rows padded to 68 floats so that one lane per row spreads over the banks while float4 loads stay aligned.
constexpr int LS = 68;
constexpr uint32_t kTmemCols = 512;

__device__ __forceinline__ unsigned char* cell(unsigned char* tile, int R, int c, int r) { return tile + ((size_t)c * R + r) * 16; }

// Eight FP32 values (TMEM words) to one 16-byte cell of bf16.
__device__ __forceinline__ uint4 pack8(const uint32_t* r) {
    return make_uint4(tc::bf16x2(__uint_as_float(r[0]), __uint_as_float(r[1])), tc::bf16x2(__uint_as_float(r[2]), __uint_as_float(r[3])),
                      tc::bf16x2(__uint_as_float(r[4]), __uint_as_float(r[5])), tc::bf16x2(__uint_as_float(r[6]), __uint_as_float(r[7])));
}

// ---- the inverse T = (I + L)^-1 of a chunk, 64 x 64 in FP32 -----------------------------------------------------------
// L is held TRANSPOSED, as the tensor core delivers it (Lm[j * LS + i] = L[i][j]); T row by row (row stride LS).  The 16 x 16
// diagonal blocks come by substitution; then the lower-left sz x sz block of every 2sz x 2sz diagonal block is
// -T22 (L21 T11), sz = 16 and 32.
//
// The merges are FP32 multiply-adds throughout.  A lane holds a 4 x 4 tile of the result over a quarter of the k range (kp = lane >> 3
// picks four of every sixteen, so that eight lanes read one row: no bank conflicts); two 16-byte reads feed sixteen products.  The
// four quarters meet by shuffles, after which kp is the tile's row.  The whole inverse, four blocks of 256 threads per SM: 5,500 cycles;
// rows of four columns a thread over all of k, 5,900 to 7,500; the warp-level tensor instruction with operands split into two tf32
// halves, 5,300, but at 2.2 to 2.7 times the FP32 error in the merged blocks.
__device__ __forceinline__ void row_fma(float2 (&c)[2], float a, const float4& b) {
    c[0] = fma2({a, a}, {b.x, b.y}, c[0]);
    c[1] = fma2({a, a}, {b.z, b.w}, c[1]);
}
__device__ __forceinline__ float pick(const float4& x, int s) { return s == 0 ? x.x : s == 1 ? x.y : s == 2 ? x.z : x.w; }
// Sixteen of k.  A transposed (AT): element (i, k) at A[k * LS + i]; else at A[i * LS + k].  (k, j) of B at B[k * BK + j].
template <bool AT, int BK>
__device__ __forceinline__ void tile_step(float2 (&c)[4][2], const float* A, const float* B, int kp) {
    A += AT ? kp * 4 * LS : kp * 4;
    B += kp * 4 * BK;
    float4 a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = *reinterpret_cast<const float4*>(A + u * LS);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const float4 b = *reinterpret_cast<const float4*>(B + s * BK);
        const float col[4] = {AT ? a[s].x : pick(a[0], s), AT ? a[s].y : pick(a[1], s), AT ? a[s].z : pick(a[2], s), AT ? a[s].w : pick(a[3], s)};
#pragma unroll
        for (int i = 0; i < 4; ++i) row_fma(c[i], col[i], b);
    }
}
__device__ __forceinline__ float4 tile_row(const float2 (&c)[4][2], int kp) {
    float h[2][4], r[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const float lo = v & 1 ? c[i][v >> 1].y : c[i][v >> 1].x, hi = v & 1 ? c[2 + i][v >> 1].y : c[2 + i][v >> 1].x;
            h[i][v] = ((kp & 2) ? hi : lo) + __shfl_xor_sync(0xffffffffu, (kp & 2) ? lo : hi, 16);
        }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) r[v] = ((kp & 1) ? h[1][v] : h[0][v]) + __shfl_xor_sync(0xffffffffu, (kp & 1) ? h[0][v] : h[1][v], 8);
    return make_float4(r[0], r[1], r[2], r[3]);
}
constexpr int PS = 36;  // row stride of the merges' intermediate product

// NT threads (numbered tid = 0 .. NT-1, at least eight warps) take part and meet at named barrier `bar`; ends with a barrier.
template <int NT>
__device__ __forceinline__ void invert(const float* Lm, float* Tm, float* Pm, int tid, int bar) {
    const int warp = tid >> 5, lane = tid & 31;
    if (tid < 64) {  // a diagonal block's columns, one thread each, by substitution: a settled row at once goes into all later ones
        const int o = (tid >> 4) * 16, j = tid & 15;
        float t[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) t[i] = i == j ? 1.0f : 0.0f;
#pragma unroll
        for (int m = 0; m < 15; ++m) {
            const float* Lc = Lm + (o + m) * LS + o;  // column m of the block
#pragma unroll
            for (int q = (m + 1) / 4; q < 4; ++q) {
                const float4 l = *reinterpret_cast<const float4*>(Lc + q * 4);
                if (q * 4 > m) t[q * 4] = fmaf(-l.x, t[m], t[q * 4]);
                if (q * 4 + 1 > m) t[q * 4 + 1] = fmaf(-l.y, t[m], t[q * 4 + 1]);
                if (q * 4 + 2 > m) t[q * 4 + 2] = fmaf(-l.z, t[m], t[q * 4 + 2]);
                if (q * 4 + 3 > m) t[q * 4 + 3] = fmaf(-l.w, t[m], t[q * 4 + 3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) Tm[(o + i) * LS + o + j] = t[i];
    } else {  // the blocks above the diagonal
        for (int e = tid - 64; e < CH * CH / 4; e += NT - 64) {
            const int i = e >> 4, j = (e & 15) * 4;
            if ((i >> 4) < (j >> 4)) *reinterpret_cast<float4*>(Tm + i * LS + j) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    named_bar_sync(bar, NT);
    const int kp = lane >> 3;
    if (warp < 4) {  // sz = 16: a warp has eight columns of one of the two blocks, which need nothing of the other columns
        const int r0 = (warp >> 1) * 32 + 16, c0 = r0 - 16, j0 = (warp & 1) * 8 + (lane & 1) * 4, i0 = ((lane >> 1) & 3) * 4;
        float* P = Pm + (warp >> 1) * 16 * PS;
        float2 c[4][2] = {};
        tile_step<true, LS>(c, Lm + c0 * LS + r0 + i0, Tm + c0 * LS + c0 + j0, kp);
        *reinterpret_cast<float4*>(P + (i0 + kp) * PS + j0) = tile_row(c, kp);
        __syncwarp();
        float2 d[4][2] = {};
        tile_step<false, PS>(d, Tm + (r0 + i0) * LS + r0, P + j0, kp);
        const float4 t = tile_row(d, kp);
        *reinterpret_cast<float4*>(Tm + (r0 + i0 + kp) * LS + c0 + j0) = make_float4(-t.x, -t.y, -t.z, -t.w);
    }
    named_bar_sync(bar, NT);
    const int i0 = (warp >> 1) * 8 + ((lane >> 2) & 1) * 4, j0 = (warp & 1) * 16 + (lane & 3) * 4;  // sz = 32: eight warps, 8 x 16 each
    if (warp < 8) {
        float2 c[4][2] = {};
        if (!(warp & 1)) tile_step<true, LS>(c, Lm + 32 + i0, Tm + j0, kp);  // T11 is lower triangular
        tile_step<true, LS>(c, Lm + 16 * LS + 32 + i0, Tm + 16 * LS + j0, kp);
        *reinterpret_cast<float4*>(Pm + (i0 + kp) * PS + j0) = tile_row(c, kp);
    }
    named_bar_sync(bar, NT);
    if (warp < 8) {
        float2 c[4][2] = {};
        tile_step<false, PS>(c, Tm + (32 + i0) * LS + 32, Pm + j0, kp);
        if (warp >= 4) tile_step<false, PS>(c, Tm + (32 + i0) * LS + 48, Pm + 16 * PS + j0, kp);  // T22 is lower triangular
        const float4 t = tile_row(c, kp);
        *reinterpret_cast<float4*>(Tm + (32 + i0 + kp) * LS + j0) = make_float4(-t.x, -t.y, -t.z, -t.w);
    }
    named_bar_sync(bar, NT);
}

}  // namespace pf
}  // namespace kda
