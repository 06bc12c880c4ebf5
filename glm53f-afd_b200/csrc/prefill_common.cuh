// Pieces shared by the chunk-64 tensor-core prefill kernels: the chunk geometry, the shared-memory map of the
// state-independent ("intra") phase, the cell helpers and the FP32 triangular inverse.
#pragma once

#include "common.cuh"
#include "tc.cuh"

namespace kda {
namespace pf {

constexpr int CH = 64;            // rows per chunk
constexpr int kCompute = 512;     // 16 compute warps: warp w reaches TMEM lanes 32*(w%4).., and takes columns 32*(w/4)..
constexpr int kThreadsTc = kCompute + 32;  // + one loader warp that streams the next chunk's rows in
constexpr int RS16 = 272;         // staging row stride, bf16 tensors (256 + 16: rows 4 banks apart)
constexpr int RS32 = 528;         // staging row stride, f32 tensor
// Shared memory map (bytes).  Tiles are 64-row (R = 64) cell arrays unless noted; buffers whose lifetimes do not
// overlap inside a chunk share space, so that the staging area is free again as soon as the operands are built and
// the next chunk's rows can stream in behind the current chunk's arithmetic.
constexpr int kTile = CH * 16 * 16;  // 16 KiB: 64 rows x 128 bf16
constexpr int oRawQ = 0, oRawK = oRawQ + CH * RS16, oRawV = oRawK + CH * RS16, oRawG = oRawV + CH * RS16;
constexpr int oKg = oRawG + CH * RS32;   // Kg                       (steps 2-6)   } later S16 [128 rows] (steps 8-9)
constexpr int oKinv = oKg + kTile;        // Kinv (2-3)                             }
constexpr int oTp = oKinv + kTile;        // T' hi | T' lo (5c-6), later D hi (steps 10-11)
constexpr int oW = oTp + kTile;           // W                        (steps 7-9)
constexpr int oV = oW + kTile;            // V                        (steps 2-6), later D lo
constexpr int oQg = oV + kTile;           // Qg                       (steps 2-9)
constexpr int oKdHi = oQg + kTile, oKdLo = oKdHi + kTile;  // Kdec hi, lo (steps 2-11)
constexpr int oMm = oKdLo + kTile;        // M, 64 x 64 bf16          (steps 4-11)
constexpr int oS16 = oKg, oDhi = oTp, oDlo = oV, oTpHi = oTp, oTpLo = oTp + kTile / 2;
// The column sides of L and M, one tile per row block I (rows 0 .. 16 I + 15, 256 bytes a row), over Kinv | T' | W
// (steps 2-3); the per-block decay factor tables (14 x 128 floats: E0[4], EL[4], F[6]) over M (steps 1-3).
constexpr int oKc = oKinv, oTab = oMm, kTabs = 14, tE0 = 0, tEL = 4, tF = 8;
__device__ __forceinline__ int kc_tile(int I) { return 2048 * I * (I + 1); }
static_assert(2 * 128 * (16 + 32 + 48 + 64) <= 3 * kTile && kTabs * 512 <= kTile / 2, "column-side tiles and tables");
// FP32 scratch of the inversion (steps 4-5) over Kinv | T' | W, all dead then: T, P, L.  Rows are padded to 68
// floats so that one lane per row spreads over the banks while float4 loads stay aligned.
constexpr int LS = 68;
constexpr int oT = oKinv, oP = oT + CH * LS * 4, oL = oKinv + 24576;
static_assert(oP + 32 * 40 * 4 <= oL && oL + CH * LS * 4 <= oKinv + 3 * kTile, "inversion scratch");
constexpr int oBeta = oMm + kTile / 2, oEGL = oBeta + 2 * CH * 4, oScan = oEGL + 128 * 4, oRed = oScan + 4 * 128 * 4;
constexpr int oBars = oRed + 4 * CH * 4, oCtl = oBars + 32;
constexpr int kSmemTc = oCtl + 32;
static_assert(kSmemTc <= 232448, "shared memory budget");
// Tensor memory columns.
constexpr uint32_t cS = 0, cL = 128, cMm = 192, cW = 256, cQS = 256, cU = 384, kTmemCols = 512;


__device__ __forceinline__ void compute_sync() { named_bar_sync(1, kCompute); }

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
// The merges run on the warp-level tensor instruction (m16n8k8, tf32) with every operand split into two tf32 halves and three
// products, 21 bits of operand mantissa: these contractions are too small for a round through tensor memory (publish, issue,
// wait, read back: about 1,000 cycles), and as multiply-adds from shared memory they took 6,500 of an item's 31,000 cycles.
__device__ __forceinline__ uint32_t tf32_of(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    hi = tf32_of(x);
    lo = tf32_of(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// c += A B over k in [k0, k1) (multiples of 8), c a 16 x 8 tile of one warp: element (i, k) of A at A[i * AI + k * AK], (k, j) of B at
// B[k * BK + j].
template <int AI, int AK, int BK>
__device__ __forceinline__ void tile_product(float (&c)[4], const float* A, const float* B, int k0, int k1, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll 2
    for (int k = k0; k < k1; k += 8) {
        uint32_t ah[4], al[4], bh[2], bl[2];
        split_tf32(A[g * AI + (k + t) * AK], ah[0], al[0]);
        split_tf32(A[(g + 8) * AI + (k + t) * AK], ah[1], al[1]);
        split_tf32(A[g * AI + (k + t + 4) * AK], ah[2], al[2]);
        split_tf32(A[(g + 8) * AI + (k + t + 4) * AK], ah[3], al[3]);
        split_tf32(B[(k + t) * BK + g], bh[0], bl[0]);
        split_tf32(B[(k + t + 4) * BK + g], bh[1], bl[1]);
        mma_tf32(c, al, bh);
        mma_tf32(c, ah, bl);
        mma_tf32(c, ah, bh);
    }
}
template <int LD>
__device__ __forceinline__ void tile_store(float* C, const float (&c)[4], float sign, int lane) {
    const int g = lane >> 2, t = lane & 3;
    *reinterpret_cast<float2*>(C + g * LD + 2 * t) = make_float2(sign * c[0], sign * c[1]);
    *reinterpret_cast<float2*>(C + (g + 8) * LD + 2 * t) = make_float2(sign * c[2], sign * c[3]);
}
constexpr int PS = 40;  // row stride of the merges' intermediate product (32 x 32): conflict-free as a B operand

// NT threads (numbered tid = 0 .. NT-1, at least eight warps) take part and meet at named barrier `bar`; ends with a barrier.
template <int NT = kCompute>
__device__ __forceinline__ void invert(const float* Lm, float* Tm, float* Pm, int tid, int bar = 1) {
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
    if (warp < 4) {  // sz = 16: a warp has eight columns of one of the two blocks, which need nothing of the other columns
        const int r0 = (warp >> 1) * 32 + 16, c0 = r0 - 16, j0 = (warp & 1) * 8;
        float* P = Pm + warp * 16 * 8;
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        tile_product<1, LS, LS>(c, Lm + c0 * LS + r0, Tm + c0 * LS + c0 + j0, j0, 16, lane);  // T11 is lower triangular
        tile_store<8>(P, c, 1.0f, lane);
        __syncwarp();
        c[0] = c[1] = c[2] = c[3] = 0.0f;
        tile_product<LS, 1, 8>(c, Tm + r0 * LS + r0, P, 0, 16, lane);
        tile_store<LS>(Tm + r0 * LS + c0 + j0, c, -1.0f, lane);
    }
    named_bar_sync(bar, NT);
    const int i0 = (warp >> 2) * 16, j0 = (warp & 3) * 8;  // sz = 32: eight warps, a 16 x 8 tile each
    if (warp < 8) {
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        tile_product<1, LS, LS>(c, Lm + 32 + i0, Tm + j0, j0, 32, lane);
        tile_store<PS>(Pm + i0 * PS + j0, c, 1.0f, lane);
    }
    named_bar_sync(bar, NT);
    if (warp < 8) {
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        tile_product<LS, 1, PS>(c, Tm + (32 + i0) * LS + 32, Pm + j0, 0, i0 + 16, lane);  // T22 is lower triangular
        tile_store<LS>(Tm + (32 + i0) * LS + j0, c, -1.0f, lane);
    }
    named_bar_sync(bar, NT);
}

}  // namespace pf
}  // namespace kda
