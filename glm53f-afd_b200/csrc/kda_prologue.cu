// The layer prologue of the chunked forms and of the exact prefill: projection rows to the core's inputs.
//
// The layer entry points take the engine's rows (q | k | v projections, beta logits, the forget-gate row); the chunked
// tensor-core kernels take what the recurrence is defined on: q and k after the short convolution, SiLU and the L2
// norms, v after the convolution and SiLU, the per-channel decay and beta.  This kernel computes those with the
// chain's own arithmetic (reference kernels/kda.cu:129-165 = kernels/kda_prefill.cu:121-208; this file is compiled
// without multiply-add contraction like the chain): four taps summed in order, one bf16 rounding after the SiLU, decay
// exp(lower * sigmoid(exp(A_log) (a + dt_bias))), beta = bf16(sigmoid(b)), each L2 norm as a lane's four consecutive
// channels summed in order, then the xor butterfly.  (Bit for bit in the verify sink; the prefill sink uses the
// hardware's approximate division, exponential and reciprocal root, four rows a warp, and multiply-adds.)
//
// A lane owns four consecutive channels, so the norms need no shared memory.  With the chain's arithmetic (verify and exact
// sinks): one warp per (request, head, row).  The work is bound by instruction issue (about 850 instructions per row and lane,
// most of them IEEE divisions and exponentials), so a warp takes ONE row and reads its three predecessors again (the four warps of a block take four
// consecutive rows; the predecessors come from L1/L2): every load of a warp is in flight at once and 79 registers
// allow 24 resident warps per SM (72 and 28 in the exact sink: 701 rows 400.8 -> 397.3 us; the verify sink gains nothing by it).  (The convolution two channels at a time
// and the two norms from one sum, its root and its division: chunked layer verify of 6 slots x 4 to 8 rows 738 -> 724 us, 9 x 3 to 6 975 -> 953, 12 slots 1,218 and 1,223; 701 rows exact 398 -> 395.)  (A warp that walks 16 rows with the three earlier rows sliding in registers needs
// 143 registers and was half as fast.)
//
// Three sinks:
//  * a prefill pass: core inputs for one pass of chunks, in the caller's workspace as the slots of kda_prefill_sp.cu take
//    them (a chunk's rows together, already in the swizzle that one bulk copy brings to the tensor core).  q and k are rounded
//    to fp16 (they lie in [-1, 1]; eleven mantissa bits), the one place where the chunked prefill departs from the chain's
//    FP32 q and k before the tensor-core products: with bf16's eight bits the rounding of k alone, which reaches the
//    state through K^T D, would take the state's whole error budget when few rows dominate it.  The decay is kept as
//    its logarithm.
//  * a verify call (VERIFY): the call's own buffers take the results, so nothing is allocated -- k (f32), v, the decay
//    multiplier exp(log decay) and beta go to the replay saves, which a verify call must write anyway and which hold
//    exactly these values (the bits the exact form saves), and q goes, as fp16, to the 256 bytes of `out` that the
//    same (row, head) output will overwrite.  Windows of up to 16 rows.
//  * a pass of the exact prefill (kda_rows.cu): as the verify sink, q in f32 with the chain's arithmetic too, all of it in
//    the caller's workspace.

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "glm53f_kda.h"
#include "kda_internal.h"

namespace kda {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kVerifyWindow = 16;

struct ProParams {
    int H, batch, pass_rows, row_shift;  // rows row_shift .. row_shift + pass_rows - 1 of every request
    const int32_t* cu;
    const uint16_t* P;
    long long p_stride, b_off;
    const uint16_t* A;
    long long a_stride;
    const uint16_t* conv;
    const long long* conv_off;
    const uint16_t* cw;
    const float* a_log;
    const float* dt_bias;
    float lower;
    unsigned char* slots;  // prefill pass: [batch][H][pass_rows / 64]
    unsigned int* tail;    // the workspace's tail
    // verify: q as fp16 into the output rows, the rest into the replay saves
    uint16_t* q;
    long long out_stride;
    float *k_save, *g_save, *b_save;
    uint16_t* v_save;
    float* qf;  // exact sink: q in f32 (k, decay multiplier, v and beta through the saves' pointers)
    int rows1;  // cu == nullptr: one request of rows1 rows
};
enum Sink : int { kVerify = 1, kExact = 2 };

// IEEE arithmetic is the chain's (its results are the replay saves, bit for bit).  q of the verify sink and everything of the
// prefill sink feed tensor-core products that round every operand to bf16 or fp16 anyway, so there the divisions, exponentials
// and reciprocal roots are the hardware approximations (a few ulp of FP32).
__device__ __forceinline__ float sigmoid_(float x) { return 1.0f / (1.0f + expf(-x)); }
template <bool FAST>
__device__ __forceinline__ float silu_(float x) {
    if constexpr (FAST) return __fdividef(x, 1.0f + __expf(-x));
    else return x / (1.0f + expf(-x));
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return fma2(a, {1.0f, 1.0f}, b); }
__device__ __forceinline__ void unpack4(uint2 w, float (&x)[4]) {
    x[0] = __uint_as_float(w.x << 16);
    x[1] = __uint_as_float(w.x & 0xffff0000u);
    x[2] = __uint_as_float(w.y << 16);
    x[3] = __uint_as_float(w.y & 0xffff0000u);
}
__device__ __forceinline__ uint2 pack4_fp16(const float (&x)[4]) {
    const __half2 lo = __floats2half2_rn(x[0], x[1]), hi = __floats2half2_rn(x[2], x[3]);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}
__device__ __forceinline__ uint2 pack4(const float (&x)[4]) {
    return make_uint2((uint32_t)f32_to_bf16_bits(x[0]) | ((uint32_t)f32_to_bf16_bits(x[1]) << 16),
                      (uint32_t)f32_to_bf16_bits(x[2]) | ((uint32_t)f32_to_bf16_bits(x[3]) << 16));
}

// Four consecutive channels of a row, element by element.  Rows of the projections are aligned for vector loads (the callers check);
// a request's conv window starts at any element of the arena its offset names, and the few warps that read one take a way of
// their own where it is not aligned: a choice at every load costs the loads their overlap (701 rows exact: 403 -> 408 us).
__device__ __forceinline__ uint2 load4(const uint16_t* at) {
    return make_uint2((uint32_t)at[0] | ((uint32_t)at[1] << 16), (uint32_t)at[2] | ((uint32_t)at[3] << 16));
}
__device__ __forceinline__ bool unaligned8(const void* at) { return (reinterpret_cast<uintptr_t>(at) & 7) != 0; }

template <int SINK>
__global__ void __launch_bounds__(128, SINK == kExact ? 7 : 6) layer_prologue_kernel(const ProParams p) {
    constexpr bool VERIFY = SINK == kVerify, EXACT = SINK == kExact;
    grid_ready();
    const int lane = threadIdx.x & 31, H = p.H;
    // a block = four consecutive rows of one (request, head): neighbours share their predecessors in L1
    const int quads = p.pass_rows / 4;
    const long long unit = blockIdx.x / quads;
    const int j_first = (int)(blockIdx.x % quads) * 4 + (threadIdx.x >> 5);  // row of the pass
    const int h = (int)(unit % H), b = (int)(unit / H);
    // A prefill pass covers pass_rows rows of every request.  A verify window is meant to have at most 16 rows; should one be
    // longer (the chunk kernel then reports status 122 and leaves the rows past 16 without outputs), its replay saves are
    // still written for EVERY row, so that a commit of any prefix replays real values: the warp goes on in steps of 16.
    const int r0 = p.cu ? p.cu[b] : 0, n_all = max((p.cu ? p.cu[b + 1] - r0 : p.rows1) - p.row_shift, 0), n = VERIFY ? n_all : min(n_all, p.pass_rows);
    for (int j = j_first; j < n; j += p.pass_rows) {
    const int c0 = lane * 4, jj = p.row_shift + j;  // row of the request
    const long long C = 3LL * H * DK, gr = (long long)r0 + jj;
    const uint16_t* window = p.conv + (p.conv_off ? p.conv_off[b] : 0);
    uint2 x[TAPS][3];  // [tap: rows jj-3 .. jj][part]; rows before the request's first come from the conv window
    auto fetch = [&](auto&& load) {
#pragma unroll
        for (int d = 0; d < TAPS; ++d) {
            const int rr = jj - 3 + d;
            const uint16_t* row = rr < 0 ? window + (long long)(WINDOW + rr) * C : p.P + ((long long)r0 + rr) * p.p_stride;
#pragma unroll
            for (int part = 0; part < 3; ++part) x[d][part] = load(row + ((long long)part * H + h) * DK + c0);
        }
    };
    if (jj < WINDOW && unaligned8(window)) fetch([](const uint16_t* at) { return load4(at); });
    else fetch([](const uint16_t* at) { return *reinterpret_cast<const uint2*>(at); });
    uint4 wq[3][2];
#pragma unroll
    for (int part = 0; part < 3; ++part) {
        const uint4* src = reinterpret_cast<const uint4*>(p.cw + (((long long)part * H + h) * DK + c0) * TAPS);
        wq[part][0] = src[0];
        wq[part][1] = src[1];
    }
    const uint2 a_bits = *reinterpret_cast<const uint2*>(p.A + gr * p.a_stride + (long long)h * DK + c0);
    const float4 dtb4 = *reinterpret_cast<const float4*>(p.dt_bias + (long long)h * DK + c0);
    const float blogit = bf16_bits_to_f32(p.P[gr * p.p_stride + p.b_off + h]);
    const float decay_rate = expf(p.a_log[h]);

    float act[3][4];
#pragma unroll
    for (int part = 0; part < 3; ++part) {
        float xv[TAPS][4];
#pragma unroll
        for (int d = 0; d < TAPS; ++d) unpack4(x[d][part], xv[d]);
        const uint32_t ww[8] = {wq[part][0].x, wq[part][0].y, wq[part][0].z, wq[part][0].w, wq[part][1].x, wq[part][1].y, wq[part][1].z, wq[part][1].w};
#pragma unroll
        for (int c = 0; c < 4; c += 2) {  // two channels at a time, every product and sum rounded by itself
            float2 acc = {0.0f, 0.0f};
#pragma unroll
            for (int d = 0; d < TAPS; ++d) {
                const uint32_t w0 = ww[2 * c + d / 2], w1 = ww[2 * c + 2 + d / 2];
                acc = add2(acc, mul2(d & 1 ? float2{__uint_as_float(w0 & 0xffff0000u), __uint_as_float(w1 & 0xffff0000u)} : float2{__uint_as_float(w0 << 16), __uint_as_float(w1 << 16)},
                                     {xv[d][c], xv[d][c + 1]}));
            }
            // q reaches only the outputs, which carry bf16-operand rounding in both chunked forms: the fast form there
            act[part][c] = bf16_round(part == 0 ? silu_<!EXACT>(acc.x) : silu_<false>(acc.x));
            act[part][c + 1] = bf16_round(part == 0 ? silu_<!EXACT>(acc.y) : silu_<false>(acc.y));
        }
    }
    // L2 norms of q and k (eps 1e-6 inside the root), q also times 128^-0.5.
    float qn[4], kn[4];
    {
        float sq = 0.0f, sk = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            sq = sq + act[0][c] * act[0][c];
            sk = sk + act[1][c] * act[1][c];
        }
        // Half of the lanes go on with q's sum, half with k's, and so does all that follows from it; the butterfly's pairs.
        const bool up = lane >= 16;
        float ss = (up ? sk : sq) + __shfl_xor_sync(FULL, up ? sq : sk, 16);
#pragma unroll
        for (int o = 8; o; o >>= 1) ss = ss + __shfl_xor_sync(FULL, ss, o);
        const float inv = 1.0f / sqrtf(ss + 1e-6f), iq = __shfl_sync(FULL, inv, 0), ik = __shfl_sync(FULL, inv, 16);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            qn[c] = (act[0][c] * iq) * (1.0f / sqrtf((float)DK));
            kn[c] = act[1][c] * ik;
        }
    }
    float a4[4], lg[4];
    unpack4(a_bits, a4);
    const float dtb[4] = {dtb4.x, dtb4.y, dtb4.z, dtb4.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) lg[c] = p.lower * sigmoid_(decay_rate * (a4[c] + dtb[c]));
    const float bt = bf16_round(sigmoid_(blogit));
    if constexpr (VERIFY) {
        const long long sv = (gr * H + h) * DK + c0;
        if (j < p.pass_rows) *reinterpret_cast<uint2*>(p.q + gr * p.out_stride + (long long)h * DK + c0) = pack4_fp16(qn);  // rows past 16 get no output: leave theirs alone
        *reinterpret_cast<float4*>(p.k_save + sv) = make_float4(kn[0], kn[1], kn[2], kn[3]);
        *reinterpret_cast<uint2*>(p.v_save + sv) = pack4(act[2]);
        *reinterpret_cast<float4*>(p.g_save + sv) = make_float4(expf(lg[0]), expf(lg[1]), expf(lg[2]), expf(lg[3]));
        if (lane == 0) p.b_save[gr * H + h] = bt;
    } else if constexpr (EXACT) {
        const long long orow = (long long)b * p.pass_rows + j, at = (orow * H + h) * DK + c0;
        *reinterpret_cast<float4*>(p.qf + at) = make_float4(qn[0], qn[1], qn[2], qn[3]);
        *reinterpret_cast<float4*>(p.k_save + at) = make_float4(kn[0], kn[1], kn[2], kn[3]);
        *reinterpret_cast<float4*>(p.g_save + at) = make_float4(expf(lg[0]), expf(lg[1]), expf(lg[2]), expf(lg[3]));
        *reinterpret_cast<uint2*>(p.v_save + at) = pack4(act[2]);
        if (lane == 0) p.b_save[orow * H + h] = bt;
    }
    }
}

// ---- the prefill sink ---------------------------------------------------------------------------------------------------
// Bound by instruction issue before it is bound by memory (a row and head: 1 KiB in, 1.3 KiB out).  A warp takes four consecutive
// rows: seven rows of inputs instead of sixteen, the weights once, and everything in pairs of channels (two-wide multiply-adds).
// 1,280 rows x 64 heads: 79 us with a warp per row as in the kernel above, 52 so with four blocks an SM; five take another 4 us off a pass of the whole call, and six, at 80 registers now that exponentials are single
// instructions, 3 more (4 x 2,048 rows 941 -> 923 us, 3 x 700 246 -> 238); seven spill (244).
// Sums of the norms by halves and a row's beta by one lane of every four, 4 x 2,048 rows 889.5 -> 880.0, passes of 1,024 785 -> 769.  (Eight rows a warp spill, 963
// to 1,000; the parts' rows fetched one part ahead instead of all at once, 899.)
constexpr int kRowsPer = 4;
__device__ __forceinline__ float2 lo_hi(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
// 1 / (1 + e^-x)
__device__ __forceinline__ float2 sigmoid2(float2 x) {
    const float2 t = mul2(x, {-kLog2e, -kLog2e}), d = add2({ex2_ftz(t.x), ex2_ftz(t.y)}, {1.0f, 1.0f});
    return make_float2(rcp_approx(d.x), rcp_approx(d.y));
}
__device__ __forceinline__ uint32_t fp16x2(float2 x) {
    const __half2 h = __float22half2_rn(x);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// The sums over the warp of a value a row: v[i] of every lane goes in, the sum of row lane / 8 comes out.  At each of the first two steps a lane gives half
// of its rows away, so four sums take six shuffles and not twenty; the tree is the butterfly's.
__device__ __forceinline__ float row_sums(float (&v)[kRowsPer], int lane) {
#pragma unroll
    for (int n = kRowsPer / 2, o = 16; n > 0; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(FULL, up ? v[i] : v[i + n], o);
    }
#pragma unroll
    for (int o = 16 / kRowsPer; o; o >>= 1) v[0] += __shfl_xor_sync(FULL, v[0], o);
    return v[0];
}

// FIRST: the pass with the requests' first rows, which reach back into the conv windows.
template <bool FIRST>
__global__ void __launch_bounds__(128, 6) prefill_prologue_kernel(const ProParams p) {
    const int lane = threadIdx.x & 31, H = p.H, groups = p.pass_rows / (4 * kRowsPer), c0 = lane * 4;
    // heads innermost: neighbouring blocks read neighbouring pieces of the same rows
    const int h = (int)(blockIdx.x % H), b = (int)(blockIdx.x / H / groups), j0 = (int)(blockIdx.x / H % groups) * 4 * kRowsPer + (threadIdx.x >> 5) * kRowsPer;
    const int r0 = p.cu[b], n = min(p.cu[b + 1] - r0 - p.row_shift, p.pass_rows);
    // The passes' counters start from zero (as a launch of its own this was 2 us of a short prompt's 50).
    if (FIRST && blockIdx.x == 0 && threadIdx.x < 2 * kTailSet) p.tail[kTailSets + threadIdx.x] = 0u;
    if (j0 >= n) return;
    const int first = p.row_shift + j0, last = p.row_shift + n - 1;  // rows of the request; rows before its first come from the conv window
    const long long C = 3LL * H * DK;
    uint2 x[3][kRowsPer + 3];
    auto fetch = [&](const uint16_t* window, auto&& load) {
#pragma unroll
        for (int d = 0; d < kRowsPer + 3; ++d) {
            const int rr = min(first - 3 + d, last);
            const uint16_t* row = (FIRST && rr < 0 ? window + (long long)(WINDOW + rr) * C : p.P + ((long long)r0 + rr) * p.p_stride) + (long long)h * DK + c0;
#pragma unroll
            for (int part = 0; part < 3; ++part) x[part][d] = load(row + (long long)part * H * DK);
        }
    };
    auto vec = [](const uint16_t* at) { return *reinterpret_cast<const uint2*>(at); };
    if constexpr (FIRST) {
        const uint16_t* window = p.conv + (p.conv_off ? p.conv_off[b] : 0);
        if (first < WINDOW && unaligned8(window)) fetch(window, [](const uint16_t* at) { return load4(at); });
        else fetch(window, vec);
    } else {
        fetch(nullptr, vec);
    }
    uint2 a_bits[kRowsPer];
#pragma unroll
    for (int i = 0; i < kRowsPer; ++i) {
        const long long gr = (long long)r0 + min(first + i, last);
        a_bits[i] = *reinterpret_cast<const uint2*>(p.A + gr * p.a_stride + (long long)h * DK + c0);
    }
    const float4 dtb = *reinterpret_cast<const float4*>(p.dt_bias + (long long)h * DK + c0);
    const float rate = expf(p.a_log[h]);
    const float bl = bf16_bits_to_f32(p.P[((long long)r0 + min(first + (lane & (kRowsPer - 1)), last)) * p.p_stride + p.b_off + h]);  // of row lane % 4
    unsigned char* slot = p.slots + (((long long)b * H + h) * (p.pass_rows / 64) + (j0 >> 6)) * kPrefillSlotBytes;
    const int r = j0 & 63;

#pragma unroll
    for (int part = 0; part < 3; ++part) {
        const uint4* src = reinterpret_cast<const uint4*>(p.cw + (((long long)part * H + h) * DK + c0) * TAPS);
        const uint4 wa = src[0], wb = src[1];  // a channel's four taps in two words
        const float2 w01[TAPS] = {{__uint_as_float(wa.x << 16), __uint_as_float(wa.z << 16)}, {__uint_as_float(wa.x & 0xffff0000u), __uint_as_float(wa.z & 0xffff0000u)},
                                  {__uint_as_float(wa.y << 16), __uint_as_float(wa.w << 16)}, {__uint_as_float(wa.y & 0xffff0000u), __uint_as_float(wa.w & 0xffff0000u)}};
        const float2 w23[TAPS] = {{__uint_as_float(wb.x << 16), __uint_as_float(wb.z << 16)}, {__uint_as_float(wb.x & 0xffff0000u), __uint_as_float(wb.z & 0xffff0000u)},
                                  {__uint_as_float(wb.y << 16), __uint_as_float(wb.w << 16)}, {__uint_as_float(wb.y & 0xffff0000u), __uint_as_float(wb.w & 0xffff0000u)}};
        float2 acc[kRowsPer][2];
#pragma unroll
        for (int d = 0; d < kRowsPer + 3; ++d) {  // input row d is tap d - i of output row i
            const float2 x01 = lo_hi(x[part][d].x), x23 = lo_hi(x[part][d].y);
#pragma unroll
            for (int i = 0; i < kRowsPer; ++i) {
                const int t = d - i;
                if (t == 0) acc[i][0] = mul2(w01[0], x01), acc[i][1] = mul2(w23[0], x23);
                else if (t > 0 && t < TAPS) acc[i][0] = fma2(w01[t], x01, acc[i][0]), acc[i][1] = fma2(w23[t], x23, acc[i][1]);
            }
        }
        float ss[kRowsPer];
        uint2 y[kRowsPer];  // bf16(silu)
#pragma unroll
        for (int i = 0; i < kRowsPer; ++i) {
            const float2 s01 = mul2(acc[i][0], sigmoid2(acc[i][0])), s23 = mul2(acc[i][1], sigmoid2(acc[i][1]));
            const __nv_bfloat162 p01 = __float22bfloat162_rn(s01), p23 = __float22bfloat162_rn(s23);
            y[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&p01), *reinterpret_cast<const uint32_t*>(&p23));
            if (part < 2) {
                const float2 f01 = lo_hi(y[i].x), f23 = lo_hi(y[i].y), q = fma2(f23, f23, mul2(f01, f01));
                ss[i] = q.x + q.y;
            }
        }
        if (part < 2) {  // L2 norms of q and k (eps 1e-6 inside the root), q also times 128^-0.5
            const float rinv = rsqrtf(row_sums(ss, lane) + 1e-6f) * (part == 0 ? 0.08838834764831845f : 1.0f);
#pragma unroll
            for (int i = 0; i < kRowsPer; ++i) {
                const float s = __shfl_sync(FULL, rinv, i * (32 / kRowsPer));
                y[i] = make_uint2(fp16x2(mul2(lo_hi(y[i].x), {s, s})), fp16x2(mul2(lo_hi(y[i].y), {s, s})));
            }
        }
        unsigned char* to = slot + (part == 0 ? kSlotInQ : part == 1 ? kSlotInK : kSlotInV) + (lane & 1) * 8;
#pragma unroll
        for (int i = 0; i < kRowsPer; ++i)
            if (j0 + i < n) *reinterpret_cast<uint2*>(to + prefill_box_piece(r + i, lane >> 1)) = y[i];
    }
#pragma unroll
    for (int i = 0; i < kRowsPer; ++i) {
        if (j0 + i >= n) break;
        const float2 s01 = sigmoid2(mul2(add2(lo_hi(a_bits[i].x), {dtb.x, dtb.y}), {rate, rate})), s23 = sigmoid2(mul2(add2(lo_hi(a_bits[i].y), {dtb.z, dtb.w}), {rate, rate}));
        const float2 g01 = mul2(s01, {p.lower, p.lower}), g23 = mul2(s23, {p.lower, p.lower});
        *reinterpret_cast<float4*>(slot + kSlotInG + prefill_box_piece(r + i, lane)) = make_float4(g01.x, g01.y, g23.x, g23.y);
    }
    if (lane < kRowsPer && j0 + lane < n) reinterpret_cast<float*>(slot + kSlotInBeta)[r + lane] = bf16_round(sigmoid2({bl, bl}).x);
}

template <int SINK>
int launch(const ProParams& pp, cudaStream_t stream) {
    const long long blocks = (long long)pp.batch * pp.H * (pp.pass_rows / 4);
    if (blocks > 0x7fffffffLL) return kInvalid;
    // Begun while the launch before drains: a chunked round of 4 slots 755 -> 703 us, of 12 slots x 8 rows 1,600 -> 1,565.  (The prefill's
    // prologue, launched further down, is the faster for a plain launch.)
    return launch_early(layer_prologue_kernel<SINK>, (unsigned)blocks, 128, 0, stream, pp);
}

}  // namespace

int layer_prologue_launch(int32_t heads, int32_t batch, const int32_t* cu_rows, int32_t chunks, int32_t chunk0,
                          const glm53f_bf16* p, int64_t p_stride, int64_t b_off, const glm53f_bf16* a, int64_t a_stride,
                          const glm53f_bf16* conv, const int64_t* conv_off, const glm53f_bf16* conv_w, const float* a_log,
                          const float* dt_bias, float lower, unsigned char* slots, unsigned int* tail, cudaStream_t stream) {
    ProParams pp{};
    pp.H = heads; pp.batch = batch; pp.pass_rows = chunks * 64; pp.row_shift = chunk0 * 64;
    pp.cu = cu_rows;
    pp.P = p; pp.p_stride = p_stride; pp.b_off = b_off;
    pp.A = a; pp.a_stride = a_stride;
    pp.conv = conv; pp.conv_off = reinterpret_cast<const long long*>(conv_off); pp.cw = conv_w;
    pp.a_log = a_log; pp.dt_bias = dt_bias; pp.lower = lower;
    pp.slots = slots;
    pp.tail = tail;
    const long long blocks = (long long)batch * heads * (pp.pass_rows / (4 * kRowsPer));
    if (blocks > 0x7fffffffLL) return kInvalid;
    if (chunk0 == 0) prefill_prologue_kernel<true><<<(unsigned)blocks, 128, 0, stream>>>(pp);
    else prefill_prologue_kernel<false><<<(unsigned)blocks, 128, 0, stream>>>(pp);
    return (int)cudaGetLastError();
}

int exact_prologue_launch(int32_t heads, int32_t batch, const int32_t* cu_rows, int32_t rows1, int32_t pass_rows, int32_t row_shift,
                          const glm53f_bf16* p, int64_t p_stride, int64_t b_off, const glm53f_bf16* a, int64_t a_stride,
                          const glm53f_bf16* conv, const int64_t* conv_off, const glm53f_bf16* conv_w, const float* a_log,
                          const float* dt_bias, float lower, float* q, float* k, float* g, glm53f_bf16* v, float* beta, cudaStream_t stream) {
    if (pass_rows < 16 || pass_rows % 16 != 0) return kInvalid;
    ProParams pp{};
    pp.H = heads; pp.batch = batch; pp.pass_rows = pass_rows; pp.row_shift = row_shift;
    pp.cu = cu_rows; pp.rows1 = rows1;
    pp.P = p; pp.p_stride = p_stride; pp.b_off = b_off;
    pp.A = a; pp.a_stride = a_stride;
    pp.conv = conv; pp.conv_off = reinterpret_cast<const long long*>(conv_off); pp.cw = conv_w;
    pp.a_log = a_log; pp.dt_bias = dt_bias; pp.lower = lower;
    pp.qf = q; pp.k_save = k; pp.g_save = g; pp.v_save = v; pp.b_save = beta;
    return launch<kExact>(pp, stream);
}

// The prologue of the chunked verify: windows of up to 16 rows per request; see the head of the file for where the
// results go.  The caller checks the alignment of every row.
int verify_prologue_launch(int32_t heads, int32_t batch, const int32_t* cu_rows, const glm53f_bf16* p, int64_t p_stride, int64_t b_off,
                           const glm53f_bf16* a, int64_t a_stride, const glm53f_bf16* conv, const int64_t* conv_off,
                           const glm53f_bf16* conv_w, const float* a_log, const float* dt_bias, float lower, glm53f_bf16* out,
                           int64_t out_stride, float* k_save, glm53f_bf16* v_save, float* g_save, float* b_save, cudaStream_t stream) {
    ProParams pp{};
    pp.H = heads; pp.batch = batch; pp.pass_rows = kVerifyWindow; pp.row_shift = 0;
    pp.cu = cu_rows;
    pp.P = p; pp.p_stride = p_stride; pp.b_off = b_off;
    pp.A = a; pp.a_stride = a_stride;
    pp.conv = conv; pp.conv_off = reinterpret_cast<const long long*>(conv_off); pp.cw = conv_w;
    pp.a_log = a_log; pp.dt_bias = dt_bias; pp.lower = lower;
    pp.q = out; pp.out_stride = out_stride;
    pp.k_save = k_save; pp.v_save = v_save; pp.g_save = g_save; pp.b_save = b_save;
    return launch<kVerify>(pp, stream);
}

}  // namespace kda
