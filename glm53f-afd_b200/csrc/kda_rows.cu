// The exact recurrence over many rows of few requests (prompt segments of the layer prefill's exact form): the rows' inputs
// are cooked beforehand, for a pass of rows at once, and the outputs are normalised afterwards, so that what is left serial
// is the delta rule alone.
//
//   layer_prologue_kernel (kda_prologue.cu)   every row of a pass in parallel: q, k, the decay multiplier (f32), v (bf16), beta
//   rows_kernel                               the state through the pass's rows; each row's read-out, rounded to bf16, in `out`
//   rows_norm_kernel                          the gated RMSNorm over every row, in place in `out`
//
// The persistent pipeline (kda_chain.cu) cooks, steps and normalises row after row on one SM per (request, head): 1.55 us a
// row, 64 of 148 SMs busy for one prompt.  Here a WARP is the unit of work -- eight of a unit's
// value rows never interact with the others --, reads what its lanes need of a cooked row straight into registers, rows
// ahead, and meets no barrier; a unit's sixteen warps are four blocks, so a prompt of 64 heads puts work on every SM.
//
// What bounds it: a row is a chain of dependent steps (decayed state, k-product, five shuffles, update) with two warps a
// scheduler (340 issue slots a row and warp, two-wide operations at 2.5 cycles).  One prompt of 701 rows, f32
// states: 1,087 -> 402 us (0.5 us a row).  Measured against it at 701 rows: three rows in flight 406,
// five blocks an SM (96 registers, spills) 515, four value rows a warp 451, rows through shared memory by asynchronous copies 457.
//
// Launches of more units (rows_launch: from 112 on, two prompts of 64 heads) run rows_octet_kernel: there the work of an SM's warps counts, not a
// row's latency.
//
// Same arithmetic in the same order with the same rounding points (a bf16 state is rounded after every row, the read-out
// before the norm): the chain's bits.

#include "common.cuh"
#include "glm53f_kda.h"
#include "kda_internal.h"
#include "recurrence.cuh"
#include "recurrence_octet.cuh"

namespace kda {
namespace {

constexpr int kRowsWarps = 4, kRowsThreads = kRowsWarps * 32, kParts = kRecWarps / kRowsWarps;
constexpr int kPerSm = 4;    // blocks an SM holds: 128 registers a thread
constexpr int kAhead = 2;    // rows in flight in registers, 14 each

struct CookedRow {
    float4 k, g, q;
    uint16_t v;  // bf16 bits, widened when the row's turn comes: a conversion at the load would wait for it there and then
    float beta;
};

template <typename S>
__global__ void __launch_bounds__(kRowsThreads, kPerSm) rows_kernel(const __grid_constant__ RowsParams p) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned unit = blockIdx.x / kParts;
    const int uw = (int)(blockIdx.x % kParts) * kRowsWarps + warp;  // this warp's place among the unit's 16
    const int h = (int)(unit % (unsigned)p.H), b = (int)(unit / (unsigned)p.H);
    const int r0 = p.cu ? p.cu[b] : 0, all = p.cu ? p.cu[b + 1] - r0 : p.rows1;
    const int n = min(max(all - p.row_shift, 0), p.pass_rows);
    if (n == 0 && p.state_in == p.state_out) return;
    const long long s_elem = (p.state_off ? p.state_off[b] : 0) + (long long)h * DV * DK;
    f32x2 s[kPairs][4];
    load_rows_global<S>(reinterpret_cast<const S*>(p.state_in) + s_elem, uw, lane, s);
    const long long first = (long long)b * p.pass_rows * p.H + h;      // (row, head) index of the pass's row 0
    const int mine = uw * kRowsPerLane + ((lane >> 1) & 7);            // the value row whose sums this lane receives
    auto fetch = [&](int r) {
        const long long rh = first + (long long)r * p.H, at = rh * DK;
        CookedRow x;
        x.k = *reinterpret_cast<const float4*>(p.k + at + lane * 4);
        x.g = *reinterpret_cast<const float4*>(p.g + at + lane * 4);
        x.q = *reinterpret_cast<const float4*>(p.q + at + lane * 4);
        x.v = p.v[at + mine];
        x.beta = p.beta[rh];
        return x;
    };
    // A row's read-out is reduced together with the next row's k-product: one chain of shuffles a row.  sums[0..7] are the
    // k-product's partial sums, sums[8..15] the read-out's; lanes 0-15 then hold the k-products, lanes 16-31 the previous
    // row's read-outs, two lanes to a value row.
    float sums[2 * kRowsPerLane] = {};
    uint16_t* out = p.out + ((long long)r0 + p.row_shift) * p.out_stride + (long long)h * DV + mine;
    auto step = [&](const CookedRow& x, bool first_row) {
        const f32x2 kk[4] = {pack2(x.k.x, x.k.x), pack2(x.k.y, x.k.y), pack2(x.k.z, x.k.z), pack2(x.k.w, x.k.w)};
        const f32x2 gg[4] = {pack2(x.g.x, x.g.x), pack2(x.g.y, x.g.y), pack2(x.g.z, x.g.z), pack2(x.g.w, x.g.w)};
        if constexpr (sizeof(S) == 2) {
            if (!first_row) round_rows(s);  // after a row's read-out; the last row's rounding is the store's
        }
#pragma unroll
        for (int jp = 0; jp < kPairs; ++jp)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[jp][i] = mul2(s[jp][i], gg[i], p.neg_zero2);
        rows_partial(s, kk, sums, p.neg_zero2);
        const float sum = butterfly_of<2 * kRowsPerLane>(sums, lane);
        if (!first_row) {
            if ((lane & 17) == 16) *out = f32_to_bf16_bits(sum);
            out += p.out_stride;
        }
        const float d = (bf16_bits_to_f32(x.v) - sum) * x.beta;
#pragma unroll
        for (int jp = 0; jp < kPairs; ++jp) {
            const f32x2 delta = pack2(__shfl_sync(FULL, d, 4 * jp), __shfl_sync(FULL, d, 4 * jp + 2));
#pragma unroll
            for (int i = 0; i < 4; ++i) s[jp][i] = add2(s[jp][i], mul2(kk[i], delta, p.neg_zero2));
        }
        const f32x2 qq[4] = {pack2(x.q.x, x.q.x), pack2(x.q.y, x.q.y), pack2(x.q.z, x.q.z), pack2(x.q.w, x.q.w)};
        rows_partial(s, qq, sums + kRowsPerLane, p.neg_zero2);
    };
    if (n > 0) {
        CookedRow ring[kAhead];  // row r waits in ring[r % kAhead]
#pragma unroll
        for (int j = 0; j < kAhead; ++j) ring[j] = fetch(min(j, n - 1));
        int r = 0;
        for (; r + kAhead <= n; r += kAhead)
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                const CookedRow x = ring[j];
                ring[j] = fetch(min(r + j + kAhead, n - 1));
                step(x, r + j == 0);
            }
#pragma unroll
        for (int j = 0; j < kAhead; ++j)
            if (r + j < n) step(ring[j], r + j == 0);
        const float o = butterfly_of<2 * kRowsPerLane>(sums, lane);
        if ((lane & 17) == 16) *out = f32_to_bf16_bits(o);
    }
    store_rows_global<S>(reinterpret_cast<S*>(p.state_out) + s_elem, uw, lane, s);
}

// The same for launches of more units than a row's latency matters to: eight lanes to a value row (recurrence_octet.cuh), four rows a thread,
// so half a unit a block of four warps, the cooked rows through shared memory, four at a time.  701 rows of 2, 3 and 4 prompts, f32:
// 699 -> 656, 1,037 -> 930 and 1,240 -> 1,206 us (bf16, 3: 1,187 -> 1,037); one prompt 403 -> 419, hence the line in rows_launch.
constexpr int kOctR = 4, kOctParts = DV / (4 * kOctR * kRowsWarps);
constexpr int kStageRows = 4, kStages = 3;  // rows that arrive and are waited for together, such groups in shared memory
struct __align__(16) StagedRow {
    float k[DK], g[DK], q[DK];
    uint16_t v[DV];
    float beta;
};

template <typename S>
__global__ void __launch_bounds__(kRowsThreads, kPerSm) rows_octet_kernel(const __grid_constant__ RowsParams p) {
    constexpr int R = kOctR;
    __shared__ StagedRow ring[kStages][kStageRows];
    grid_ready();
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const unsigned unit = blockIdx.x / kOctParts;
    const int uw = (int)(blockIdx.x % kOctParts) * kRowsWarps + warp;  // this warp's place among the unit's
    const int h = (int)(unit % (unsigned)p.H), b = (int)(unit / (unsigned)p.H);
    const int r0 = p.cu ? p.cu[b] : 0, all = p.cu ? p.cu[b + 1] - r0 : p.rows1;
    const int n = min(max(all - p.row_shift, 0), p.pass_rows);
    if (n == 0 && p.state_in == p.state_out) return;
    const long long s_elem = (p.state_off ? p.state_off[b] : 0) + (long long)h * DV * DK;
    const long long first = (long long)b * p.pass_rows * p.H + h;  // (row, head) index of the pass's row 0
    auto fetch = [&](int stage) {  // 16 or 8 bytes a thread and row
#pragma unroll
        for (int i = 0; i < kStageRows; ++i) {
            const int r = stage * kStageRows + i;
            if (r >= n) break;
            StagedRow& x = ring[stage % kStages][i];
            const long long rh = first + (long long)r * p.H, at = rh * DK;
            if (t < 32) oct::copy16(&x.k[t * 4], p.k + at + t * 4);
            else if (t < 64) oct::copy16(&x.g[(t - 32) * 4], p.g + at + (t - 32) * 4);
            else if (t < 96) oct::copy16(&x.q[(t - 64) * 4], p.q + at + (t - 64) * 4);
            else oct::copy8(&x.v[(t - 96) * 4], p.v + at + (t - 96) * 4);
            if (t == 0) oct::copy4(&x.beta, p.beta + rh);
        }
        oct::copies_commit();
    };
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) fetch(i);
    f32x2 s[R][oct::kRowPairs];
    oct::load_rows(reinterpret_cast<const S*>(p.state_in) + s_elem, uw, lane, s);
    // As above, a row's read-out is reduced together with the next row's k-product: lanes 0-3 of a group receive its four rows' k-products, lanes
    // 4-7 the previous row's read-outs.
    float sums[2 * R] = {};
    const int mine = uw * 4 * R + (lane >> 3) * R + (lane & 3);  // the value row whose sums this lane receives
    const bool reads_out = (lane & 4) != 0;
    uint16_t* out = p.out + ((long long)r0 + p.row_shift) * p.out_stride + (long long)h * DV + mine;
    for (int stage = 0; stage * kStageRows < n; ++stage) {
        oct::copies_wait<kStages - 2>();
        __syncthreads();  // the group is there for all, and nobody reads the one before any more
        fetch(stage + kStages - 1);
#pragma unroll
        for (int i = 0; i < kStageRows; ++i) {
            const int r = stage * kStageRows + i;
            if (r >= n) break;
            const StagedRow& x = ring[stage % kStages][i];
            f32x2 kk[oct::kRowPairs], gg[oct::kRowPairs], qq[oct::kRowPairs];
            oct::load_leaves(x.g, lane, gg);
            oct::load_leaves(x.k, lane, kk);
            const float v = bf16_bits_to_f32(x.v[mine]), beta = x.beta;
            if constexpr (sizeof(S) == 2) {
                if (r != 0) oct::round_rows(s);  // after a row's read-out; the last row's rounding is the store's
            }
            oct::decay_rows(s, gg, p.neg_zero2);
            oct::rows_partial(s, kk, sums, p.neg_zero2);
            const float sum = butterfly_of<2 * R>(sums, lane, 4);
            if (r != 0) {
                if (reads_out) *out = f32_to_bf16_bits(sum);
                out += p.out_stride;
            }
            oct::update_rows<R, 1>(s, kk, (v - sum) * beta, lane, p.neg_zero2);
            oct::load_leaves(x.q, lane, qq);
            oct::rows_partial(s, qq, sums + R, p.neg_zero2);
        }
    }
    if (n > 0) {
        const float o = butterfly_of<2 * R>(sums, lane, 4);
        if (reads_out) *out = f32_to_bf16_bits(o);
    }
    oct::store_rows(reinterpret_cast<S*>(p.state_out) + s_elem, uw, lane, s);
}

// The gated RMSNorm of every row (kda.cu:188-201), one warp per (row, head): `out` holds bf16(y) and receives the output.
__global__ void __launch_bounds__(128) rows_norm_kernel(const __grid_constant__ RowsParams p) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31;
    const unsigned quads = (unsigned)(p.max_rows + 3) / 4, unit = blockIdx.x / quads;
    const int j = (int)(blockIdx.x % quads) * 4 + (threadIdx.x >> 5);
    const int h = (int)(unit % (unsigned)p.H), b = (int)(unit / (unsigned)p.H);
    const int r0 = p.cu ? p.cu[b] : 0, n = p.cu ? p.cu[b + 1] - r0 : p.rows1;
    if (j >= n) return;
    const long long gr = (long long)r0 + j, col = (long long)h * DV + lane * 4;
    uint16_t* dst = p.out + gr * p.out_stride + col;
    const uint2 yb = *reinterpret_cast<const uint2*>(dst), gb = *reinterpret_cast<const uint2*>(p.gate + gr * p.gate_stride + col);
    const uint2 wb = *reinterpret_cast<const uint2*>(p.norm_w + lane * 4);
    const uint32_t yw4[4] = {yb.x << 16, yb.x & 0xffff0000u, yb.y << 16, yb.y & 0xffff0000u};
    const uint32_t gw4[4] = {gb.x << 16, gb.x & 0xffff0000u, gb.y << 16, gb.y & 0xffff0000u};
    const uint32_t nw4[4] = {wb.x << 16, wb.x & 0xffff0000u, wb.y << 16, wb.y & 0xffff0000u};
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) ss = ss + __uint_as_float(yw4[i]) * __uint_as_float(yw4[i]);
    ss = butterfly1(ss);
    const float rinv = 1.0f / sqrtf(ss / (float)DV + p.eps);
    uint16_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float yn = __uint_as_float(yw4[i]) * rinv;
        const float yw = __uint_as_float(nw4[i]) * yn;
        o[i] = f32_to_bf16_bits(yw * sigmoidf_(__uint_as_float(gw4[i])));
    }
    *reinterpret_cast<uint2*>(dst) = make_uint2((uint32_t)o[0] | ((uint32_t)o[1] << 16), (uint32_t)o[2] | ((uint32_t)o[3] << 16));
}

}  // namespace

int rows_launch(RowsParams p, int batch, bool bf16_state, cudaStream_t stream) {
    p.neg_zero2 = 0x8000000080000000ull;
    const long long units = (long long)p.H * batch;
    // From four blocks of rows_kernel on some SM, four warps a scheduler.  Up to three a row's latency still counts: 256 rows, f32, 80, 96 and
    // 104 units 192, 199 and 209 us on rows_kernel, 222, 227 and 234 on the other; 112, 128 and 208 units 246, 256 and 391 against 235, 242 and 348
    // (bf16 219, 224 and 232 against 250, 255 and 261; 280, 287 and 439 against 263, 269 and 384).
    const bool many = units * kParts > 3LL * sm_count();
    const long long blocks = units * (many ? kOctParts : kParts);
    if (units * kParts > 0x7fffffffLL) return kInvalid;
    using Kernel = void (*)(RowsParams);
    static const Kernel kernels[2][2] = {{rows_kernel<float>, rows_kernel<__nv_bfloat16>}, {rows_octet_kernel<float>, rows_octet_kernel<__nv_bfloat16>}};
    const Kernel kernel = kernels[many][bf16_state];
    // Blocks that start while the prologue before them still fills most SMs would crowd onto the SMs that free up first, and
    // a row takes as long as the fullest SM needs: shared memory nobody uses keeps a launch to its fair share of blocks per SM (701 rows
    // of two prompts without it 1,074 us, so 656).
    constexpr size_t kSmemPerSm = 227 * 1024, kRing = kStages * kStageRows * sizeof(StagedRow);
    const size_t own = many ? kRing : 0;
    const long long share = (blocks + sm_count() - 1) / sm_count();
    const size_t pad = share < kPerSm ? kSmemPerSm / (size_t)(share + 1) + 1024 - own : 0;
    static int configured[2][2] = {{-1, -1}, {-1, -1}};
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured[many][bf16_state] != dev) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmemPerSm - own));
        if (e != cudaSuccess) return (int)e;
        configured[many][bf16_state] = dev;
    }
    return launch_early(kernel, (unsigned)blocks, kRowsThreads, pad, stream, p);
}

int rows_norm_launch(const RowsParams& p, int batch, cudaStream_t stream) {
    const long long blocks = (long long)p.H * batch * ((p.max_rows + 3) / 4);
    if (blocks > 0x7fffffffLL) return kInvalid;
    return blocks == 0 ? 0 : launch_early(rows_norm_kernel, (unsigned)blocks, kRowsThreads, 0, stream, p);
}

}  // namespace kda
