// What the two projection kernels' translation units share.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace kda {

// One GEMM of a launch on SM pairs: tensor maps of the weight (boxes of 128 rows), the activations (boxes of row_tile / 2 rows)
// and, for bf16 results in aligned rows, of the output (boxes of 16 rows x 64 features); (k or feature, row, group), or
// (., group, row) when `swapped`.
struct PairProblem {
    CUtensorMap tm_w, tm_x, tm_out;
    void* out;
    long long ldo, o_gstride;
    int rows, n, kblocks, segments;  // k blocks of 64; k runs in `segments` equal parts
    int out_f32, tensor_out;
    int row_tile, n_tiles, r_tiles;
    int w_swapped, x_swapped, out_swapped;
    long long tiles;
};

constexpr int kPairProblems = 2;
constexpr int kPairSplitRows = 192;  // rows per tile at most when k runs in segments
// proj_gemm_pair.cu: launches the tiles of n (1 or 2) problems.
int proj_gemm_pair_launch(const PairProblem* problems, int n, int* status, cudaStream_t stream);

}  // namespace kda
