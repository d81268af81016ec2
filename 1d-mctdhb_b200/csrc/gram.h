// gram.h -- sizes of the Gram-matrix density kernels (gram_tmpl.cuh), shared
// with the host code that allocates their partial sums.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mctdhb {

__host__ __device__ constexpr int gram_p(int M) { return M * (M + 1) / 2; }
// complex entries of one block partial: the upper triangle of P x P, row-major
__host__ __device__ constexpr int gram_entries(int M) { return gram_p(M) * (gram_p(M) + 1) / 2; }
constexpr int kGramThreads = 256;
constexpr int kGramMaxBlocks = 296;  // 2 x 148: fixed, so the sums depend on (N, M) only

// A tile: rows of PS 16-byte words, PS a multiple of 8, column c of row r at
// word c ^ swz(r): the stores of 8 consecutive rows (one column) and the
// fragment loads of 4 rows x 2 columns each fall in 8 different bank groups
__host__ __device__ constexpr int gram_row_words(int M) { return (gram_p(M) + 7) / 8 * 8; }
__host__ __device__ constexpr int gram_swz(int r) { return ((r & 3) << 1) | ((r >> 2) & 1); }
// rows per tile: two blocks fit an SM (98 KB a tile at 6 orbitals)
__host__ __device__ constexpr int gram_rows(int M) { return M >= 7 ? 128 : 256; }
__host__ __device__ constexpr int gram_smem(int M) { return gram_rows(M) * gram_row_words(M) * 16; }

// blocks (= partial slices) for Dp rows: a function of (N, M) only
inline int gram_blocks(int M, uint32_t Dp) {
    const uint32_t need = (Dp + gram_rows(M) - 1) / gram_rows(M);
    return (int)(need < (uint32_t)kGramMaxBlocks ? need : (uint32_t)kGramMaxBlocks);
}

}  // namespace mctdhb
