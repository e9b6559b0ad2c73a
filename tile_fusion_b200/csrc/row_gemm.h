// T = B * W for a tall B on the tensor cores (row_gemm.cu): the dense product of a GeMM-SpMM chain in a launch of its own.
#pragma once
#include <cuda_runtime.h>

namespace tfk {

struct RowGemmParams {
  const float *x;  // read directly where rows do not start on 16-byte boundaries (`direct`), and by the precise form's exact sums
  const float *w;  // (the latter) the weight from the panel's first column on: element (k, c) at k * w_k + c * w_c
  float *out;
  int *error;
  int m, n_real, n_pad, n_slices, tiles, stages, accs, ld_out, k, ld_x;
  int direct, relu, tma_store, wait_limit, w_k, w_c;
  int cut_low, small_first;  // the low halves of X are not rounded; the small products of a slice come first whatever the accumulators
};

// Whose sums a product's are, bit for bit: nobody's; the ticket executor's tile, where there is one (one accumulator whatever the
// width, no low half rounded); those of spmm_gemm.cu where that has one accumulator, above 128 columns (the small products of a
// slice first).
enum RowGemmSums { kSumsFree, kSumsTicket, kSumsSpmmGemm };
bool row_gemm_supported(int n);  // n <= 256 columns
// Which of its forms a product takes (see row_gemm.cu).
enum RowGemmForm { kRowTile, kRowPrecise, kRowFma };
RowGemmForm row_gemm_form(int K, int n);
int row_gemm_pad_n(int n);       // rows of the split weight
int row_gemm_pad_k(int k);       // floats per row of it
// hi, lo: row_gemm_pad_n(n) x row_gemm_pad_k(K) floats each.  W is K x n, or n x K when w_transposed.  (kRowFma needs neither:
// nothing is launched.)
cudaError_t row_gemm_split(const float *W, int w_transposed, int K, int n, RowGemmSums sums, float *hi, float *lo, cudaStream_t s);
// out[m][ld_out] (n columns written) = X[m][ld_x] (K columns read) * W, optionally max(0, .); hi, lo as row_gemm_split leaves
// them.  Rows of X on 16-byte boundaries come by TMA, others value by value; rows of `out` leave likewise.
// (hi, lo of a row_gemm_split of the same sums.)
int row_gemm(const float *X, int m, int K, int ld_x, const float *W, int w_transposed, const float *hi, const float *lo, int n,
             float *out, int ld_out, bool relu, RowGemmSums sums, int *error, int wait_limit, int sm_count, cudaStream_t s);

}  // namespace tfk
