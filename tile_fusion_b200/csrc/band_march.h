// SpMM-SpMM on banded operators: host form and launcher; the kernel is in band_march.cu.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace tf {

// A square operator whose nonzeros lie within a block (64 or 128 rows) of the diagonal, in blocks of as many rows.  The
// nonzeros of a row are kept two by two in order, `pairs` of them for every row: quads[((b * pairs) + k) * block + r] =
// {byte offset, value, byte offset, value} of the nonzeros 2 k and 2 k + 1 of row r of block b, the offset being
// (column - row) * 128; places without a nonzero have the odd offset 1.
struct BandOp {
  bool ok = false;
  int block = 0, pairs = 0;
  std::vector<int> quads;  // 4 ints each
};
// Rows and reach of a square operator: false where it is no band or rows differ too much in length.
bool band_shape(int m, int n, const int *ap, const int *ai, int *reach, int *pairs);
void build_band_operator(int m, const int *ap, const int *ai, const float *ax, int block, int pairs, BandOp &out);

}  // namespace tf

namespace tfk {

struct BandParams {
  const int4 *quads_f, *quads_a;
  float *out;
  int *error;
  int m, n_cols, chunks, blocks, seg_blocks, pairs_f, pairs_a;
  int block_begin, block_end;  // blocks of rows of D of this launch
  int wait_limit;
  bool same;                   // one operator on both sides: quads_f is read for both products
};

// Tensor map of C (of D): boxes of 32 columns x `block` rows.
int band_make_map(CUtensorMap *out, const float *c, long long rows, int n_cols, int block);
constexpr int kBandThreads = 512;
// Shared memory of the kernel for these widths; plans whose operators need more than kBandSmemMax are not made.
constexpr int kBandSmemMax = 226 * 1024;
size_t band_smem(int block, int pairs_f, int pairs_a, bool same);
// Threads per CTA of the kernel that a plan runs on.
int band_threads(int block, const BandParams &p, int sm_count);
// Fills in chunks, blocks and seg_blocks and launches; tm_d: the map of D with boxes of 32 rows.
cudaError_t launch_band_march(const CUtensorMap &tm_c, const CUtensorMap &tm_d, int block, BandParams &p, int sm_count, cudaStream_t s);

}  // namespace tfk
