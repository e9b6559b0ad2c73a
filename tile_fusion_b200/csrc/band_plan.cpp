// Recognising a banded CSR operator and rewriting it for the band-marching executor (band_march.h).
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "band_march.h"
#include "segments.h"
#include "tf_internal.h"

namespace tf {

bool band_shape(int m, int n, const int *ap, const int *ai, int *reach, int *pairs) {
  if (m != n) return false;
  int far = 0, longest = 0;
  for (int r = 0; r < m; ++r) {
    longest = std::max(longest, ap[r + 1] - ap[r]);
    for (int j = ap[r]; j < ap[r + 1]; ++j) far = std::max(far, std::abs(ai[j] - r));
    if (far > 128) return false;
  }
  *reach = far;
  *pairs = std::max(1, (longest + 1) / 2);
  // every row takes as long as the longest: not worth it where that is half as much again as the average
  return 2LL * *pairs * m <= 3LL * ap[m] / 2 + 4LL * m;
}

void build_band_operator(int m, const int *ap, const int *ai, const float *ax, int block, int pairs, BandOp &out) {
  const size_t blocks = ((size_t)m + block - 1) / block;
  out.block = block;
  out.pairs = pairs;
  out.quads.assign(blocks * pairs * block * 4, 0);
  for (size_t i = 0; i < out.quads.size(); i += 2) out.quads[i] = 1;
  for (int r = 0; r < m; ++r)
    for (int j = ap[r]; j < ap[r + 1]; ++j) {
      const int k = j - ap[r];
      int *q = &out.quads[4 * (((size_t)(r / block) * pairs + k / 2) * block + r % block) + 2 * (k & 1)];
      q[0] = (ai[j] - r) * 128;
      std::memcpy(&q[1], &ax[j], 4);
    }
  out.ok = true;
}

}  // namespace tf

// Host-only view of the segment length, for tests.
extern "C" int tf_segment_preview(int n, long long columns, long long resident, int lead, int min_len) {
  if (n <= 0 || columns <= 0 || resident <= 0 || lead <= 0 || min_len <= 0) return TF_ERR_ARG;
  return tf::segment_length(n, columns, resident, lead, min_len);
}
