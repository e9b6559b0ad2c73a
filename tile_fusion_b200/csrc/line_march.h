// SpMM-SpMM on 2-D five-point operators: grid analysis (host) and launcher; the kernel is in line_march.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace tf {

constexpr int kLineSpan = 32;        // points of a line that a warp reads
constexpr int kLineOut = 28;         // of which the inner ones are rows of D that it completes
constexpr int kLineMaxClasses = 31;  // distinct coefficient vectors of an operator

// A five-point operator on an nx x ny grid in natural order: every row names its own point and all of its neighbours
// that exist, in column order.  Rows are grouped into classes of equal coefficient vectors {y-, x-, centre, x+, y+}
// (the most frequent one is class 0, class n_classes is the row that does not exist).  words[(y * tiles + t) * 8 + g]
// holds the classes of the points 28 t - 2 + 4 g + {0 .. 3} of line y, one per byte.
struct LineOp {
  bool ok = false;
  int nx = 0, ny = 0, tiles = 0, n_classes = 0;
  std::vector<float> dict;  // 8 floats per class
  std::vector<uint32_t> words;
};
void analyse_line_operator(int m, int n, const int *ap, const int *ai, const float *ax, LineOp &out);

}  // namespace tf

namespace tfk {

constexpr int kLineWarps = 4;  // per CTA

struct LineParams {
  const float *in;
  float *out;
  const unsigned *words_f, *words_a;
  int nx, ny, n_cols, tiles, chunks, seg_len, n_items;
  int y_begin, y_end;        // lines of D of this launch
  unsigned none_f, none_a;   // word of four points that do not exist
  float4 dict_f[2 * (tf::kLineMaxClasses + 1)], dict_a[2 * (tf::kLineMaxClasses + 1)];
};

// Fills in chunks, seg_len and n_items and launches; vec: rows start on 16-byte boundaries.
cudaError_t launch_line_march(LineParams &p, bool vec, bool same, int sm_count, cudaStream_t s);

}  // namespace tfk
