// Recognising a CSR operator as a five-point operator on a 2-D grid (line_march.h).
#include <algorithm>
#include <cstring>
#include <map>
#include <array>

#include "line_march.h"

namespace tf {

void analyse_line_operator(int m, int n, const int *ap, const int *ai, const float *ax, LineOp &out) {
  out = LineOp();
  if (m != n || m < 6 || ap[1] - ap[0] != 3 || ai[0] != 0 || ai[1] != 1) return;
  const int nx = ai[2];  // the first row names its own point and its neighbours along x and y
  if (nx < 3 || m % nx != 0 || m / nx < 2) return;
  const int ny = m / nx;
  std::map<std::array<uint32_t, 5>, int> ids;
  std::vector<std::array<uint32_t, 5>> vecs;
  std::vector<long long> count;
  std::vector<uint8_t> cls((size_t)m);
  int last = -1;
  for (int y = 0, r = 0; y < ny; ++y)
    for (int x = 0; x < nx; ++x, ++r) {
      const int off[5] = {-nx, -1, 0, 1, nx};
      const bool in[5] = {y > 0, x > 0, true, x < nx - 1, y < ny - 1};
      std::array<uint32_t, 5> k{};
      int j = ap[r];
      for (int q = 0; q < 5; ++q) {
        if (!in[q]) continue;
        if (j >= ap[r + 1] || ai[j] != r + off[q]) return;  // a neighbour that is missing, or another column
        std::memcpy(&k[q], &ax[j++], 4);
      }
      if (j != ap[r + 1]) return;
      if (last < 0 || vecs[last] != k) {
        auto it = ids.find(k);
        if (it == ids.end()) {
          if ((int)vecs.size() >= kLineMaxClasses) return;
          it = ids.emplace(k, (int)vecs.size()).first;
          vecs.push_back(k);
          count.push_back(0);
        }
        last = it->second;
      }
      ++count[last];
      cls[r] = (uint8_t)last;
    }
  const int nc = (int)vecs.size();
  std::vector<int> order(nc), rank(nc);
  for (int i = 0; i < nc; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return count[a] > count[b]; });
  out.dict.assign((size_t)(nc + 1) * 8, 0.f);
  for (int i = 0; i < nc; ++i) {
    rank[order[i]] = i;
    std::memcpy(&out.dict[(size_t)i * 8], vecs[order[i]].data(), 20);
  }
  const int tiles = (nx + kLineOut - 1) / kLineOut;
  out.words.assign((size_t)ny * tiles * 8, 0x01010101u * (uint32_t)nc);
  for (int y = 0; y < ny; ++y)
    for (int t = 0; t < tiles; ++t)
      for (int i = 0; i < kLineSpan; ++i) {
        const int x = t * kLineOut - 2 + i;
        if (x < 0 || x >= nx) continue;
        uint32_t &w = out.words[((size_t)y * tiles + t) * 8 + i / 4];
        const int sh = 8 * (i & 3);
        w = (w & ~(0xFFu << sh)) | ((uint32_t)rank[cls[(size_t)y * nx + x]] << sh);
      }
  out.nx = nx; out.ny = ny; out.tiles = tiles; out.n_classes = nc;
  out.ok = true;
}

}  // namespace tf
