// Host side of the one-launch GeMM-SpMM (spmm_gemm.h): recognising the stencil and cutting its grid into bricks.
#include <algorithm>
#include <cmath>

#include "spmm_gemm.h"

namespace tf {

void analyse_star_operator(int m, int n, const int *ap, const int *ai, const float *ax, StarOp &out) {
  out = StarOp();
  if (m != n || m < 16) return;
  // the extents, from a row in the middle with the most neighbours
  int best = m / 2;
  for (int r = m / 2; r < std::min(m, m / 2 + 4096); ++r)
    if (ap[r + 1] - ap[r] > ap[best + 1] - ap[best]) best = r;
  long long up[4];
  int n_up = 0;
  for (int j = ap[best]; j < ap[best + 1]; ++j)
    if (ai[j] > best) {
      if (n_up == 3) return;
      up[n_up++] = (long long)ai[j] - best;
    }
  if (n_up < 2 || up[0] != 1 || up[1] < 4 || (n_up == 3 && up[2] % up[1] != 0)) return;
  const long long nx = up[1], ny = n_up == 3 ? up[2] / nx : m / nx, nz = n_up == 3 ? m / (nx * ny) : 1;
  if (ny < 2 || nx * ny * nz != m || (n_up == 3 && nz < 2)) return;
  const long long step[7] = {-nx * ny, -nx, -1, 0, 1, nx, nx * ny};
  out.coef.assign(8, 0.f);
  bool known[7] = {}, uniform = true;
  auto neighbours = [&](long long x, long long y, long long z, bool (&has)[7]) {
    has[0] = z > 0; has[1] = y > 0; has[2] = x > 0; has[3] = true; has[4] = x < nx - 1; has[5] = y < ny - 1; has[6] = z < nz - 1;
  };
  int r = 0;
  for (long long z = 0; z < nz; ++z)
    for (long long y = 0; y < ny; ++y)
      for (long long x = 0; x < nx; ++x, ++r) {
        bool has[7];
        neighbours(x, y, z, has);
        int j = ap[r];
        for (int i = 0; i < 7; ++i)
          if (has[i]) {
            if (j == ap[r + 1] || ai[j] != r + step[i]) return;
            if (!known[i]) { known[i] = true; out.coef[i] = ax[j]; }
            // (a coefficient that no row names may stand for one that is not there: it meets zeros)
            uniform = uniform && out.coef[i] == ax[j] && std::isfinite(ax[j]);
            ++j;
          }
        if (j != ap[r + 1]) return;
      }
  out.uniform = uniform;
  if (!uniform) {
    out.coef.assign(8 * (size_t)m, 0.f);
    r = 0;
    for (long long z = 0; z < nz; ++z)
      for (long long y = 0; y < ny; ++y)
        for (long long x = 0; x < nx; ++x, ++r) {
          bool has[7];
          neighbours(x, y, z, has);
          for (int i = 0, j = ap[r]; i < 7; ++i)
            if (has[i]) out.coef[8 * (size_t)r + i] = ax[j++];
        }
  }
  out.nx = (int)nx; out.ny = (int)ny; out.nz = (int)nz;
}

bool choose_bricks(const StarOp &op, int most, BrickGrid &out) {
  double least = -1;
  for (int lx = 2; lx <= 5; ++lx)
    for (int ly = 1; lx + ly <= 7; ++ly) {
      const int lz = 7 - lx - ly;
      if (op.nz == 1 ? lz != 0 : lz < 1) continue;
      const BrickGrid g{op.nx, op.ny, op.nz, lx, ly, lz};
      const double cost = (double)g.bricks() * (brick_points(g) + 2 * kStarRows);
      if (brick_points(g) <= most && (least < 0 || cost < least)) { least = cost; out = g; }
    }
  return least >= 0;
}

}  // namespace tf
