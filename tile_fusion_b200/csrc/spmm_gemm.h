// GeMM-SpMM in one launch, D = (A B) W, for star stencils on a grid (spmm_gemm.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <vector>

namespace tf {

constexpr int kStarRows = 128;  // grid points of a brick

// A five-point operator on an nx x ny grid or a seven-point one on nx x ny x nz, natural order, every row naming all of its
// neighbours that exist.
struct StarOp {
  int nx = 0, ny = 0, nz = 0;  // nx 0: the operator is none
  bool uniform = false;        // the coefficients are the same in every row: coef[0 .. 7]
  std::vector<float> coef;     // {z-, y-, x-, centre, x+, y+, z+, 0}, zero where there is no neighbour; else eight per row
};
void analyse_star_operator(int m, int n, const int *ap, const int *ai, const float *ax, StarOp &out);

// Bricks of 2^lx x 2^ly x 2^lz = 128 points that cover the grid, numbered along x, then y, then z.
struct BrickGrid {
  int nx, ny, nz, lx, ly, lz;
  int bx() const { return (nx + (1 << lx) - 1) >> lx; }
  int by() const { return (ny + (1 << ly) - 1) >> ly; }
  int bz() const { return (nz + (1 << lz) - 1) >> lz; }
  int bricks() const { return bx() * by() * bz(); }
};
// Points of B that a brick reads.
inline int brick_points(const BrickGrid &g) {
  const int x = 1 << g.lx, y = 1 << g.ly, z = 1 << g.lz;
  return (x + 2) * (y + 2) * z + (g.nz > 1 ? 2 * x * y : 0);
}
// The shape that costs least, of those that read at most `most` points: every brick its own work, full or not, and the points
// around it that it reads.  False where there is none.
bool choose_bricks(const StarOp &op, int most, BrickGrid &out);

}  // namespace tf

namespace tfk {

struct SpmmGemmParams {
  const float *b, *w;   // the weight: element (k, c) at k * w_k + c * w_c
  float *out;
  int *error;
  const float *coef;    // eight per row; null: uniform[] for all
  float uniform[8];
  tf::BrickGrid grid;
  int k, n, w_transposed, relu, wait_limit;
  int brick_begin, brick_end;
  // filled in by the launcher
  int n_pad, w_k, w_c, slices, stages, raws, accs, raw_bytes;
};

constexpr int kSpmmGemmThreads = 480;
int spmm_gemm_points(int K, int n);      // of B that a brick may read (shapes of the tensor-core tile)
bool spmm_gemm_resident(int K, int n);  // the weight is split by the kernel: no row_gemm_split
// hi, lo: row_gemm_split's.  Rows of B and D start on 16-byte boundaries.
int spmm_gemm(SpmmGemmParams p, const float *hi, const float *lo, int sm_count, cudaStream_t s);

}  // namespace tfk
