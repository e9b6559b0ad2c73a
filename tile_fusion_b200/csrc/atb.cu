// G = A^T * B for two tall fp32 matrices of up to a few hundred columns: the weight gradient of a layer's backward pass.
//
// The sum runs over all rows, the result is small: one output tile would keep one SM busy.  So the rows are cut into as many
// ranges as there are resident CTAs, each adds up the outer products of its rows for a tile of 128 x 128 (or 64 x 128) in
// registers, and a second launch adds the partial tiles in order, so the result does not depend on scheduling.  Rows are
// staged 16 at a time in shared memory, the next 16 on their way in registers meanwhile.  A thread holds 8 x 8 sums: per
// row it reads 16 floats for 64 fused multiply-adds, which are what bounds the kernel.  fp32 throughout, and the sums are
// shorter than one over all rows.
//
// m = 120 001, 128 x 128: 88 us; 40 x 128: 53 us.  The library GEMM behind torch.matmul took 205 and 188 (it cuts the
// sum into too few parts).
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "tf_internal.h"

namespace tfk {

namespace {

constexpr int kAtbThreads = 256, kAtbRows = 16, kAtbCols = 128;

// Four columns of a row, those that do not exist as zero.
__device__ __forceinline__ float4 load_four(const float *row, int col, int width, bool vec) {
  if (vec) return col < width ? __ldg(reinterpret_cast<const float4 *>(row + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(col < width ? __ldg(row + col) : 0.f, col + 1 < width ? __ldg(row + col + 1) : 0.f,
                     col + 2 < width ? __ldg(row + col + 2) : 0.f, col + 3 < width ? __ldg(row + col + 3) : 0.f);
}

// TN: columns of A per tile.  part[split][na][nb] receives the sums over the rows [split * rows, split * rows + rows).
template <int TN>
__global__ void __launch_bounds__(kAtbThreads, 2)
atb_kernel(const float *__restrict__ A, int na, const float *__restrict__ B, int nb, int m, int rows, bool vec_a, bool vec_b,
           float *__restrict__ part) {
  constexpr int QA = kAtbRows * TN / 4 / kAtbThreads, QB = kAtbRows * kAtbCols / 4 / kAtbThreads, H = TN / 64;
  __shared__ float4 sa[2][kAtbRows][TN / 4], sb[2][kAtbRows][kAtbCols / 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int a0 = blockIdx.y * TN, b0 = blockIdx.z * kAtbCols;
  const int r0 = blockIdx.x * rows, r1 = min(m, r0 + rows);
  float acc[4 * H][8];
#pragma unroll
  for (int i = 0; i < 4 * H; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  float4 ra[QA], rb[QB];
  auto fetch = [&](int r) {
#pragma unroll
    for (int i = 0; i < QA; ++i) {
      const int q = tid + i * kAtbThreads, row = r + q / (TN / 4), col = a0 + q % (TN / 4) * 4;
      ra[i] = row < r1 ? load_four(A + (size_t)row * na, col, na, vec_a) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < QB; ++i) {
      const int q = tid + i * kAtbThreads, row = r + q / (kAtbCols / 4), col = b0 + q % (kAtbCols / 4) * 4;
      rb[i] = row < r1 ? load_four(B + (size_t)row * nb, col, nb, vec_b) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int i = 0; i < QA; ++i) { const int q = tid + i * kAtbThreads; sa[buf][q / (TN / 4)][q % (TN / 4)] = ra[i]; }
#pragma unroll
    for (int i = 0; i < QB; ++i) { const int q = tid + i * kAtbThreads; sb[buf][q / (kAtbCols / 4)][q % (kAtbCols / 4)] = rb[i]; }
  };
  fetch(r0);
  stash(0);
  __syncthreads();
  int buf = 0;
  for (int r = r0; r < r1; r += kAtbRows) {
    const bool more = r + kAtbRows < r1;
    if (more) fetch(r + kAtbRows);
#pragma unroll
    for (int k = 0; k < kAtbRows; ++k) {
      float a[4 * H], b[8];
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const float4 v = sa[buf][k][h * 16 + ty];
        a[4 * h] = v.x; a[4 * h + 1] = v.y; a[4 * h + 2] = v.z; a[4 * h + 3] = v.w;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v = sb[buf][k][h * 16 + tx];
        b[4 * h] = v.x; b[4 * h + 1] = v.y; b[4 * h + 2] = v.z; b[4 * h + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < 4 * H; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if (more) stash(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }
  float *o = part + (size_t)blockIdx.x * na * nb;
#pragma unroll
  for (int i = 0; i < 4 * H; ++i) {
    const int row = a0 + i / 4 * 64 + ty * 4 + i % 4;
    if (row >= na) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int col = b0 + j / 4 * 64 + tx * 4 + j % 4;
      if (col < nb) o[(size_t)row * nb + col] = acc[i][j];
    }
  }
}

// out[i] = part[0][i] + part[1][i] + ..., in order; four lanes share an element's parts and are added pairwise.
__global__ void atb_sum_kernel(const float *__restrict__ part, int splits, int n, float *__restrict__ out) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / 4, l = threadIdx.x & 3;
  float s = 0.f;
  if (i < n)
#pragma unroll 8
    for (int k = l; k < splits; k += 4) s += __ldg(part + (size_t)k * n + i);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  if (i < n && l == 0) out[i] = s;
}

int atb_tile(int na) { return na <= 64 ? 64 : 128; }
int atb_splits(int m, int na, int nb) {
  const int tn = atb_tile(na), tiles = (na + tn - 1) / tn * ((nb + kAtbCols - 1) / kAtbCols);
  // two CTAs of an SM hide each other's waits; a range of fewer than 64 rows spends its time on the result
  return std::max(1, std::min(2 * 148 / tiles, (m + 63) / 64));
}

}  // namespace

}  // namespace tfk

extern "C" long long tf_atb_work_floats(int m, int na, int nb) {
  if (m <= 0 || na <= 0 || nb <= 0) return 0;
  return (long long)tfk::atb_splits(m, na, nb) * na * nb;
}

extern "C" int tf_atb_dev(const float *A, int na, const float *B, int nb, int m, float *out, float *work, long long work_floats,
                          void *stream) {
  if (!A || !B || !out || !work) return tf::fail(TF_ERR_ARG, "tf_atb_dev: null argument");
  if (m <= 0 || na <= 0 || nb <= 0 || (long long)na * nb > (1 << 24)) return tf::fail(TF_ERR_ARG, "tf_atb_dev: bad size");
  if (work_floats < tf_atb_work_floats(m, na, nb)) return tf::fail(TF_ERR_ARG, "tf_atb_dev: work space too small");
  cudaStream_t s = (cudaStream_t)stream;
  const int tn = tfk::atb_tile(na);
  int splits = tfk::atb_splits(m, na, nb);
  const int rows = ((m + splits - 1) / splits + tfk::kAtbRows - 1) / tfk::kAtbRows * tfk::kAtbRows;
  splits = (m + rows - 1) / rows;
  const dim3 grid(splits, (na + tn - 1) / tn, (nb + tfk::kAtbCols - 1) / tfk::kAtbCols);
  auto vec = [](const float *p, int n) { return n % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  (tn == 64 ? tfk::atb_kernel<64> : tfk::atb_kernel<128>)<<<grid, tfk::kAtbThreads, 0, s>>>(A, na, B, nb, m, rows, vec(A, na),
                                                                                            vec(B, nb), work);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) {
    const int n = na * nb;
    tfk::atb_sum_kernel<<<(4 * n + 255) / 256, 256, 0, s>>>(work, splits, n, out);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return tf::fail(TF_ERR_CUDA, std::string("tf_atb_dev: ") + cudaGetErrorString(e));
  return TF_OK;
}
