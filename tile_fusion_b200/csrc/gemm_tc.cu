// Host side of the ticket executor's tensor-core producer (gemm_tc.cuh), and the dense product alone.
#include "gemm_tc.cuh"

#include <string>

#include "gemm_tc_host.h"
#include "row_gemm.h"
#include "tf_internal.h"

namespace tfk {

static_assert(kTcRowsHost == kTcRows, "host and device tile heights differ");

// Wt_hi / Wt_lo [N][K] (K contiguous) from W [K][N], or from W [N][K] when w_transposed.
__global__ void split_weight_kernel(const float *__restrict__ W, int w_transposed, int K, int N,
                                    float *__restrict__ hi, float *__restrict__ lo) {
  const long long total = (long long)K * N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int n = (int)(i / K), k = (int)(i % K);
    const float w = w_transposed ? W[i] : W[(size_t)k * N + n];
    const float h = tf32_round(w);
    hi[i] = h;
    lo[i] = w - h;
  }
}

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess
               ? (EncodeTiledFn)p
               : (EncodeTiledFn) nullptr;
  }();
  return fn;
}

bool tc_supported(int K, int N) { return K >= 4 && K % 4 == 0 && N >= 16 && N % 16 == 0 && N <= kTcMaxN; }

// fp32 row-major [rows][K] tensor with rows ld floats apart (0: K), box = 32 columns (128 bytes) x box_rows, zero fill
int tc_make_map(CUtensorMap *out, const float *base, long long rows, int K, int box_rows, int ld, bool swizzle) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return tf::fail(TF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) return tf::fail(TF_ERR_ARG, "tensor-core producer: operand must be 16-byte aligned");
  cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)(ld > 0 ? ld : K) * 4};
  cuuint32_t box[2] = {(cuuint32_t)kTcKSlice, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(base), gdim, gstride, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return tf::fail(TF_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return TF_OK;
}

cudaError_t tc_split_weight(const float *W, int w_transposed, int K, int N, float *hi, float *lo, cudaStream_t s) {
  const long long total = (long long)K * N;
  const int grid = (int)std::min<long long>((total + 255) / 256, 148LL * 8);
  split_weight_kernel<<<grid, 256, 0, s>>>(W, w_transposed, K, N, hi, lo);
  return cudaGetLastError();
}

}  // namespace tfk

// T = B * W on device pointers, nothing else.
extern "C" int tf_gemm_tc_dev(const float *B, const float *W, int w_transposed, int m, int K, int N, float *T,
                              void *stream) {
  if (!B || !W || !T) return tf::fail(TF_ERR_ARG, "tf_gemm_tc_dev: null argument");
  if (m <= 0 || !tfk::tc_supported(K, N))
    return tf::fail(TF_ERR_UNSUPPORTED, "tf_gemm_tc_dev: needs K % 4 == 0, N % 16 == 0, N <= 256");
  cudaStream_t s = (cudaStream_t)stream;
  float *hi = nullptr, *lo = nullptr;
  int *err = nullptr;
  const size_t wn = (size_t)tfk::row_gemm_pad_n(N) * tfk::row_gemm_pad_k(K);
  cudaError_t e = cudaMalloc(&hi, wn * 4);
  if (e == cudaSuccess) e = cudaMalloc(&lo, wn * 4);
  if (e == cudaSuccess) e = cudaMalloc(&err, 4);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, 4, s);
  int rc = TF_OK;
  if (e != cudaSuccess) rc = tf::fail(TF_ERR_NOMEM, std::string("tf_gemm_tc_dev: ") + cudaGetErrorString(e));
  if (rc == TF_OK) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    e = tfk::row_gemm_split(W, w_transposed, K, N, tfk::kSumsFree, hi, lo, s);
    if (e == cudaSuccess) rc = tfk::row_gemm(B, m, K, K, W, w_transposed, hi, lo, N, T, N, false, tfk::kSumsFree, err, 1 << 20, sms, s);
    if (e == cudaSuccess && rc == TF_OK) e = cudaStreamSynchronize(s);
    int h_err = 0;
    if (e == cudaSuccess && rc == TF_OK) e = cudaMemcpy(&h_err, err, 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = tf::fail(TF_ERR_CUDA, std::string("tf_gemm_tc_dev: ") + cudaGetErrorString(e));
    else if (h_err) rc = tf::fail(TF_ERR_TIMEOUT, "tf_gemm_tc_dev: a bounded wait on a copy or on the tensor core ran out");
  }
  cudaFree(hi); cudaFree(lo); cudaFree(err);
  return rc;
}
