// SDDMM-SpMM, D = (A .* (Q K^T)) V, over the units of the balanced gather (gather.h); the sampled values are never stored.
//
// Per nonzero one row of K and one row of V come from L2 (from HBM where they exceed it), so what bounds the product is
// the same as in gather.cu: how many of those reads are in flight and how evenly they are spread.  A group of 16 lanes (8
// where neither row is wider than 32 columns) works through a unit as one stream of nonzeros, a lane holding one or two
// float4 of each row.  For four nonzeros at a time it issues the rows of K and the rows of V, which do not wait for the
// dot products; the partial dot products are then reduced across the group in one transposed pass (five shuffles for the
// four of them) and the rows of V are added.  The row of Q that follows is read while a row is worked on.  Pieces of long
// rows leave their sums in slots that the last piece adds up in order.  The groups of a warp step together, so that every
// shuffle is one of the whole warp; a group that has finished its unit repeats its last step without a result.
//
// R-MAT n = 262 144, degree 32, K = 64, N = 128: 494 us (12.0 TB/s of row reads; 589 with 16 warps per SM and every column tested for
// whether it exists; two sets of rows in turn, on 12 warps, 654).  The ticket executor took 1 695 (its warps waited at
// barriers behind long rows); a warp per nonzero, one float2 and one float4 a lane, 805 (50 instructions per nonzero, 46 %
// of the issue slots, 16 warps per SM waiting for L2 most of the time).
#include <algorithm>

#include "gather.h"
#include "kernels.cuh"

namespace tfk {

namespace {

constexpr int kSdThreads = 128;
// CTAs per SM: what the registers of a lane's rows leave room for.  Every further warp hides latency: K = N = 64: 487 us with 16
// warps per SM, 415 with 20, 391 with 24; K = 64, N = 128: 563, 494 and (spilling) 681; K = 100, N = 128: 661 with 16, 1 071
// (spilling) with 20.
__host__ __device__ constexpr int sd_ctas(int qk, int qn) { return qk + qn == 2 ? 6 : (qk + qn == 3 ? 5 : 4); }

// Columns of one lane: Q float4 that are 4 * G columns apart (VEC), or 4 * Q single columns that are G apart; those that do
// not exist read as zero.  (FULL: all exist.)
template <int G, int Q, bool VEC, bool FULL = false>
__device__ __forceinline__ void load_cols(float (&x)[4 * Q], const float *row, int lane, int width) {
#pragma unroll
  for (int j = 0; j < Q; ++j) {
    if (VEC && FULL) {
      const float4 t = __ldg(reinterpret_cast<const float4 *>(row) + lane + j * G);
      x[4 * j] = t.x; x[4 * j + 1] = t.y; x[4 * j + 2] = t.z; x[4 * j + 3] = t.w;
    } else if (VEC) {
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
      if (4 * (lane + j * G) < width) t = __ldg(reinterpret_cast<const float4 *>(row) + lane + j * G);
      x[4 * j] = t.x; x[4 * j + 1] = t.y; x[4 * j + 2] = t.z; x[4 * j + 3] = t.w;
    } else {
#pragma unroll
      for (int i = 4 * j; i < 4 * j + 4; ++i) x[i] = lane + G * i < width ? __ldg(row + lane + G * i) : 0.f;
    }
  }
}
// The same of a row of V, for columns whose sums are not stored where they do not exist: the last four again there.
template <int G, int Q, bool VEC>
__device__ __forceinline__ void load_any(float (&x)[4 * Q], const float *row, const int (&at)[Q], int lane, int width) {
  if (!VEC) {
    load_cols<G, Q, VEC>(x, row, lane, width);
  } else {
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      const float4 t = __ldg(reinterpret_cast<const float4 *>(row + at[j]));
      x[4 * j] = t.x; x[4 * j + 1] = t.y; x[4 * j + 2] = t.z; x[4 * j + 3] = t.w;
    }
  }
}
template <int G, int Q, bool VEC>
__device__ __forceinline__ void store_cols(float *row, const float (&x)[4 * Q], int lane, int width) {
#pragma unroll
  for (int j = 0; j < Q; ++j) {
    if (VEC) {
      if (4 * (lane + j * G) < width)
        reinterpret_cast<float4 *>(row)[lane + j * G] = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
    } else {
#pragma unroll
      for (int i = 4 * j; i < 4 * j + 4; ++i)
        if (lane + G * i < width) row[lane + G * i] = x[i];
    }
  }
}

// G: lanes per group.  QK, QN: float4 of K and of V per lane.  KVEC, NVEC: rows start on 16-byte boundaries.  KFULL: every lane has
// all its columns of K.
template <int G, int QK, int QN, bool KVEC, bool KFULL, bool NVEC>
__global__ void __launch_bounds__(kSdThreads, sd_ctas(QK, QN)) sddmm_gather_kernel(const GatherParams P, const float *__restrict__ Qm,
                                                                     const float *__restrict__ Km, int kq, int m) {
  constexpr int B = 4;  // nonzeros at a time
  static_assert(tf::kGatherBatch % B == 0, "a batch of the plan is worked on in halves");
  const int lane = threadIdx.x & (G - 1);
  const int nv = P.n_cols;
  int at[QN];
#pragma unroll
  for (int j = 0; j < QN; ++j) at[j] = min(4 * (lane + j * G), (nv - 4) & ~3);
  int unit = blockIdx.x * (kSdThreads / G) + threadIdx.x / G;
  const bool has = unit < P.n_units;
  unit = min(unit, P.n_units - 1);
  const int4 u = __ldg(P.units + unit);
  const bool piece = u.w >= 0;
  const int4 h = piece ? __ldg(P.heavy + u.w) : make_int4(0, 0, 0, 0);
  const bool listed = P.rows != nullptr;
  // a piece belongs to one row; otherwise `row` is the row at position `pos`, `row_next` the one behind it (the entries that
  // fill up a unit follow its last row end and name none: any row that exists will do)
  int pos = u.x, row, row_next;
  auto row_at = [&](int p) { return listed ? __ldg(P.rows + p) : min(p, m - 1); };
  row = piece ? h.x : row_at(pos);
  row_next = piece ? row : row_at(pos + 1);
  float q[4 * QK], q_next[4 * QK], acc[4 * QN];
  load_cols<G, QK, KVEC, KFULL>(q, Qm + (size_t)row * kq, lane, kq);
  load_cols<G, QK, KVEC, KFULL>(q_next, Qm + (size_t)row_next * kq, lane, kq);
#pragma unroll
  for (int i = 0; i < 4 * QN; ++i) acc[i] = 0.f;
  const int4 *pc = reinterpret_cast<const int4 *>(P.cols + u.y);
  const float4 *pv = reinterpret_cast<const float4 *>(P.vals + u.y);
  const int steps = has ? u.z * (tf::kGatherBatch / B) : 0;
  const int all = __reduce_max_sync(kFull, steps);
  int4 nxt = __ldg(pc);
  for (int b = 0; b < all; ++b) {
    const bool live = b < steps;
    const int c[B] = {nxt.x, nxt.y, nxt.z, nxt.w};
    float x[B][4 * QK], y[B][4 * QN], part[B];
#pragma unroll
    for (int t = 0; t < B; ++t) {
      const size_t col = (size_t)(unsigned)(c[t] & 0x7fffffff);
      load_cols<G, QK, KVEC, KFULL>(x[t], Km + col * kq, lane, kq);
      load_any<G, QN, NVEC>(y[t], P.dense + col * nv, at, lane, nv);
    }
    const float4 f = __ldg(pv);
    const float w[B] = {f.x, f.y, f.z, f.w};
    if (b + 1 < steps) {
      ++pc; ++pv;
      nxt = __ldg(pc);
    }
    // the rows end here and there in the batch, so the dot products take the row of Q along as it changes
    unsigned ends = 0;
#pragma unroll
    for (int t = 0; t < B; ++t) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < 4 * QK; ++i) s = fmaf(q[i], x[t][i], s);
      part[t] = s;
      if (live && c[t] < 0) {
        ends |= 1u << t;
        if (!piece) {
#pragma unroll
          for (int i = 0; i < 4 * QK; ++i) q[i] = q_next[i];
          row_next = row_at(pos + 1 + __popc(ends));
          load_cols<G, QK, KVEC, KFULL>(q_next, Qm + (size_t)row_next * kq, lane, kq);
        }
      }
    }
    // transposed reduction: afterwards the G / 4 lanes from G / 4 * t on hold the dot product of nonzero t
    float h2[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const bool up = lane & (G / 2);
      const float send = up ? part[i] : part[i + 2], keep = up ? part[i + 2] : part[i];
      h2[i] = keep + __shfl_xor_sync(kFull, send, G / 2);
    }
    const bool up = lane & (G / 4);
    const float send = up ? h2[0] : h2[1], keep = up ? h2[1] : h2[0];
    float dot = keep + __shfl_xor_sync(kFull, send, G / 4);
#pragma unroll
    for (int d = G / 8; d > 0; d /= 2) dot += __shfl_xor_sync(kFull, dot, d);
#pragma unroll
    for (int t = 0; t < B; ++t) {
      const float s = __shfl_sync(kFull, dot, G / 4 * t, G) * w[t];
#pragma unroll
      for (int i = 0; i < 4 * QN; ++i) acc[i] = fmaf(s, y[t][i], acc[i]);
      if (ends >> t & 1u) {
        float *o = piece ? P.partial + (size_t)pos * P.partial_ld : P.out + (size_t)row_at(pos) * nv;
        store_cols<G, QN, NVEC>(o, acc, lane, nv);
#pragma unroll
        for (int i = 0; i < 4 * QN; ++i) acc[i] = 0.f;
        if (!piece) ++pos;
      }
    }
  }
  // the group that delivers the last piece of a long row adds them up
  const bool deliver = has && piece;
  if (!__any_sync(kFull, deliver)) return;
  __threadfence();
  __syncwarp();
  int last = 0;
  if (deliver && lane == 0) last = atomicAdd(P.heavy_cnt + u.w, 1) == h.z - 1;
  last = __shfl_sync(kFull, last, 0, G);
  if (!last) return;
  __threadfence();
  if (lane == 0) P.heavy_cnt[u.w] = 0;  // ready for the next launch
#pragma unroll
  for (int i = 0; i < 4 * QN; ++i) acc[i] = 0.f;
  const float *ps = P.partial + (size_t)h.y * P.partial_ld;
#pragma unroll 4
  for (int s = 0; s < h.z; ++s, ps += P.partial_ld) {
#pragma unroll
    for (int i = 0; i < 4 * QN; ++i) {
      const int col = NVEC ? 4 * (lane + i / 4 * G) + i % 4 : lane + G * i;
      if (col < nv) acc[i] += __ldcg(ps + col);
    }
  }
  store_cols<G, QN, NVEC>(P.out + (size_t)h.x * nv, acc, lane, nv);
}

typedef void (*SddmmFn)(const GatherParams, const float *, const float *, int, int);
template <int G, int QK, int QN>
SddmmFn pick(bool kvec, bool nvec, int kq) {
  if (!kvec) return nvec ? (SddmmFn)sddmm_gather_kernel<G, QK, QN, false, false, true> : (SddmmFn)sddmm_gather_kernel<G, QK, QN, false, false, false>;
  if (kq == 4 * QK * G) return nvec ? (SddmmFn)sddmm_gather_kernel<G, QK, QN, true, true, true> : (SddmmFn)sddmm_gather_kernel<G, QK, QN, true, true, false>;
  return nvec ? (SddmmFn)sddmm_gather_kernel<G, QK, QN, true, false, true> : (SddmmFn)sddmm_gather_kernel<G, QK, QN, true, false, false>;
}

}  // namespace

int sddmm_resident(int kq, int nv) {
  return kSdThreads * (sddmm_group(kq, nv) == 8 ? sd_ctas(1, 1) : sd_ctas(kq <= 64 ? 1 : 2, nv <= 64 ? 1 : 2));
}
int sddmm_group(int kq, int nv) { return std::max(kq, nv) <= 32 ? 8 : 16; }
bool sddmm_gather_supported(int kq, int nv) { return kq >= 1 && kq <= 128 && nv >= 1 && nv <= 128; }

cudaError_t launch_sddmm_gather(const GatherParams &p, const float *Q, const float *K, int kq, int m, cudaStream_t s) {
  if (p.n_units <= 0) return cudaSuccess;
  const int nv = p.n_cols, group = sddmm_group(kq, nv);
  auto on = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const bool kvec = kq % 4 == 0 && on(Q) && on(K), nvec = nv % 4 == 0 && on(p.dense) && on(p.out);  // (partial_ld is a multiple of four)
  SddmmFn f = group == 8  ? pick<8, 1, 1>(kvec, nvec, kq)
              : kq <= 64 ? (nv <= 64 ? pick<16, 1, 1>(kvec, nvec, kq) : pick<16, 1, 2>(kvec, nvec, kq))
                         : (nv <= 64 ? pick<16, 2, 1>(kvec, nvec, kq) : pick<16, 2, 2>(kvec, nvec, kq));
  f<<<(p.n_units + kSdThreads / group - 1) / (kSdThreads / group), kSdThreads, 0, s>>>(p, Q, K, kq, m);
  return cudaGetLastError();
}

}  // namespace tfk
