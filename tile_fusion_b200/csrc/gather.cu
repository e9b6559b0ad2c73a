// Balanced gather: out = A * X on CSR operators without row reuse that a tile could hold (power-law graphs).
//
// The rows of X that the nonzeros name come from L2 (from HBM where X exceeds it), one row per nonzero, and nothing
// can be reused but by luck.  What bounds such a product is how many of those row reads are in flight and how evenly
// they are spread, so the work is cut by nonzeros and not by rows:
//   * The host cuts the nonzeros into units of about equal work (gather_plan.cpp): whole rows up to `target` nonzeros,
//     and pieces of the rows that are longer than that.
//   * A unit is worked on by a group of 8, 16 or 32 lanes, four columns per lane (one float4), so that a narrow X
//     still moves 512 bytes per warp instruction.  The group walks its nonzeros as one stream: eight row reads are
//     issued together whatever rows of A they belong to, and a bit in the column id says where a row of A ends.
//     Nothing waits at the head of a row, no two warps ever wait for each other, and because units are filled up to
//     whole batches and lanes without a column read the last one again, the loop has no bounds to check (ten
//     instructions per nonzero; a version that broadcast the entries by shuffles and checked bounds needed 37 and
//     filled two thirds of the issue slots).
//   * A piece of a long row leaves its sum in a slot of `partial`; the group that delivers the last piece of the row
//     adds the slots up in order, so a result does not depend on the order in which groups run.
// Products of a row are added in CSR order with fused multiply-adds from zero, as in the reference's row loop
// (SpMM_SpMM.cpp:211-248); only rows that were cut are added in pieces.
//
// A CTA is one warp.  Where a group is a whole warp (more than 64 columns) the entries are then the CTA's, so they and the addresses
// of the rows are worked out once by the uniform datapath and not by every lane; and a warp that has finished makes room for the
// next whatever its neighbours do.
//
// Measured (R-MAT, n = 500 009, degree 25, one product): 128 columns 383 us (17 TB/s of row reads, 15 % of them from L1), 100 columns
// 368, in CTAs of four warps 440 and 428, of eight 454 and 443; 64 columns 242, 48 columns 237 (a row costs its 128-byte lines, whole
// or not).  n = 200 000, degree 20, 64 columns, both products of a chain: 175 us, the ticket executor took 784 (58 % of its warps'
// time at barriers behind long rows).
// Eight reads in flight and 24 warps per SM: 28 warps 376 at 100 columns and slower at small sizes, 32 spill (307 at 64 columns); four
// reads and 40 warps, or asking for half a batch again as soon as it has been added up (569 at 100 columns), are slower, and so are 32
// lanes of two columns each for up to 64 (272; sixteen in flight 327).
#include <algorithm>

#include "gather.h"
#include "kernels.cuh"

namespace tfk {

namespace {

constexpr int kGatherThreads = 32, kGatherCtas = kGatherResident / kGatherThreads;
constexpr int kBatch = tf::kGatherBatch;

// The columns of one lane: four in a row (VEC), or E of them at the offsets `at`, those that do not exist clamped to one that does.
template <bool VEC, int E>
__device__ __forceinline__ float4 load_quad(const float *p, const int (&at)[4]) {
  if (VEC) return __ldg(reinterpret_cast<const float4 *>(p));
  return make_float4(__ldg(p), E > 1 ? __ldg(p + at[1]) : 0.f, E > 2 ? __ldg(p + at[2]) : 0.f, E > 3 ? __ldg(p + at[3]) : 0.f);
}
__device__ __forceinline__ void fma_quad(float4 &a, float v, const float4 &x) {
  a.x = fmaf(v, x.x, a.x); a.y = fmaf(v, x.y, a.y); a.z = fmaf(v, x.z, a.z); a.w = fmaf(v, x.w, a.w);
}

// G: lanes per group.  VIN: rows of X are read as float4, else E columns per lane, G apart.  VOUT: rows of the result are written
// as float4.
template <int G, bool VIN, bool VOUT, int E = 4>
__global__ void __launch_bounds__(kGatherThreads, kGatherCtas) gather_kernel(const GatherParams P) {
  static_assert(!VOUT || VIN, "strided columns are stored one by one");
  const int lane = threadIdx.x & (G - 1);
  const int panel = blockIdx.x / P.unit_blocks;
  const int unit = (blockIdx.x - panel * P.unit_blocks) * (kGatherThreads / G) + threadIdx.x / G;
  if (unit >= P.n_units) return;
  const int c0 = panel * P.panel_w, c1 = min(P.n_cols, c0 + P.panel_w);
  // A lane without a column of its own reads the last one again instead of branching around every load.
  const int own = c0 + (VIN ? lane * 4 : lane);
  const int left = c1 - own;  // columns of this lane that exist (VIN: from `own` on; else element e while G * e < left)
  const int col = left > 0 ? own : (VIN ? (c1 - 1) & ~3 : c1 - 1);
  const int at[4] = {0, G < left ? G : 0, 2 * G < left ? 2 * G : 0, 3 * G < left ? 3 * G : 0};
  const int4 u = __ldg(P.units + unit);
  const bool piece = u.w >= 0;
  const float *src = P.dense + col;
  const int ld_in = P.ld_in;
  float *dst = (piece ? P.partial : P.out) + own;
  const int ld_dst = piece ? P.partial_ld : P.ld_out;
  const bool relu = P.relu != 0 && !piece;
  const bool listed = P.rows != nullptr && !piece;
  int pos = u.x;
  int row = listed ? __ldg(P.rows + pos) : pos;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);

  auto put = [&](float *o, bool clamp) {
    if (clamp) { acc.x = fmaxf(acc.x, 0.f); acc.y = fmaxf(acc.y, 0.f); acc.z = fmaxf(acc.z, 0.f); acc.w = fmaxf(acc.w, 0.f); }
    constexpr int d = VIN ? 1 : G;
    if (VOUT) {
      if (left > 0) *reinterpret_cast<float4 *>(o) = acc;
    } else {
      if (0 < left) o[0] = acc.x;
      if (E > 1 && d < left) o[d] = acc.y;
      if (E > 2 && 2 * d < left) o[2 * d] = acc.z;
      if (E > 3 && 3 * d < left) o[3 * d] = acc.w;
    }
  };

  // columns are read one batch ahead, values with the rows they multiply; all lanes of the group read the same ones
  const int4 *pc = reinterpret_cast<const int4 *>(P.cols + u.y);
  const float4 *pv = reinterpret_cast<const float4 *>(P.vals + u.y);
  int4 nxt[kBatch / 4];
#pragma unroll
  for (int q = 0; q < kBatch / 4; ++q) nxt[q] = __ldg(pc + q);
  for (int b = 0; b < u.z; ++b) {
    int c[kBatch];
    float v[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch / 4; ++q) {
      c[4 * q] = nxt[q].x; c[4 * q + 1] = nxt[q].y; c[4 * q + 2] = nxt[q].z; c[4 * q + 3] = nxt[q].w;
    }
    float4 x[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch; ++q) x[q] = load_quad<VIN, E>(src + (size_t)(unsigned)(c[q] & 0x7fffffff) * ld_in, at);
    pc += kBatch / 4;
#pragma unroll
    for (int q = 0; q < kBatch / 4; ++q) {
      const float4 w = __ldg(pv + q);
      v[4 * q] = w.x; v[4 * q + 1] = w.y; v[4 * q + 2] = w.z; v[4 * q + 3] = w.w;
      nxt[q] = __ldg(pc + q);
    }
    pv += kBatch / 4;
#pragma unroll
    for (int q = 0; q < kBatch; ++q) {
      fma_quad(acc, v[q], x[q]);
      if (c[q] < 0) {  // the row (or piece) is complete
        put(dst + (size_t)row * ld_dst, relu);
        acc = make_float4(0.f, 0.f, 0.f, 0.f);
        ++pos;
        row = listed ? __ldg(P.rows + pos) : pos;  // (one entry more than there are rows, see the host plan)
      }
    }
  }
  if (!piece) return;
  // a piece of a long row has been delivered; the group that delivers the last one adds them up
  const unsigned gmask = G == 32 ? kFull : (((1u << (G & 31)) - 1u) << (threadIdx.x & 31 & ~(G - 1)));
  const int4 h = __ldg(P.heavy + u.w);
  __threadfence();
  __syncwarp(gmask);
  int last = 0;
  int *cnt = P.heavy_cnt + (size_t)u.w * P.panels + panel;
  if (lane == 0) last = atomicAdd(cnt, 1) == h.z - 1;
  last = __shfl_sync(gmask, last, 0, G);
  if (!last) return;
  __threadfence();
  if (lane == 0) *cnt = 0;  // ready for the next launch
  acc = make_float4(0.f, 0.f, 0.f, 0.f);  // (the entries that fill up the unit went into it: 0 * infinity)
  const float *ps = P.partial + (size_t)h.y * P.partial_ld + col;
  for (int s = 0; s < h.z; s += kBatch) {
    float4 x[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch; ++q) {
      const float *o = ps + (size_t)min(s + q, h.z - 1) * P.partial_ld;
      x[q] = VIN ? __ldcg(reinterpret_cast<const float4 *>(o)) : make_float4(__ldcg(o), __ldcg(o + at[1]), __ldcg(o + at[2]), __ldcg(o + at[3]));
    }
#pragma unroll
    for (int q = 0; q < kBatch; ++q)
      if (s + q < h.z) { acc.x += x[q].x; acc.y += x[q].y; acc.z += x[q].z; acc.w += x[q].w; }
  }
  put(P.out + own + (size_t)h.x * P.ld_out, P.relu != 0);
}

// Rows of n_cols floats to rows of ld, the next multiple of four, with zeros behind.  Memory bounds it where no thread divides
// for every element: a thread steps through (row, column) instead (100 000 rows of 47, two products of a graph behind it: 81 us, 75 now).
__global__ void pad_rows_kernel(const float *__restrict__ src, long long rows, int n_cols, int ld, float *__restrict__ dst) {
  const int q = ld / 4;
  const long long step = (long long)gridDim.x * blockDim.x, first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long dr = step / q;
  const int dc = (int)(step - dr * q);
  long long r = first / q;
  int c = (int)(first - r * q);
  while (r < rows) {
    const float *p = src + r * n_cols + 4 * c;
    const int left = n_cols - 4 * c;
    float4 v;
    v.x = __ldg(p);  // (left > 0: ld is less than four columns wider)
    v.y = left > 1 ? __ldg(p + 1) : 0.f;
    v.z = left > 2 ? __ldg(p + 2) : 0.f;
    v.w = left > 3 ? __ldg(p + 3) : 0.f;
    *reinterpret_cast<float4 *>(dst + r * ld + 4 * c) = v;
    r += dr;
    c += dc;
    if (c >= q) { c -= q; ++r; }
  }
}

typedef void (*GatherFn)(const GatherParams);
template <int G>
GatherFn pick(bool vec_out) { return vec_out ? gather_kernel<G, true, true> : gather_kernel<G, true, false>; }

// Rows read value by value: the lanes of a group and the columns of a lane, so that the fewest reads are made (a read brings G
// columns of 32 / G rows), with as few lanes as that allows.  (R-MAT n = 500 009, degree 25: 7 columns 493 us as 32 x 4, where columns that
// do not exist are read too, 106 like this; 31: 502 and 238, with 32 lanes 273; 47: 514 and 277; 57: 521 and 332, with 32 lanes 360.)
struct Single {
  int width, group;
  GatherFn f;
};
const Single kSingles[] = {{8, 8, gather_kernel<8, false, false, 1>},    {16, 8, gather_kernel<8, false, false, 2>},
                           {24, 8, gather_kernel<8, false, false, 3>},   {32, 8, gather_kernel<8, false, false, 4>},
                           {48, 16, gather_kernel<16, false, false, 3>}, {64, 16, gather_kernel<16, false, false, 4>},
                           {96, 32, gather_kernel<32, false, false, 3>}, {128, 32, gather_kernel<32, false, false, 4>}};

}  // namespace

// (R-MAT n = 500 000, degree 25, 32 columns: 377 us with 8 lanes, 703 with 16, 1 018 with 32.)
int gather_group(int n_cols) { return n_cols <= 32 ? 8 : (n_cols <= 64 ? 16 : 32); }

cudaError_t launch_gather(bool vec_in, bool vec_out, const GatherParams &p, cudaStream_t s) {
  if (p.n_units <= 0) return cudaSuccess;
  GatherFn f;
  GatherParams q = p;
  int group = gather_group(p.n_cols);
  q.panel_w = vec_in ? 4 * group : 128;
  if (!vec_in) {
    const Single *w = kSingles;
    while (w->width < std::min(p.n_cols, 128)) ++w;
    f = w->f;
    group = w->group;
  } else if (group == 8) f = pick<8>(vec_out);
  else if (group == 16) f = pick<16>(vec_out);
  else f = pick<32>(vec_out);
  q.panels = (p.n_cols + q.panel_w - 1) / q.panel_w;
  q.unit_blocks = (p.n_units + kGatherThreads / group - 1) / (kGatherThreads / group);
  f<<<q.unit_blocks * q.panels, kGatherThreads, 0, s>>>(q);
  return cudaGetLastError();
}

cudaError_t launch_pad_rows(const float *src, long long rows, int n_cols, int ld, float *dst, cudaStream_t s) {
  const long long total = rows * (ld / 4);
  if (total <= 0) return cudaSuccess;
  pad_rows_kernel<<<(int)std::min<long long>((total + 255) / 256, 148LL * 8), 256, 0, s>>>(src, rows, n_cols, ld, dst);
  return cudaGetLastError();
}

}  // namespace tfk
