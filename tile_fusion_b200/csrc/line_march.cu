// SpMM-SpMM on 2-D five-point operators (line_march.h): D = A * (F * C), one launch, T = F * C in registers.
//
// A warp owns 32 consecutive points of a line and 16 dense columns (64 bytes of a row: four lanes with a float4 each, or
// sixteen with a float where rows do not start on 16-byte boundaries) and marches along y.  When line k of C arrives it
// completes the rows of T of line k - 1 and the rows of D of line k - 2 and starts those of the lines k and k - 1; what
// they need of the lines before is in the lane's registers, what they need of the neighbours along x is in the lane's own
// points or comes by shuffle.  The two outermost points on each side are read and computed for their neighbours only
// (28 of 32 points are completed: 14 % more reads, which L2 or L1 serves), so warps never wait for each other and there is
// no shared memory and no barrier.  Loads run two lines ahead.
// Products are added in column order (y-, x-, centre, x+, y+) with fused multiply-adds from zero, so results are bit for
// bit those of the CSR executors.  Rows of T that do not exist are set to zero and not multiplied by it, so an infinity
// in C stays where it belongs.
// What bounds it is memory: every element of C is read once and every element of D written once.  1023 x 777, 64 columns:
// 94.9 us (4.3 TB/s of those bytes; 96.5 before L2 was asked for lines ahead); the tile pipeline, which writes T and reads it back, took 183.
#include <algorithm>

#include "line_march.h"
#include "segments.h"

namespace tfk {

namespace {

constexpr unsigned kAll = 0xffffffffu;
// Lines between the line that a warp asks L2 for and the one that it completes, and the shortest segment that does so.  Two
// lines in registers do not cover a read from memory; asking L2 for a line six ahead does, without a register.  Measured (no
// request; 4, 6, 8, 12 lines): 1400 x 1400, 96 columns 342 us; 308, 308, 313, 352; 1000 x 1000, 100 columns 197; 190, 186, 188,
// 199; 1023 x 777, 64 columns 100.4; 98.3, 99.1, 102, 106.  Short segments have no line left to ask for: the requests cost
// 500 x 300, 32 columns (seven lines) 19.5 -> 21.5.  With single columns a line of a warp is sixteen instructions of two
// points each, and asking for it too costs more than it hides: 900 x 700, 33 columns 117 -> 164, with a lane per point 124.
constexpr int kLineAhead = 6, kLineAheadSegment = 24;
constexpr int line_ctas(bool vec) { return vec ? 3 : 2; }  // resident per SM (with single columns a lane holds four times the points)

template <int V>
struct Cols {
  float v[V];
};
template <int V>
__device__ __forceinline__ Cols<V> zero_cols() {
  Cols<V> r;
#pragma unroll
  for (int i = 0; i < V; ++i) r.v[i] = 0.f;
  return r;
}
template <int V>
__device__ __forceinline__ Cols<V> fma_cols(float a, const Cols<V> &x, const Cols<V> &c) {
  Cols<V> r;
#pragma unroll
  for (int i = 0; i < V; ++i) r.v[i] = fmaf(a, x.v[i], c.v[i]);
  return r;
}
template <int V>
__device__ __forceinline__ Cols<V> read_cols(const float *p) {
  Cols<V> r;
  if (V == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
    r.v[0] = t.x; r.v[1 % V] = t.y; r.v[2 % V] = t.z; r.v[3 % V] = t.w;
  } else {
    r.v[0] = __ldg(p);
  }
  return r;
}
template <int V>
__device__ __forceinline__ void write_cols(float *p, const Cols<V> &x) {
  if (V == 4) *reinterpret_cast<float4 *>(p) = make_float4(x.v[0], x.v[1 % V], x.v[2 % V], x.v[3 % V]);
  else p[0] = x.v[0];
}
template <int V>
__device__ __forceinline__ Cols<V> from_lane_below(const Cols<V> &x, int d) {
  Cols<V> r;
#pragma unroll
  for (int i = 0; i < V; ++i) r.v[i] = __shfl_up_sync(kAll, x.v[i], d);
  return r;
}
template <int V>
__device__ __forceinline__ Cols<V> from_lane_above(const Cols<V> &x, int d) {
  Cols<V> r;
#pragma unroll
  for (int i = 0; i < V; ++i) r.v[i] = __shfl_down_sync(kAll, x.v[i], d);
  return r;
}

// V: columns per lane; a group of 16 / V lanes holds P points of the line.
template <int V>
struct LineShape {
  static constexpr int L = 16 / V, G = 32 / L, P = tf::kLineSpan / G, W = P / 4;  // W: class words per thread
};

template <int V, bool SAME>
__global__ void __launch_bounds__(32 * kLineWarps, line_ctas(V == 4)) line_march_kernel(const __grid_constant__ LineParams A) {
  using S = LineShape<V>;
  constexpr int L = S::L, P = S::P, W = S::W;
  const int lane = threadIdx.x & 31;
  const int item = blockIdx.x * kLineWarps + (threadIdx.x >> 5);
  if (item >= A.n_items) return;
  const int chunk = item % A.chunks, rest = item / A.chunks, tile = rest % A.tiles, seg = rest / A.tiles;
  const int ys = A.y_begin + seg * A.seg_len, ye = min(A.y_end, ys + A.seg_len);
  const int g = lane / L, col = chunk * 16 + (lane % L) * V;
  const int x0 = tile * tf::kLineOut - 2 + g * P;  // first point of this lane
  const bool col_in = col < A.n_cols;
  unsigned in = 0, own = 0;  // points that exist; points whose rows of D are this lane's to write
#pragma unroll
  for (int p = 0; p < P; ++p) {
    if (col_in && x0 + p >= 0 && x0 + p < A.nx) {
      in |= 1u << p;
      const int i = g * P + p;
      if (i >= 2 && i < 2 + tf::kLineOut) own |= 1u << p;
    }
  }
  const size_t line = (size_t)A.nx * A.n_cols;
  const long long at0 = (long long)x0 * A.n_cols + col;
  const float *src = A.in + at0;
  float *dst = A.out + at0;
  const int word_line = A.tiles * 8;
  const unsigned *wf_at = A.words_f + tile * 8 + g * W, *wa_at = A.words_a + tile * 8 + g * W;

  typedef Cols<V> Vec;
  auto load_line = [&](int k, Vec (&x)[P]) {
    const bool exists = k >= 0 && k < A.ny;
    const float *p = src + (long long)k * (long long)line;
#pragma unroll
    for (int i = 0; i < P; ++i) x[i] = exists && (in >> i & 1u) ? read_cols<V>(p + (size_t)i * A.n_cols) : zero_cols<V>();
  };
  auto load_words = [&](const unsigned *at, unsigned none, int k, unsigned (&w)[W]) {
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = k >= 0 && k < A.ny ? __ldg(at + (size_t)k * word_line + i) : none;
  };

  // ring: the lines k - 1 .. k + 2 of C, and the class words of the same lines
  Vec c[4][P], accT[P], accD[P], t1[P];
  unsigned wf[4][W], wa[4][W];  // (wa is used where the operators differ)
  unsigned wap[W];              // words of the second operator's line k - 2
#pragma unroll
  for (int i = 0; i < P; ++i) { c[3][i] = accT[i] = accD[i] = t1[i] = zero_cols<V>(); }
#pragma unroll
  for (int i = 0; i < W; ++i) { wf[3][i] = A.none_f; wap[i] = A.none_a; wa[3][i] = A.none_a; }
  const int k0 = ys - 2, k1 = ye + 1;  // lines of C that the segment reads
  const bool ahead = A.seg_len >= kLineAheadSegment;
  load_line(k0, c[0]);
  load_line(k0 + 1, c[1]);
  load_words(wf_at, A.none_f, k0, wf[0]);
  load_words(wf_at, A.none_f, k0 + 1, wf[1]);
  if (!SAME) {
    load_words(wa_at, A.none_a, k0, wa[0]);
    load_words(wa_at, A.none_a, k0 + 1, wa[1]);
  }

  // interior coefficients
  const float4 fl = A.dict_f[0], al = A.dict_a[0];
  const float fh = A.dict_f[1].x, ah = A.dict_a[1].x;

  for (int kb = k0; kb <= k1; kb += 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = kb + j;
      if (k > k1) break;
      Vec (&cm)[P] = c[(j + 3) & 3];
      Vec (&cc)[P] = c[j];
      unsigned (&wfm)[W] = wf[(j + 3) & 3];
      unsigned (&wfc)[W] = wf[j];
      unsigned (&wac)[W] = SAME ? wf[(j + 3) & 3] : wa[(j + 3) & 3];  // second operator, line k - 1
      load_line(k + 2 <= k1 ? k + 2 : -1, c[(j + 2) & 3]);
      if (V == 4 && ahead && k + kLineAhead <= k1 && k + kLineAhead < A.ny) {  // (k >= -2, so the line exists)
        const float *q = src + (long long)(k + kLineAhead) * (long long)line;
#pragma unroll
        for (int i = 0; i < P; ++i)
          if (in >> i & 1u) asm volatile("prefetch.global.L2 [%0];" ::"l"(q + (size_t)i * A.n_cols));
      }
      load_words(wf_at, A.none_f, k + 2, wf[(j + 2) & 3]);
      if (!SAME) load_words(wa_at, A.none_a, k + 2, wa[(j + 2) & 3]);
      unsigned any = 0;
#pragma unroll
      for (int i = 0; i < W; ++i) any |= wfm[i] | wfc[i] | wac[i] | wap[i];
      const bool plain = __all_sync(kAll, any == 0);
      const Vec cl = from_lane_below(cc[P - 1], L), cr = from_lane_above(cc[0], L);
      Vec t[P];
      if (plain) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          t[p] = fma_cols(fh, cc[p], accT[p]);
          Vec s = fma_cols(fl.x, cm[p], zero_cols<V>());
          s = fma_cols(fl.y, p ? cc[p ? p - 1 : 0] : cl, s);
          s = fma_cols(fl.z, cc[p], s);
          accT[p] = fma_cols(fl.w, p < P - 1 ? cc[p < P - 1 ? p + 1 : p] : cr, s);
        }
      } else {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const unsigned km = wfm[p / 4] >> (8 * (p & 3)) & 255u, kc = wfc[p / 4] >> (8 * (p & 3)) & 255u;
          t[p] = fma_cols(A.dict_f[2 * km + 1].x, cc[p], accT[p]);
          if (km == (A.none_f & 255u)) t[p] = zero_cols<V>();
          const float4 f = A.dict_f[2 * kc];
          Vec s = fma_cols(f.x, cm[p], zero_cols<V>());
          s = fma_cols(f.y, p ? cc[p ? p - 1 : 0] : cl, s);
          s = fma_cols(f.z, cc[p], s);
          accT[p] = fma_cols(f.w, p < P - 1 ? cc[p < P - 1 ? p + 1 : p] : cr, s);
        }
      }
      const Vec tl = from_lane_below(t[P - 1], L), tr = from_lane_above(t[0], L);
      const bool store = k - 2 >= ys && k - 2 < ye;
      float *o = dst + (long long)(k - 2) * (long long)line;
      if (plain) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const Vec d = fma_cols(ah, t[p], accD[p]);
          if (store && (own >> p & 1u)) write_cols<V>(o + (size_t)p * A.n_cols, d);
          Vec s = fma_cols(al.x, t1[p], zero_cols<V>());
          s = fma_cols(al.y, p ? t[p ? p - 1 : 0] : tl, s);
          s = fma_cols(al.z, t[p], s);
          accD[p] = fma_cols(al.w, p < P - 1 ? t[p < P - 1 ? p + 1 : p] : tr, s);
        }
      } else {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const unsigned km = wap[p / 4] >> (8 * (p & 3)) & 255u, kc = wac[p / 4] >> (8 * (p & 3)) & 255u;
          const Vec d = fma_cols(A.dict_a[2 * km + 1].x, t[p], accD[p]);
          if (store && (own >> p & 1u)) write_cols<V>(o + (size_t)p * A.n_cols, d);
          const float4 f = A.dict_a[2 * kc];
          Vec s = fma_cols(f.x, t1[p], zero_cols<V>());
          s = fma_cols(f.y, p ? t[p ? p - 1 : 0] : tl, s);
          s = fma_cols(f.z, t[p], s);
          accD[p] = fma_cols(f.w, p < P - 1 ? t[p < P - 1 ? p + 1 : p] : tr, s);
        }
      }
#pragma unroll
      for (int p = 0; p < P; ++p) t1[p] = t[p];
#pragma unroll
      for (int i = 0; i < W; ++i) wap[i] = wac[i];
    }
  }
}

typedef void (*LineFn)(const LineParams);

}  // namespace

cudaError_t launch_line_march(LineParams &p, bool vec, bool same, int sm_count, cudaStream_t s) {
  const int lines = p.y_end - p.y_begin;
  if (lines <= 0) return cudaSuccess;
  LineFn f = vec ? (same ? (LineFn)line_march_kernel<4, true> : (LineFn)line_march_kernel<4, false>)
                 : (same ? (LineFn)line_march_kernel<1, true> : (LineFn)line_march_kernel<1, false>);
  p.chunks = (p.n_cols + 15) / 16;
  // a segment of n lines costs n + 4 steps, which on a small grid is what the launch takes, so segments may be one line long
  // (40 x 33, 64 columns: 7.7 us with four lines at least, 6.0 with two, 5.5 with one; 100 x 100, 16 columns: 7.5, 5.9 and 5.4)
  const long long columns = (long long)p.tiles * p.chunks, resident = (long long)sm_count * line_ctas(vec) * kLineWarps;
  p.seg_len = tf::segment_length(lines, columns, resident, 4, 1);
  const long long items = columns * ((lines + p.seg_len - 1) / p.seg_len);
  if (items > 0x7fffffff) return cudaErrorInvalidValue;
  p.n_items = (int)items;
  f<<<(p.n_items + kLineWarps - 1) / kLineWarps, 32 * kLineWarps, 0, s>>>(p);
  return cudaGetLastError();
}

}  // namespace tfk
