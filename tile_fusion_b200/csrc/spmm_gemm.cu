// GeMM-SpMM in one launch, D = act((A B) W), for star stencils on a grid: the sparse product is the producer of the tensor
// cores' operand, and no intermediate goes to memory.
//
// A CTA takes bricks of 128 grid points, a pair of CTAs one tile of 256 rows (cta_group::2, as in row_gemm.cu).  Per slice of
// 32 columns one TMA box brings the brick's points of B and their neighbours (on a 3-D grid two more boxes the layers below and
// above, without corners) into a ring; eight warps add up the rows of A B there, four points in a row along x to a group of
// eight lanes, so that a line is read once for three products, split them for the tensor core and leave them in the swizzled
// tile; one warp issues the products; four warps drain the accumulators, turn 32 x 32 blocks round in shared memory and write
// whole 128-byte segments of D's rows.  The weight stays in shared memory where half of it (hi and lo) takes up to 64 KB, split
// by the CTA itself; wider ones come from L2 slice by slice, split by a launch in front.
// lo * hi and hi * lo have an accumulator of their own where there is room (up to 128 columns), hi * hi one or, in turn, three:
// the tensor core cuts off what it adds, so the fewer sums on large values the better (rel. error at K = 256: 64 columns
// 2.4e-7, 4.6e-7 with the steps of row_gemm.cu in turn on four; 128 columns 6.3e-7, 8.8e-7 before; 256 columns 1.7e-6, 1.9e-6).
// What bounds it on 3-D grids is shared memory (per slice, K = N = 256: 768 cycles of the tensor core's reads, 960 of the
// sparse product's, 560 of the copies', of 2 400), on flat grids memory and the latency of a round of bricks.
// Against the dense product and the march or gather of their own launches, us: 65 536 points flat, 64 -> 64: 12.6 and 27;
// 700 000 flat, 32 -> 256: 156 and 513, 128 -> 128: 155 and 303, 256 -> 64: 226 and 280; 1 M in 3-D, 64 -> 64: 142 and 193,
// 256 -> 256: 646 and 910; 561 661 in 3-D, 100 -> 64: 157 and 154, 256 -> 16: 265 and 161 (see one_launch_depth).
// (Tried: rows gathered by nonzeros into registers, two CTAs of eight warps in turns of everything: 440 us instead of 233 at
// 700 000 points, 256 -> 64; rows listed and copied by a warp's cp.async: 619; four warps to a slice with 4 x 2 points to a group: 235, on
// 3-D grids 178 instead of 160.)
// All waits are bounded: the one that runs out sets the error flag, and every role leaves.
#include "spmm_gemm.h"

#include <algorithm>
#include <cstring>
#include <string>

#include "gemm_tc_host.h"
#include "pair_mma.cuh"
#include "row_gemm.h"
#include "tf_internal.h"

namespace tfk {

namespace {

constexpr int kSgRows = tf::kStarRows;
constexpr int kSgEpiWarps = 4, kSgWorkWarps = 8;
constexpr int kSgWarpW = kSgEpiWarps + kSgWorkWarps, kSgWarpMma = kSgWarpW + 1, kSgWarpRaw = kSgWarpW + 2;
constexpr int kSgThreads = 32 * (kSgWarpRaw + 1);
static_assert(kSgThreads == kSpmmGemmThreads, "what a plan says of itself");
constexpr int kSgMaxStages = 4, kSgMaxRaws = 6;
constexpr int kSgStageA = 2 * kSgRows * 128;  // hi and lo of a slice of 32 columns
constexpr int kSgEpiBytes = kSgEpiWarps * 4096;
constexpr int kSgSmemMax = 226 * 1024;
static_assert(kSgRows == kTcRows, "a brick is half as high as the product of a pair");

struct SgShared {
  unsigned long long raw_full[kSgMaxRaws], raw_empty[kSgMaxRaws];  // points of B, this CTA's
  unsigned long long wfull[kSgMaxStages], ready[kSgMaxStages], empty[kSgMaxStages];
  unsigned long long acc_full[2], acc_empty[2], drained;
  unsigned tmem_base;
  int dead;
};

__device__ __forceinline__ void arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// A box of grid points: coordinates (column, x, y, z), zeros outside the grid.
__device__ __forceinline__ void load_points(void *smem, const CUtensorMap *tm, int col, int x, int y, int z, unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem)), "l"((unsigned long long)tm), "r"(smem_u32(bar)), "r"(col), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ float4 lds4(const char *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void fma4(float4 &a, float v, const float4 &x) {
  a.x = fmaf(v, x.x, a.x); a.y = fmaf(v, x.y, a.y); a.z = fmaf(v, x.z, a.z); a.w = fmaf(v, x.w, a.w);
}
// First point of a brick.
__device__ __forceinline__ void brick_origin(const tf::BrickGrid &g, int brick, int &x, int &y, int &z) {
  const int nbx = (g.nx + (1 << g.lx) - 1) >> g.lx, nby = (g.ny + (1 << g.ly) - 1) >> g.ly;
  const int layer = brick / (nbx * nby), r = brick - layer * nbx * nby, row = r / nbx;
  x = (r - row * nbx) << g.lx;
  y = row << g.ly;
  z = layer << g.lz;
}

// D3: seven points, else five.  RES: the weight lies in shared memory, else its slices come with the stages.
template <bool D3, bool RES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kSgThreads, 1)
spmm_gemm_kernel(const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_cap, const __grid_constant__ CUtensorMap tm_whi,
                 const __grid_constant__ CUtensorMap tm_wlo, const __grid_constant__ SpmmGemmParams A) {
  extern __shared__ char dyn[];
  __shared__ SgShared s;
  char *smem = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = __shfl_sync(kFull, tid >> 5, 0), lane = tid & 31;  // (known to be uniform)
  const unsigned rank = pair_rank();
  const int N = A.n_pad, half = N / 2, slice_w = half * 256;  // bytes of this CTA's half of a slice of the split weight
  const int stage_bytes = kSgStageA + (RES ? 0 : slice_w), raw_bytes = A.raw_bytes;
  char *wbuf = smem + A.stages * stage_bytes;
  char *raw = wbuf + (RES ? A.slices * slice_w : 0);
  char *epi = raw + A.raws * raw_bytes;
  const int pairs = gridDim.x >> 1, first = blockIdx.x >> 1, tiles = (A.brick_end - A.brick_begin + 1) >> 1;  // pairs of bricks
  const int brick0 = A.brick_begin + (int)rank;  // of pair t of bricks this CTA has number brick0 + 2 t
  const int acc_cols = 256 / A.accs;
  const int g = lane >> 3, c = lane & 7;
  const int sx = 1 << A.grid.lx, sy = 1 << A.grid.ly, sz = 1 << A.grid.lz;

  if (tid == 0) {
    for (int i = 0; i < A.raws; ++i) { mbar_init(&s.raw_full[i], 1); mbar_init(&s.raw_empty[i], kSgWorkWarps); }
    for (int i = 0; i < A.stages; ++i) { mbar_init(&s.wfull[i], 1); mbar_init(&s.ready[i], 2 * kSgWorkWarps); mbar_init(&s.empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s.acc_full[i], 1); mbar_init(&s.acc_empty[i], 2 * kSgEpiWarps); }
    mbar_init(&s.drained, 1);
    s.dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (RES) {  // this CTA's columns of the weight, K rounded up to slices
    const int quads = A.slices * 8;
    for (int i = tid; i < quads * half; i += kSgThreads) {
      const int q = A.w_k == 1 ? i % quads : i / half, r = A.w_k == 1 ? i / quads : i - q * half, k = q * 4, col = (int)rank * half + r;
      const float *w = A.w + (size_t)k * A.w_k + (size_t)col * A.w_c;
      const bool in = col < A.n;
      const float4 x = make_float4(in && k < A.k ? __ldg(w) : 0.f, in && k + 1 < A.k ? __ldg(w + A.w_k) : 0.f,
                                   in && k + 2 < A.k ? __ldg(w + 2 * A.w_k) : 0.f, in && k + 3 < A.k ? __ldg(w + 3 * A.w_k) : 0.f);
      const float4 h = make_float4(tf32_round(x.x), tf32_round(x.y), tf32_round(x.z), tf32_round(x.w));
      char *o = wbuf + (q >> 3) * slice_w + r * 128 + (((q & 7) ^ (r & 7)) << 4);
      *reinterpret_cast<float4 *>(o) = h;
      *reinterpret_cast<float4 *>(o + half * 128) =
          make_float4(tf32_round(x.x - h.x), tf32_round(x.y - h.y), tf32_round(x.z - h.z), tf32_round(x.w - h.w));
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  pair_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  if (warp == kSgWarpRaw) {
    // ---- the points of B that a brick reads, a slice at a time (the whole warp, see elect_one) ----
    int rs = 0, used = 0;
    unsigned rph = 0;
    bool ok = true;
    for (int t = first; t < tiles && ok; t += pairs) {
      int x, y, z;
      brick_origin(A.grid, brick0 + 2 * t, x, y, z);
      for (int sl = 0; sl < A.slices; ++sl) {
        if (used >= A.raws && !(ok = __all_sync(kFull, pair_wait(&s.raw_empty[rs], rph ^ 1u, s.dead, A.wait_limit)))) break;
        char *o = raw + rs * raw_bytes;
        if (elect_one()) {
          mbar_expect_tx(&s.raw_full[rs], (unsigned)raw_bytes);
          load_points(o, &tm_b, sl * kTcKSlice, x - 1, y - 1, z, &s.raw_full[rs]);
          if (D3) {  // the layers below and above, without their neighbours
            load_points(o + raw_bytes - 2 * sx * sy * 128, &tm_cap, sl * kTcKSlice, x, y, z - 1, &s.raw_full[rs]);
            load_points(o + raw_bytes - sx * sy * 128, &tm_cap, sl * kTcKSlice, x, y, z + sz, &s.raw_full[rs]);
          }
        }
        __syncwarp();
        if (used < A.raws) ++used;
        if (++rs == A.raws) { rs = 0; rph ^= 1u; }
      }
    }
    // (a copy still in flight must not outlive the CTA: only after a wait ran out is one possible)
    if (!ok || s.dead)
      for (int i = 0; i < used; ++i) mbar_wait(&s.raw_full[i], i < rs ? rph : rph ^ 1u, A.wait_limit);
  } else if (warp == kSgWarpW) {
    // ---- slices of the weight (where they come with the stages) ----
    int st = 0, issued = 0;
    unsigned ph = 0;
    bool ok = true;
    auto wait = [&](unsigned long long *bar, unsigned parity) {
      return ok = __all_sync(kFull, pair_wait(bar, parity, s.dead, A.wait_limit));
    };
    for (int t = RES ? tiles : first; t < tiles && ok; t += pairs)
      for (int sl = 0; sl < A.slices; ++sl) {
        if (issued >= A.stages && !wait(&s.empty[st], ph ^ 1u)) break;
        if (elect_one()) {
          char *w = smem + st * stage_bytes + kSgStageA;
          mbar_expect_tx(&s.wfull[st], (unsigned)slice_w);
          tma_load_2d(w, &tm_whi, sl * kTcKSlice, (int)rank * half, &s.wfull[st]);
          tma_load_2d(w + half * 128, &tm_wlo, sl * kTcKSlice, (int)rank * half, &s.wfull[st]);
        }
        __syncwarp();
        if (issued < A.stages) ++issued;
        if (++st == A.stages) { st = 0; ph ^= 1u; }
      }
    if (!ok || s.dead)
      for (int i = 0; i < issued; ++i) mbar_wait(&s.wfull[i], i < st ? ph : ph ^ 1u, A.wait_limit);
  } else if (warp == kSgWarpMma) {
    // ---- products (even CTA): the whole warp, see elect_one ----
    if (rank == 0) {
      const unsigned idesc = pair_idesc(N);
      int st = 0, buf = 0, uses = 0;
      unsigned ph = 0, acc_ph = 0;
      bool ok = true;
      auto wait = [&](unsigned long long *bar, unsigned parity) {
        return ok = __all_sync(kFull, pair_wait<true>(bar, parity, s.dead, A.wait_limit));
      };
      const unsigned tmem = s.tmem_base;
      for (int t = first; t < tiles && ok; t += pairs) {
        if (uses >= 2 && !wait(&s.acc_empty[buf], acc_ph ^ 1u)) break;
        if (uses < 2) ++uses;
        const unsigned d = tmem + (unsigned)(buf * 256);
        // lo * hi and hi * lo go into the last accumulator, hi * hi in turn into the others; all into the one where there is one
        const unsigned small = d + (unsigned)(A.accs - 1) * acc_cols, wrap = A.accs > 1 ? small : d + acc_cols;
        unsigned big = d;
        for (int sl = 0; sl < A.slices; ++sl) {
          if (!wait(&s.ready[st], ph)) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned at = smem_u32(smem + st * stage_bytes), wat = RES ? smem_u32(wbuf + sl * slice_w) : at + kSgStageA;
          const unsigned long long ah = umma_desc_sw128(at), al = umma_desc_sw128(at + kSgRows * 128);
          const unsigned long long wh = umma_desc_sw128(wat), wl = umma_desc_sw128(wat + half * 128);
          const bool first_slice = sl == 0, last_slice = sl == A.slices - 1;
          unsigned to[kTcKSlice / 8], fresh[kTcKSlice / 8];
#pragma unroll
          for (int j = 0; j < kTcKSlice / 8; ++j) {
            to[j] = big;
            fresh[j] = A.accs > 1 && first_slice && (j == 0 || (j < A.accs - 1));
            big += acc_cols;
            if (big == wrap) big = d;
          }
          if (elect_one()) {
#pragma unroll
            for (int j = 0; j < kTcKSlice / 8; ++j) pair_mma(small, al + j * kUmmaStep, wh + j * kUmmaStep, idesc, first_slice && j == 0 ? 0u : 1u);
#pragma unroll
            for (int j = 0; j < kTcKSlice / 8; ++j) pair_mma(small, ah + j * kUmmaStep, wl + j * kUmmaStep, idesc, 1u);
#pragma unroll
            for (int j = 0; j < kTcKSlice / 8; ++j) pair_mma(to[j], ah + j * kUmmaStep, wh + j * kUmmaStep, idesc, fresh[j] ? 0u : 1u);
            pair_commit(&s.empty[st]);
            if (last_slice) pair_commit(&s.acc_full[buf]);
          }
          __syncwarp();
          if (last_slice) {
            buf ^= 1;
            if (buf == 0) acc_ph ^= 1u;
          }
          if (++st == A.stages) { st = 0; ph ^= 1u; }
        }
      }
      if (!ok) {  // products still running read shared memory of both CTAs
        if (elect_one()) pair_commit(&s.drained);
        mbar_wait(&s.drained, 0, A.wait_limit);
      }
    }
  } else if (warp >= kSgEpiWarps) {
    // ---- the sparse product: rows of A B, split for the tensor core ----
    // A group of eight lanes has four points in a row along x, r = 16 w + 4 g + i of the brick, a lane four columns of each.
    const int w = warp - kSgEpiWarps, r0 = w * 16 + 4 * g;
    const int x0 = r0 & (sx - 1), y0 = (r0 >> A.grid.lx) & (sy - 1), z0 = r0 >> (A.grid.lx + A.grid.ly);
    const int py = (sx + 2) * 128, pz = (sy + 2) * py;
    const int centre = ((z0 * (sy + 2) + y0 + 1) * (sx + 2) + x0 + 1) * 128 + c * 16;
    const int cap = raw_bytes + (y0 * sx + x0) * 128 + c * 16;
    const int below = z0 > 0 ? centre - pz : cap - 2 * sx * sy * 128, above = z0 < sz - 1 ? centre + pz : cap - sx * sy * 128;
    int at[4];  // the swizzled places of the four rows
#pragma unroll
    for (int i = 0; i < 4; ++i) at[i] = (r0 + i) * 128 + ((c ^ ((r0 + i) & 7)) << 4);
    float v[4][7];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int p = 0; p < 7; ++p) v[i][p] = A.uniform[p];
    int st = 0, rs = 0, n = 0;
    unsigned ph = 0, rph = 0;
    bool ok = true;
    for (int t = first; t < tiles && ok; t += pairs) {
      if (A.coef) {
        int x, y, z;
        brick_origin(A.grid, brick0 + 2 * t, x, y, z);
        x += x0; y += y0; z += z0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool in = x + i < A.grid.nx && y < A.grid.ny && z < A.grid.nz;
          const float4 *q = reinterpret_cast<const float4 *>(A.coef) + 2 * (((size_t)z * A.grid.ny + y) * A.grid.nx + x + i);
          const float4 lo = in ? __ldg(q) : make_float4(0.f, 0.f, 0.f, 0.f), hi = in ? __ldg(q + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
          v[i][0] = lo.x; v[i][1] = lo.y; v[i][2] = lo.z; v[i][3] = lo.w; v[i][4] = hi.x; v[i][5] = hi.y; v[i][6] = hi.z;
        }
      }
      for (int sl = 0; sl < A.slices; ++sl) {
        ok = pair_wait(&s.raw_full[rs], rph, s.dead, A.wait_limit);
        if (ok && n >= A.stages) ok = pair_wait(&s.empty[st], ph ^ 1u, s.dead, A.wait_limit);
        if (!(ok = __all_sync(kFull, ok))) break;
        if (n < A.stages) ++n;
        const char *x = raw + rs * raw_bytes;
        char *stage = smem + st * stage_bytes;
        float4 line[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) line[i] = lds4(x + centre + (i - 1) * 128);
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // in column order
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
          if (D3) fma4(a, v[i][0], lds4(x + below + i * 128));
          fma4(a, v[i][1], lds4(x + centre - py + i * 128));
          fma4(a, v[i][2], line[i]);
          fma4(a, v[i][3], line[i + 1]);
          fma4(a, v[i][4], line[i + 2]);
          fma4(a, v[i][5], lds4(x + centre + py + i * 128));
          if (D3) fma4(a, v[i][6], lds4(x + above + i * 128));
          float4 hi, lo;
          split_pair(a.x, kRoundLow, hi.x, lo.x); split_pair(a.y, kRoundLow, hi.y, lo.y);
          split_pair(a.z, kRoundLow, hi.z, lo.z); split_pair(a.w, kRoundLow, hi.w, lo.w);
          *reinterpret_cast<float4 *>(stage + at[i]) = hi;
          *reinterpret_cast<float4 *>(stage + at[i] + kSgRows * 128) = lo;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // read next by the tensor core
        if (!RES && w == 0 && !(ok = __all_sync(kFull, pair_wait(&s.wfull[st], ph, s.dead, A.wait_limit)))) break;
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          arrive(&s.raw_empty[rs]);
          pair_arrive_leader(&s.ready[st]);
        }
        if (++st == A.stages) { st = 0; ph ^= 1u; }
        if (++rs == A.raws) { rs = 0; rph ^= 1u; }
      }
    }
    // The tensor core's arrivals on the stages of this CTA come from the other one too: the last of them must be in before the CTA
    // may end.  (For this a warp that waits for every phase as it comes: one that has nothing to do in between can be a phase of the
    // same parity late, and then waits for one that never comes.)
    for (int i = 0; w == 0 && ok && i < n; ++i) ok = __all_sync(kFull, pair_wait(&s.empty[i], i < st ? ph : ph ^ 1u, s.dead, A.wait_limit));
  } else {
    // ---- rows of D: warp w drains the rows 32 w .. 32 w + 31 of the CTA's tile ----
    int buf = 0;
    unsigned acc_ph = 0;
    bool ok = true;
    const unsigned lanes = s.tmem_base + ((unsigned)(warp * 32) << 16);
    float4 *blk = reinterpret_cast<float4 *>(epi + warp * 4096);
    for (int t = first; t < tiles; t += pairs) {
      int rows[8], x, y, z;  // of D, -1: none
      brick_origin(A.grid, brick0 + 2 * t, x, y, z);
      const bool brick = brick0 + 2 * t < A.brick_end;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = warp * 32 + 4 * i + g, px = x + (r & (sx - 1)), py = y + ((r >> A.grid.lx) & (sy - 1)), pz = z + (r >> (A.grid.lx + A.grid.ly));
        rows[i] = brick && px < A.grid.nx && py < A.grid.ny && pz < A.grid.nz ? (pz * A.grid.ny + py) * A.grid.nx + px : -1;
      }
      if (!(ok = __all_sync(kFull, pair_wait(&s.acc_full[buf], acc_ph, s.dead, A.wait_limit)))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int c0 = 0; c0 < N; c0 += 32) {
        float v[32];
        const unsigned from = lanes + (unsigned)(buf * 256 + c0);
        tmem_load32(v, from);
        if (A.accs == 2) {  // both on their way at once (700 000 points, 32 -> 128: 106 us one after the other, 99 like this)
          float a[32];
          tmem_load32(a, from + acc_cols);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          tmem_loaded(v);
          tmem_loaded(a);
#pragma unroll
          for (int q = 0; q < 32; ++q) v[q] += a[q];
        } else {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          tmem_loaded(v);
          if (A.accs > 2) {  // (two at a time: no faster, 2 % slower where the tensor core is busy)
#pragma unroll 1
            for (int i = 1; i < 4; ++i) {
              float a[32];
              tmem_load32(a, from + (unsigned)(i * acc_cols));
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              tmem_loaded(a);
#pragma unroll
              for (int q = 0; q < 32; ++q) v[q] += a[q];
            }
          }
        }
        if (c0 + 32 >= N) {  // the accumulator has been read: its next use may overwrite it
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) pair_arrive_leader(&s.acc_empty[buf]);
        }
        if (A.relu) {
#pragma unroll
          for (int q = 0; q < 32; ++q) v[q] = fmaxf(v[q], 0.f);
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q) blk[lane * 8 + (q ^ (lane & 7))] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = 4 * i + g;
          if (rows[i] >= 0 && c0 + 4 * c < A.n) *reinterpret_cast<float4 *>(A.out + (size_t)rows[i] * A.n + c0 + 4 * c) = blk[r * 8 + (c ^ (r & 7))];
        }
      }
      buf ^= 1;
      if (buf == 0) acc_ph ^= 1u;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && s.dead) atomicExch(A.error, 1);
  pair_sync();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(s.tmem_base), "n"(512) : "memory");
  }
}

int resident_bytes(int K, int n) { return (K + kTcKSlice - 1) / kTcKSlice * row_gemm_pad_n(n) * 128; }
size_t fixed_bytes(int K, int n) { return 1024 + kSgEpiBytes + (spmm_gemm_resident(K, n) ? resident_bytes(K, n) : 0); }
size_t stage_size(int K, int n) { return kSgStageA + (spmm_gemm_resident(K, n) ? 0 : row_gemm_pad_n(n) * 128); }
// Stages and slices of B's points that fit the shared memory: as many of the latter as of the former, or one more.
bool fit(int K, int n, const tf::BrickGrid &g, int &stages, int &raws, size_t &smem) {
  const size_t stage = stage_size(K, n), raw = (size_t)tf::brick_points(g) * 128, fixed = fixed_bytes(K, n);
  stages = raws = 0;
  for (;;) {
    const bool more_raw = raws <= stages && raws < kSgMaxRaws;
    if (!more_raw && stages >= kSgMaxStages) break;
    if (fixed + (stages + !more_raw) * stage + (raws + more_raw) * raw > kSgSmemMax) break;
    more_raw ? ++raws : ++stages;
  }
  while (raws < kSgMaxRaws && fixed + stages * stage + (raws + 1) * raw <= kSgSmemMax) ++raws;
  smem = fixed + stages * stage + raws * raw;
  return stages >= 2 && raws >= 2;
}

// B as (column, x, y, z), boxes of 32 columns x bx x by x bz points.
int points_map(CUtensorMap *out, const float *b, int K, const tf::BrickGrid &g, int bx, int by, int bz) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return tf::fail(TF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t row = (cuuint64_t)K * 4;
  cuuint64_t gdim[4] = {(cuuint64_t)K, (cuuint64_t)g.nx, (cuuint64_t)g.ny, (cuuint64_t)g.nz};
  cuuint64_t gstride[3] = {row, row * g.nx, row * g.nx * g.ny};
  cuuint32_t box[4] = {(cuuint32_t)kTcKSlice, (cuuint32_t)bx, (cuuint32_t)by, (cuuint32_t)bz};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(b), gdim, gstride, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? TF_OK : tf::fail(TF_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
}

}  // namespace

bool spmm_gemm_resident(int K, int n) { return resident_bytes(K, n) <= 64 * 1024; }
int spmm_gemm_points(int K, int n) { return (int)((kSgSmemMax - fixed_bytes(K, n) - 2 * stage_size(K, n)) / 2 / 128); }  // (twice, as the stages)

int spmm_gemm(SpmmGemmParams p, const float *hi, const float *lo, int sm_count, cudaStream_t s) {
  const bool res = spmm_gemm_resident(p.k, p.n), deep = p.grid.nz > 1;
  const int n = (p.brick_end - p.brick_begin + 1) / 2;
  if (n <= 0) return TF_OK;
  size_t smem = 0;
  if (!fit(p.k, p.n, p.grid, p.stages, p.raws, smem)) return tf::fail(TF_ERR_UNSUPPORTED, "spmm_gemm: too wide");
  p.raw_bytes = tf::brick_points(p.grid) * 128;
  p.n_pad = row_gemm_pad_n(p.n);
  p.w_k = p.w_transposed ? 1 : p.n;
  p.w_c = p.w_transposed ? p.k : 1;
  p.slices = (p.k + kTcKSlice - 1) / kTcKSlice;
  p.accs = p.n_pad > 128 ? 1 : (p.n_pad > 64 ? 2 : 4);
  const int x = 1 << p.grid.lx, y = 1 << p.grid.ly, z = 1 << p.grid.lz, ldk = row_gemm_pad_k(p.k);
  CUtensorMap mb, mc, mh, ml;
  int rc = points_map(&mb, p.b, p.k, p.grid, x + 2, y + 2, z);
  mc = mh = ml = mb;  // (not used by the variants that have no map of their own)
  if (rc == TF_OK && deep) rc = points_map(&mc, p.b, p.k, p.grid, x, y, 1);
  if (rc == TF_OK && !res) rc = tc_make_map(&mh, hi, p.n_pad, ldk, p.n_pad / 2, ldk);
  if (rc == TF_OK && !res) rc = tc_make_map(&ml, lo, p.n_pad, ldk, p.n_pad / 2, ldk);
  if (rc != TF_OK) return rc;
  auto f = deep ? (res ? spmm_gemm_kernel<true, true> : spmm_gemm_kernel<true, false>)
                : (res ? spmm_gemm_kernel<false, true> : spmm_gemm_kernel<false, false>);
  // (the limit is the kernel's, not the call's, see row_gemm.cu)
  cudaError_t e = cudaFuncSetAttribute((const void *)f, cudaFuncAttributeMaxDynamicSharedMemorySize, kSgSmemMax);
  if (e == cudaSuccess) {
    f<<<2 * std::max(1, std::min(n, sm_count / 2)), kSgThreads, smem, s>>>(mb, mc, mh, ml, p);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return tf::fail(TF_ERR_CUDA, std::string("spmm_gemm: ") + cudaGetErrorString(e));
  return TF_OK;
}

}  // namespace tfk
