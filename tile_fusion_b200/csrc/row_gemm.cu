// T = B * W (optionally max(0, .)) for a tall fp32 B on the 5th-generation tensor cores, 3xTF32 inside.
//
// The arithmetic is that of gemm_tc.cuh, product by product: every operand is split as x = hi + lo, both rounded to TF32
// (lo only where that tile's bits are not asked for; 1 to 3 % of the error), and hi*hi + hi*lo + lo*hi is accumulated in
// fp32 in tensor memory.  What differs is that nothing waits for anything it does not need:
//   * Two CTAs on neighbouring SMs work on one tile of 256 rows with tcgen05.mma.cta_group::2.  Each holds 128 rows of B
//     and half of the columns of W, so W crosses from L2 once per 256 rows, and the tensor core reads half of it from
//     each SM's shared memory.  (One CTA with 128 rows and all of W would need 180 bytes per clock of shared memory at
//     N = 256, 40 % more than there are.)
//   * A warp keeps the TMA loads of K slices of 32 columns running ahead through a ring of stages, eight warps split
//     the raw rows, one warp of the even CTA issues the products (see elect_one: by a thread alone 2 % slower at K = N = 256,
//     262 144 rows, K = N = 128: 65.0 us and 54.1; 500 009 rows, 256 -> 47: 243 and 198), four warps drain the accumulator of
//     the tile before (two accumulators of up to 256 columns in tensor memory) and write it with TMA stores.  (Splitting warps
//     in two teams with a slice each: no faster, and wrong where the stages are odd in number -- a team that visits a stage
//     every other time cannot tell the phase before the last from the last.)
//   * The grid is one pair per two SMs and walks the tiles.
// The tensor core cuts off what it adds to an accumulator instead of rounding it, so a chain of K / 8 sums drifts (rel.
// error 2e-6 at K = 256, ten times that of fp32 FMAs).  Widths and depths that the ticket executor's tensor-core tile does
// not take have always been multiplied with fp32 FMAs; for them the kernel has a second form that is as exact as those from
// 32 terms on: panels of up to 64 columns, whose four accumulators are read back and added in registers after every slice, by eight
// warps (500 009 rows, 256 -> 47: 193 us with four, 178 with eight, 155 with the split of rg_split, 3.9 TB/s of B and D).
// Fewer terms are multiplied with FMAs still, by row_fma_kernel.
// The plain form keeps its chains short where tensor memory has room: up to 128 columns the K steps of a slice go round two
// accumulators, up to 64 round four, the small products first (K = 256: rel. error 1.9e-6 with one, 8.8e-7 with two, 4.6e-7
// with four).
// All waits are bounded: the one that runs out sets the error flag, and every role leaves.
#include "row_gemm.h"

#include <algorithm>
#include <string>

#include "gemm_tc_host.h"
#include "pair_mma.cuh"
#include "tf_internal.h"

namespace tfk {

namespace {

__host__ __device__ constexpr int rg_epi_warps(bool precise) { return precise ? 8 : 4; }
constexpr int kRgSplitWarps = 8;
__host__ __device__ constexpr int rg_threads(bool precise) { return 32 * (rg_epi_warps(precise) + kRgSplitWarps + 2); }
constexpr int kRgMaxStages = 5;
// Slices of B that are on their way to L2 in front of the loads, where a tile has many or the product is narrow and leaves the
// loads to bound it (2.1 M rows, K = N = 256: 1 085 us without, 1 044 with 3, 8 and 20 are slower than 3; 262 144 rows, 128 -> 128:
// 52.8 and 48.5, 64 -> 64: 29.2 and 27.7, with 6 50.5 and 29.9; but 500 009 rows, 100 -> 256: 159 and 166).
constexpr int kRgAhead = 3, kRgAheadSlices = 8, kRgAheadWidth = 128;
// Terms from which on the precise form's error is no larger than that of fp32 FMAs (40 000 rows, rel.: 9.2e-8 and 1.03e-7 on
// uniform operands, 1.02e-7 and 1.03e-7 on normal ones, 6.1e-8 and 8.3e-8 on positive ones; 17 terms: 8.6e-8 and 7.6e-8);
// shapes of fewer that the tensor-core tile does not take are multiplied with those.
constexpr int kRgPreciseMinK = 32;
constexpr int kRgPrecisePanel = 64;  // columns: four accumulators, twice, in 512 columns of tensor memory
constexpr int kRgSmemMax = 227 * 1024;
constexpr int kRgEpiBytes = 8 * 32 * 128;  // 32 x 32 blocks: two per warp, one where eight warps drain

struct RgShared {
  unsigned long long raw[kRgMaxStages], ready[kRgMaxStages], empty[kRgMaxStages];
  unsigned long long acc_full[2], acc_empty[2], drained;
  unsigned tmem_base;
  int dead;
};

__host__ __device__ constexpr int rg_stage_bytes(int n) { return 2 * kTcRows * 128 + n * 128; }
constexpr int rg_stages(int n) {
  const int s = (kRgSmemMax - 2048 - kRgEpiBytes) / rg_stage_bytes(n);
  return s < kRgMaxStages ? s : kRgMaxStages;
}
static_assert(rg_stages(256) >= 2, "a full-width tile needs two stages");

// PRECISE: see above; n_pad <= 64.
// n_pad: columns of W rounded up to 32 (rows of the split weight beyond n_real are zero).
template <bool PRECISE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(rg_threads(PRECISE), 1)
row_gemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_whi,
                const __grid_constant__ CUtensorMap tm_wlo, const __grid_constant__ CUtensorMap tm_out, const RowGemmParams P) {
  constexpr int kRgEpiWarps = rg_epi_warps(PRECISE);
  extern __shared__ char dyn[];
  __shared__ RgShared s;
  char *smem = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = __shfl_sync(kFull, tid >> 5, 0), lane = tid & 31;  // (known to be uniform)
  const unsigned rank = pair_rank();
  const int N = P.n_pad, half = N / 2, stage_bytes = rg_stage_bytes(N), stages = P.stages;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int accs = PRECISE ? 4 : P.accs, acc_cols = PRECISE ? 64 : 256 / P.accs;  // accumulators of a tile, columns from one to the next
  char *epi = smem + stages * stage_bytes;

  if (tid == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&s.raw[i], 1);
      mbar_init(&s.ready[i], 2 * kRgSplitWarps);
      mbar_init(&s.empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s.acc_full[i], 1);
      mbar_init(&s.acc_empty[i], 2 * kRgEpiWarps);
    }
    mbar_init(&s.drained, 1);
    s.dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  pair_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  if (warp == kRgEpiWarps + kRgSplitWarps) {
    // ---- loads: the whole warp, see elect_one ----
    int st = 0, issued = 0;
    unsigned ph = 0;
    bool ok = true;
    auto wait = [&](unsigned long long *bar, unsigned parity) {
      return ok = __all_sync(kFull, pair_wait(bar, parity, s.dead, P.wait_limit));
    };
    int pt = pair, psl = 0;
    const bool ahead = !P.direct && (P.n_slices >= kRgAheadSlices || (P.n_slices > 1 && N <= kRgAheadWidth));
    auto prefetch = [&]() {
      if (!ahead || pt >= P.tiles) return;
      const int row = pt * 2 * kTcRows + (int)rank * kTcRows;
      if (row < P.m && elect_one())
        asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"((unsigned long long)&tm_a),
                     "r"(psl * kTcKSlice), "r"(row) : "memory");
      __syncwarp();
      if (++psl == P.n_slices) { psl = 0; pt += pairs; }
    };
    for (int i = 0; i < kRgAhead; ++i) prefetch();
    for (int t = pair; t < P.tiles && ok; t += pairs) {
      const int row = t * 2 * kTcRows + (int)rank * kTcRows;
      for (int sl = 0; sl < P.n_slices; ++sl) {
        prefetch();
        if (issued >= stages && !wait(&s.empty[st], ph ^ 1u)) break;
        char *b = smem + st * stage_bytes;
        if (elect_one()) {
          mbar_expect_tx(&s.raw[st], (unsigned)((P.direct ? 0 : kTcRows * 128) + N * 128));
          if (!P.direct) tma_load_2d(b, &tm_a, sl * kTcKSlice, row, &s.raw[st]);
          tma_load_2d(b + 2 * kTcRows * 128, &tm_whi, sl * kTcKSlice, (int)rank * half, &s.raw[st]);
          tma_load_2d(b + 2 * kTcRows * 128 + half * 128, &tm_wlo, sl * kTcKSlice, (int)rank * half, &s.raw[st]);
        }
        __syncwarp();
        if (issued < stages) ++issued;
        if (++st == stages) { st = 0; ph ^= 1u; }
      }
    }
    // the tensor core's arrivals on the stages of this CTA come from the other one too: the last of them must be in before
    // the CTA may end
    for (int i = 0; ok && i < issued; ++i) wait(&s.empty[i], i < st ? ph : ph ^ 1u);
    // a copy still in flight must not outlive the CTA (only after a wait ran out is one possible)
    if (!ok || s.dead)
      for (int i = 0; i < issued; ++i)
        for (int k = 0; k < P.wait_limit && !mbar_wait(&s.raw[i], (i < st ? ph : ph ^ 1u), 1); ++k) {}
  } else if (warp == kRgEpiWarps + kRgSplitWarps + 1) {
    // ---- products (even CTA): the whole warp, see elect_one ----
    if (rank == 0) {
      const unsigned idesc = pair_idesc(N);
      int st = 0, buf = 0, uses = 0;  // uses: accumulators handed out so far
      unsigned ph = 0, acc_ph = 0;
      bool ok = true;
      auto wait = [&](unsigned long long *bar, unsigned parity) {
        return ok = __all_sync(kFull, pair_wait<true>(bar, parity, s.dead, P.wait_limit));
      };
      auto take = [&]() {  // the accumulator has been read
        if (uses >= 2 && !wait(&s.acc_empty[buf], acc_ph ^ 1u)) return false;
        if (uses < 2) ++uses;
        return true;
      };
      const unsigned tmem = s.tmem_base;
      for (int t = pair; t < P.tiles && ok; t += pairs) {
        if (!PRECISE && !take()) break;
        for (int sl = 0; sl < P.n_slices; ++sl) {
          if (PRECISE && !take()) break;
          if (!wait(&s.ready[st], ph)) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned d = tmem + (unsigned)(buf * 256);
          const unsigned b = smem_u32(smem + st * stage_bytes);
          const unsigned long long ah = umma_desc_sw128(b), al = umma_desc_sw128(b + kTcRows * 128);
          const unsigned long long wh = umma_desc_sw128(b + 2 * kTcRows * 128), wl = umma_desc_sw128(b + 2 * kTcRows * 128 + half * 128);
          const unsigned fresh = PRECISE || sl == 0;
          const bool last = PRECISE || sl == P.n_slices - 1;
          auto mma = [&](int j, int term, unsigned add) {  // K step j (eight TF32 values inside the swizzle row) of lo*hi, hi*lo, hi*hi
            pair_mma(d + (unsigned)((j & (accs - 1)) * acc_cols), (term == 0 ? al : ah) + j * kUmmaStep, (term == 1 ? wl : wh) + j * kUmmaStep,
                     idesc, add);
          };
          if (elect_one()) {
            if (accs > 1 || P.small_first) {
#pragma unroll
              for (int term = 0; term < 3; ++term)
#pragma unroll
                for (int j = 0; j < kTcKSlice / 8; ++j) mma(j, term, fresh && term == 0 && j < accs ? 0u : 1u);
            } else {  // in the order of gemm_tc.cuh: the same bits
#pragma unroll
              for (int j = 0; j < kTcKSlice / 8; ++j) {
                mma(j, 2, fresh && j == 0 ? 0u : 1u);
                mma(j, 1, 1u);
                mma(j, 0, 1u);
              }
            }
            pair_commit(&s.empty[st]);
            if (last) pair_commit(&s.acc_full[buf]);
          }
          __syncwarp();
          if (last) {
            buf ^= 1;
            if (buf == 0) acc_ph ^= 1u;
          }
          if (++st == stages) { st = 0; ph ^= 1u; }
        }
      }
      if (!ok) {  // products still running read shared memory of both CTAs
        if (elect_one()) pair_commit(&s.drained);
        mbar_wait(&s.drained, 0, P.wait_limit);
      }
    }
  } else if (warp >= kRgEpiWarps) {
    // ---- split the raw rows: hi in place, lo beside it ----
    const int w = tid - 32 * kRgEpiWarps;
    constexpr int kStep = 32 * kRgSplitWarps, kQuads = kTcRows * 8 / kStep;  // quads of a thread in a slice, from one to the next
    const float round_low = P.cut_low ? 1.f : kRoundLow;
    int st = 0;
    unsigned ph = 0;
    bool ok = true;
    for (int t = pair; t < P.tiles && ok; t += pairs)
      for (int sl = 0; sl < P.n_slices; ++sl) {
        if (!(ok = __all_sync(kFull, pair_wait(&s.raw[st], ph, s.dead, P.wait_limit)))) break;  // (the warp leaves as one)
        float4 *hi = reinterpret_cast<float4 *>(smem + st * stage_bytes), *lo = hi + kTcRows * 8;
        float4 a[kQuads];
        if (!P.direct) {
#pragma unroll
          for (int i = 0; i < kQuads; ++i) a[i] = hi[w + i * kStep];
        } else {  // rows that TMA cannot read: the same quads of the swizzled tile, value by value
#pragma unroll
          for (int i = 0; i < kQuads; ++i) {
            const int q = w + i * kStep, r = q >> 3, row = t * 2 * kTcRows + (int)rank * kTcRows + r;
            const int k = sl * kTcKSlice + ((q & 7) ^ (r & 7)) * 4;
            const float *x = P.x + (size_t)row * P.ld_x + k;
            const bool in = row < P.m;
            a[i] = make_float4(in && k < P.k ? __ldg(x) : 0.f, in && k + 1 < P.k ? __ldg(x + 1) : 0.f,
                               in && k + 2 < P.k ? __ldg(x + 2) : 0.f, in && k + 3 < P.k ? __ldg(x + 3) : 0.f);
          }
        }
#pragma unroll
        for (int i = 0; i < kQuads; ++i) {
          float4 h, l;
          split_pair(a[i].x, round_low, h.x, l.x); split_pair(a[i].y, round_low, h.y, l.y);
          split_pair(a[i].z, round_low, h.z, l.z); split_pair(a[i].w, round_low, h.w, l.w);
          hi[w + i * kStep] = h;
          lo[w + i * kStep] = l;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // read next by the tensor core
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) pair_arrive_leader(&s.ready[st]);
        if (++st == stages) { st = 0; ph ^= 1u; }
      }
  } else {
    // ---- drain: warp w holds the rows 32 (w % 4) .. + 31 of the CTA's half of the tile (PRECISE: 32 columns of them) ----
    const int quadrant = warp & 3, side = warp >> 2;
    int buf = 0, eb = 0;
    unsigned acc_ph = 0;
    bool ok = true;
    const unsigned lanes = s.tmem_base + ((unsigned)(quadrant * 32) << 16);
    auto release = [&]() {  // the accumulator has been read: its next use may overwrite it
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) pair_arrive_leader(&s.acc_empty[buf]);
    };
    auto next = [&]() {
      buf ^= 1;
      if (buf == 0) acc_ph ^= 1u;
    };
    // 32 columns from c on of this lane's row
    auto put = [&](const float (&x)[32], int c, int row0) {
      // (PRECISE) A sum that is no finite number is taken once more with FMAs: the halves of an infinity, or of a number that
      // rounding carries to one, give infinity - infinity where FMAs give the infinity, or the finite sum.
      unsigned odd = 0;
      if (PRECISE) {
#pragma unroll
        for (int q = 0; q < 32; ++q)
          if (!isfinite(x[q]) && c + q < P.n_real && row0 + lane < P.m) odd |= 1u << q;
      }
      auto exact = [&](int col) {  // (one addition at a time: rare, and registers are short)
        const float *xr = P.x + (size_t)(row0 + lane) * P.ld_x, *wc = P.w + (size_t)col * P.w_c;
        float sum = 0.f;
#pragma unroll 1
        for (int k = 0; k < P.k; ++k) sum = fmaf(__ldg(xr + k), __ldg(wc + (size_t)k * P.w_k), sum);
        return P.relu ? fmaxf(sum, 0.f) : sum;
      };
      float v[32];
#pragma unroll
      for (int q = 0; q < 32; ++q) v[q] = P.relu ? fmaxf(x[q], 0.f) : x[q];
      if (P.tma_store) {
        float4 *blk = reinterpret_cast<float4 *>(epi + (PRECISE ? warp : warp * 2 + eb) * 4096);
        if (PRECISE) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the store before has left the buffer
        else asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");          // (there are two)
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q) blk[lane * 8 + (q ^ (lane & 7))] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        for (; PRECISE && odd; odd &= odd - 1) {
          const int q = __ffs(odd) - 1;
          reinterpret_cast<float *>(blk + lane * 8 + (q / 4 ^ (lane & 7)))[q % 4] = exact(c + q);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (elect_one())
          asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                           (unsigned long long)&tm_out), "r"(smem_u32(blk)), "r"(c), "r"(row0) : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        eb ^= 1;
      } else if (row0 + lane < P.m) {
        float *d = P.out + (size_t)(row0 + lane) * P.ld_out + c;
#pragma unroll
        for (int q = 0; q < 32; ++q)
          if (c + q < P.n_real) d[q] = v[q];
        for (; PRECISE && odd; odd &= odd - 1) d[__ffs(odd) - 1] = exact(c + __ffs(odd) - 1);
      }
    };
    for (int t = pair; t < P.tiles && ok; t += pairs) {
      const int row0 = t * 2 * kTcRows + (int)rank * kTcRows + quadrant * 32;
      if (PRECISE) {
        float acc[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) acc[q] = 0.f;
        for (int sl = 0; sl < P.n_slices; ++sl) {
          if (!(ok = __all_sync(kFull, pair_wait(&s.acc_full[buf], acc_ph, s.dead, P.wait_limit)))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (side * 32 < N) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float a[32];
              tmem_load32(a, lanes + (unsigned)(buf * 256 + j * 64 + side * 32));
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              tmem_loaded(a);
#pragma unroll
              for (int q = 0; q < 32; ++q) acc[q] += a[q];
            }
          }
          release();
          next();
        }
        if (!ok) break;
        if (row0 < P.m && side * 32 < P.n_real) put(acc, side * 32, row0);
      } else {
        if (!(ok = __all_sync(kFull, pair_wait(&s.acc_full[buf], acc_ph, s.dead, P.wait_limit)))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int c = 0; c < N; c += 32) {
          float v[32];
          tmem_load32(v, lanes + (unsigned)(buf * 256 + c));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          tmem_loaded(v);
          for (int i = 1; i < accs; ++i) {
            float a[32];
            tmem_load32(a, lanes + (unsigned)(buf * 256 + i * acc_cols + c));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            tmem_loaded(a);
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] += a[q];
          }
          if (c + 32 >= N) release();
          if (c < P.n_real && row0 < P.m) put(v, c, row0);
        }
        next();
      }
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && s.dead) atomicExch(P.error, 1);
  pair_sync();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(s.tmem_base), "n"(512) : "memory");
  }
}

// out = X * W for few terms (K < kRgPreciseMinK) with fp32 FMAs in the order of the terms, as the ticket executor's CUDA-core
// tile has them: the same bits.  W stays in shared memory, a CTA walks tiles of 128 rows (transposed, so that a thread reads
// four of a term at once), a thread computes 8 rows x 4 columns at a time: three reads for 32 FMAs.  The result, written once,
// bounds it.  (Whole GeMM-SpMM calls, 17 terms, 128 x 128 x 64 points: 64 columns 262 us, 205 with the precise form, 1 127 on
// the ticket executor; 256 columns 768, 853 and 2 728.)
constexpr int kFmaThreads = 256, kFmaRows = 128, kFmaLd = kFmaRows + 4;
static_assert((256 + kFmaLd) * (kRgPreciseMinK - 1) * 4 <= 48 * 1024, "W and the rows fit the shared memory every launch has");
__global__ void __launch_bounds__(kFmaThreads)
row_fma_kernel(const float *__restrict__ X, int m, int K, int ld_x, const float *__restrict__ W, int w_transposed, int n,
               float *__restrict__ out, int ld_out, int relu, bool vec) {
  extern __shared__ float4 fma_smem[];
  const int quads = (n + 3) / 4, tid = threadIdx.x;
  float *w = reinterpret_cast<float *>(fma_smem), *x = w + 4 * quads * K;  // W [K][4 * quads], the rows [K][kFmaLd]
  for (int i = tid; i < 4 * quads * K; i += kFmaThreads) {
    const int k = i / (4 * quads), c = i - k * 4 * quads;
    w[i] = c < n ? __ldg(w_transposed ? W + (size_t)c * K + k : W + (size_t)k * n + c) : 0.f;
  }
  for (long long r0 = (long long)blockIdx.x * kFmaRows; r0 < m; r0 += (long long)gridDim.x * kFmaRows) {
    __syncthreads();  // W is complete, or the rows of the tile before have been read
    for (int i = tid; i < kFmaRows * K; i += kFmaThreads) {
      const int r = i / K, k = i - r * K;
      x[k * kFmaLd + r] = r0 + r < m ? __ldg(X + (size_t)(r0 + r) * ld_x + k) : 0.f;
    }
    __syncthreads();
    for (int i = tid; i < quads * (kFmaRows / 8); i += kFmaThreads) {
      const int g = i / quads, q = i - g * quads;
      float4 acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      const float *xg = x + 8 * g, *wq = w + 4 * q;
      for (int k = 0; k < K; ++k, xg += kFmaLd, wq += 4 * quads) {
        const float4 b = *reinterpret_cast<const float4 *>(wq);
        const float4 lo = *reinterpret_cast<const float4 *>(xg), hi = *reinterpret_cast<const float4 *>(xg + 4);
        const float a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[j].x = fmaf(a[j], b.x, acc[j].x); acc[j].y = fmaf(a[j], b.y, acc[j].y);
          acc[j].z = fmaf(a[j], b.z, acc[j].z); acc[j].w = fmaf(a[j], b.w, acc[j].w);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (r0 + 8 * g + j >= m) break;
        float4 v = acc[j];
        if (relu) v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
        float *o = out + (size_t)(r0 + 8 * g + j) * ld_out + 4 * q;
        if (vec && 4 * q + 3 < n) *reinterpret_cast<float4 *>(o) = v;
        else {
          o[0] = v.x;
          if (4 * q + 1 < n) o[1] = v.y;
          if (4 * q + 2 < n) o[2] = v.z;
          if (4 * q + 3 < n) o[3] = v.w;
        }
      }
    }
  }
}

// hi / lo [n_pad][ldk] (K contiguous, rows from n on and columns from K on zero) from W [K][n], or from W [n][K] when w_transposed.
__global__ void split_weight_pad_kernel(const float *__restrict__ W, int w_transposed, int K, int ldk, int n, int n_pad, bool ticket,
                                        float *__restrict__ hi, float *__restrict__ lo) {
  const int total = n_pad * ldk;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int r = i / ldk, k = i - r * ldk;
    float w = 0.f;
    if (r < n && k < K) w = w_transposed ? __ldg(W + (size_t)r * K + k) : __ldg(W + (size_t)k * n + r);
    const float h = tf32_round(w);
    hi[i] = h;
    lo[i] = ticket ? w - h : tf32_round(w - h);
  }
}

}  // namespace

bool row_gemm_supported(int n) { return n >= 1 && n <= kTcMaxN; }
int row_gemm_pad_n(int n) { return (n + 31) / 32 * 32; }  // cta_group::2 takes multiples of 32
int row_gemm_pad_k(int k) { return (k + 3) / 4 * 4; }

RowGemmForm row_gemm_form(int K, int n) { return tc_supported(K, n) ? kRowTile : (K >= kRgPreciseMinK ? kRowPrecise : kRowFma); }

cudaError_t row_gemm_split(const float *W, int w_transposed, int K, int n, RowGemmSums sums, float *hi, float *lo, cudaStream_t s) {
  if (row_gemm_form(K, n) == kRowFma) return cudaSuccess;
  const bool ticket = sums == kSumsTicket && row_gemm_form(K, n) == kRowTile;
  const int ldk = row_gemm_pad_k(K), n_pad = row_gemm_pad_n(n);
  split_weight_pad_kernel<<<std::min((n_pad * ldk + 255) / 256, 148 * 4), 256, 0, s>>>(W, w_transposed, K, ldk, n, n_pad, ticket, hi, lo);
  return cudaGetLastError();
}

static int launch_fma(const float *X, int m, int K, int ld_x, const float *W, int w_transposed, int n, float *out, int ld_out, bool relu,
                      int sm_count, cudaStream_t s) {
  const int quads = (n + 3) / 4;
  const size_t smem = (size_t)(4 * quads + kFmaLd) * K * 4;
  const bool vec = ld_out % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  row_fma_kernel<<<std::max(1, std::min((m + kFmaRows - 1) / kFmaRows, sm_count * 4)), kFmaThreads, smem, s>>>(
      X, m, K, ld_x, W, w_transposed, n, out, ld_out, relu ? 1 : 0, vec);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TF_OK : tf::fail(TF_ERR_CUDA, std::string("row_gemm: ") + cudaGetErrorString(e));
}

static int launch_panel(const float *X, int m, int K, int ld_x, const float *W, int w_k, int w_c, const float *hi, const float *lo, int n, float *out, int ld_out, bool relu,
                        bool precise, RowGemmSums sums, int *error, int wait_limit, int sm_count, cudaStream_t s) {
  const int n_pad = row_gemm_pad_n(n), ldk = row_gemm_pad_k(K);
  CUtensorMap ma, mh, ml, mo;
  RowGemmParams P;
  P.x = X; P.k = K; P.ld_x = ld_x;
  P.w = W; P.w_k = w_k; P.w_c = w_c;
  P.cut_low = sums == kSumsTicket ? 1 : 0;
  P.small_first = sums == kSumsSpmmGemm ? 1 : 0;
  P.direct = ld_x % 4 != 0 || (reinterpret_cast<uintptr_t>(X) & 15) != 0;
  int rc = tc_make_map(&mh, hi, n_pad, ldk, n_pad / 2, ldk);
  if (rc == TF_OK) rc = tc_make_map(&ml, lo, n_pad, ldk, n_pad / 2, ldk);
  P.m = m; P.n_pad = n_pad; P.n_real = n; P.n_slices = (K + kTcKSlice - 1) / kTcKSlice;
  P.tiles = (m + 2 * kTcRows - 1) / (2 * kTcRows);
  P.stages = rg_stages(n_pad);
  P.accs = sums == kSumsTicket || n_pad > 128 ? 1 : (n_pad > 64 ? 2 : 4);
  P.out = out; P.ld_out = ld_out; P.relu = relu ? 1 : 0;
  P.tma_store = ld_out % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  P.error = error; P.wait_limit = wait_limit;
  if (rc != TF_OK) return rc;
  ma = mo = mh;  // (not used by the variants that have no map of their own)
  if (!P.direct) rc = tc_make_map(&ma, X, m, K, kTcRows, ld_x);
  if (rc == TF_OK && P.tma_store) rc = tc_make_map(&mo, out, m, n, 32, ld_out);
  if (rc != TF_OK) return rc;
  const size_t smem = (size_t)P.stages * rg_stage_bytes(n_pad) + kRgEpiBytes + 1024;
  auto f = precise ? row_gemm_kernel<true> : row_gemm_kernel<false>;
  // (the limit is the kernel's, not the call's: the same for all widths, so that threads with different plans don't lower it
  // for one another)
  cudaError_t e = cudaFuncSetAttribute((const void *)f, cudaFuncAttributeMaxDynamicSharedMemorySize, kRgSmemMax - 1024);
  if (e == cudaSuccess) {
    f<<<2 * std::max(1, std::min(P.tiles, sm_count / 2)), rg_threads(precise), smem, s>>>(ma, mh, ml, mo, P);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return tf::fail(TF_ERR_CUDA, std::string("row_gemm: ") + cudaGetErrorString(e));
  return TF_OK;
}

int row_gemm(const float *X, int m, int K, int ld_x, const float *W, int w_transposed, const float *hi, const float *lo, int n,
             float *out, int ld_out, bool relu, RowGemmSums sums, int *error, int wait_limit, int sm_count, cudaStream_t s) {
  const RowGemmForm form = row_gemm_form(K, n);
  if (form == kRowFma) return launch_fma(X, m, K, ld_x, W, w_transposed, n, out, ld_out, relu, sm_count, s);
  const bool precise = form == kRowPrecise;
  if (precise) sums = kSumsFree;
  const int panel = precise ? kRgPrecisePanel : n;
  for (int c = 0; c < n; c += panel) {
    const size_t off = (size_t)c * row_gemm_pad_k(K);
    const int w_k = w_transposed ? 1 : n, w_c = w_transposed ? K : 1;
    const int rc = launch_panel(X, m, K, ld_x, W + (size_t)c * w_c, w_k, w_c, hi + off, lo + off, std::min(panel, n - c), out + c, ld_out,
                                relu, precise, sums, error, wait_limit, sm_count, s);
    if (rc != TF_OK) return rc;
  }
  return TF_OK;
}

}  // namespace tfk
