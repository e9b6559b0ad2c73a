// SpMM-SpMM on banded operators (band_march.h): D = A * (F * C), one launch, T = F * C in shared memory.
//
// A CTA takes 32 dense columns (128 bytes of a row) and a range of rows and marches down the band in blocks of as many rows
// as a nonzero can be away from the diagonal (64, or 128).  A ring of four blocks of C and one of four blocks of T hold
// whatever a row can name: in step s the CTA computes block s of T from the blocks s - 1 .. s + 1 of C and block s - 2 of D
// from the blocks s - 3 .. s - 1 of T, while TMA brings block s + 2 of C and the nonzeros of the rows of that block (a ring
// of five, because block s - 2 is still being read).  The two products of a step do not depend on each other, so a step has
// one barrier.
// Two kernels do this.  In band_march_kernel a warp works on four rows at a time, eight lanes with a float4 each per row: a
// quarter-warp reads one row of 128 bytes, which is free of bank conflicts whatever rows are named.  What bounds it is the
// shared memory pipe: one wavefront per nonzero, product and 32 columns, and half of one for the nonzero itself, which eight
// lanes read.  band_lane_kernel gives a lane a row of its own and reads a nonzero once (n = 200 003, 12 nonzeros within 40 of the diagonal,
// 96 columns: 100.6 us and 78.4; 400 000, 16 within 60, 128 columns: 322 and 245; 5 within 12: 159 and 107); see band_threads.  (Read from global memory,
// the nonzeros took their warps to L2 for every four rows, since the rings leave no L1: 168 us instead of 104 for
// n = 200 003, 12 nonzeros within 40 of the diagonal, 96 columns; the tile pipeline takes 150.)
// Products are added in CSR order with fused multiply-adds from zero, and nothing is multiplied that is not stored, so
// results are bit for bit those of the CSR executors.
#include <algorithm>

#include "band_march.h"
#include "gemm_tc.cuh"
#include "gemm_tc_host.h"
#include "segments.h"

namespace tfk {

namespace {

constexpr int kBandSlots = 5;

// Four rows of one product: row (lane >> 3) of the four that start at `row`, this lane's four columns.  ring: the operand;
// quads: the nonzeros of the block that the rows belong to.
template <int S>
__device__ __forceinline__ float4 band_row(const int4 *quads, int pairs, int row, const char *ring, int lane) {
  constexpr unsigned mask = 4u * S * 128u - 1;
  const int r = row + (lane >> 3);
  const int4 *q = quads + (r & (S - 1));
  const unsigned base = (unsigned)r * 128u;  // (modulo the ring, which is a power of two; the row count is not bounded by it)
  const char *col = ring + (lane & 7) * 16;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < pairs; ++k) {
    const int4 e = q[k * S];
    const float4 x = *reinterpret_cast<const float4 *>(col + ((base + (unsigned)(e.x & ~1)) & mask));
    const float4 y = *reinterpret_cast<const float4 *>(col + ((base + (unsigned)(e.z & ~1)) & mask));
    if (!(e.x & 1)) {
      const float v = __int_as_float(e.y);
      acc.x = fmaf(v, x.x, acc.x); acc.y = fmaf(v, x.y, acc.y); acc.z = fmaf(v, x.z, acc.z); acc.w = fmaf(v, x.w, acc.w);
    }
    if (!(e.z & 1)) {
      const float v = __int_as_float(e.w);
      acc.x = fmaf(v, y.x, acc.x); acc.y = fmaf(v, y.y, acc.y); acc.z = fmaf(v, y.z, acc.z); acc.w = fmaf(v, y.w, acc.w);
    }
  }
  return acc;
}

__device__ __forceinline__ void bulk_load(void *smem, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

template <int S>
__global__ void __launch_bounds__(kBandThreads, S == 64 ? 2 : 1)
band_march_kernel(const __grid_constant__ CUtensorMap tm_c, const BandParams P) {
  constexpr unsigned kRing = 4u * S * 128u;
  constexpr int kWarps = kBandThreads / 32;
  extern __shared__ char dyn[];
  __shared__ unsigned long long full[4];
  char *c_ring = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~(uintptr_t)1023);
  char *t_ring = c_ring + kRing;
  const unsigned bytes_f = (unsigned)P.pairs_f * S * 16, bytes_a = P.same ? 0u : (unsigned)P.pairs_a * S * 16;
  char *f_ring = t_ring + kRing, *a_ring = P.same ? f_ring : f_ring + kBandSlots * bytes_f;
  const unsigned step_a = P.same ? bytes_f : bytes_a;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunk = blockIdx.x % P.chunks, seg = blockIdx.x / P.chunks;
  const int jb = P.block_begin + seg * P.seg_blocks, je = min(P.block_end, jb + P.seg_blocks);
  const int col0 = chunk * 32, col = col0 + (lane & 7) * 4;
  const int first = max(0, jb - 2), end = min(P.blocks, je + 2);  // blocks of C that the segment reads
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(&full[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto load = [&](int b) {
    unsigned long long *bar = &full[b & 3];
    mbar_expect_tx(bar, S * 128 + bytes_f + bytes_a);
    tma_load_2d(c_ring + (size_t)(b & 3) * (S * 128), &tm_c, col0, b * S, bar);
    bulk_load(f_ring + (b % kBandSlots) * bytes_f, P.quads_f + (size_t)b * P.pairs_f * S, bytes_f, bar);
    if (bytes_a) bulk_load(a_ring + (b % kBandSlots) * bytes_a, P.quads_a + (size_t)b * P.pairs_a * S, bytes_a, bar);
  };
  int issued = first;
  if (tid == 0)
    for (; issued < min(end, jb + 1); ++issued) load(issued);
  int landed = first;  // blocks that have arrived
  bool ok = true;
  for (int s = jb - 1; s <= je + 1; ++s) {
    if (tid == 0 && s + 2 >= issued && s + 2 < end) { load(s + 2); issued = s + 3; }
    for (; ok && landed < min(end, s + 2); ++landed)
      ok = mbar_wait(&full[landed & 3], (unsigned)((landed - first) >> 2) & 1u, P.wait_limit);
    if (ok && s >= 0 && s < P.blocks && s <= je) {
      const int4 *quads = reinterpret_cast<const int4 *>(f_ring + (s % kBandSlots) * bytes_f);
#pragma unroll
      for (int q = 0; q < S / 4; q += kWarps) {
        const int row = s * S + 4 * (q + warp);
        const float4 t = band_row<S>(quads, P.pairs_f, row, c_ring, lane);
        *reinterpret_cast<float4 *>(t_ring + (((unsigned)(row + (lane >> 3)) * 128u) & (kRing - 1)) + (lane & 7) * 16) = t;
      }
    }
    if (ok && s - 2 >= jb) {
      const int4 *quads = reinterpret_cast<const int4 *>(a_ring + ((s - 2) % kBandSlots) * step_a);
#pragma unroll
      for (int q = 0; q < S / 4; q += kWarps) {
        const int row = (s - 2) * S + 4 * (q + warp), mine = row + (lane >> 3);
        const float4 d = band_row<S>(quads, P.same ? P.pairs_f : P.pairs_a, row, t_ring, lane);
        if (mine < P.m && col < P.n_cols) *reinterpret_cast<float4 *>(P.out + (size_t)mine * P.n_cols + col) = d;
      }
    }
    if (__syncthreads_or(!ok)) { ok = false; break; }
  }
  if (!ok && tid == 0) {
    // a wait ran out: no copy may outlive the CTA, so wait (again with a limit) for those in flight
    for (int b = max(first, issued - 4); b < issued; ++b)
      mbar_wait(&full[b & 3], (unsigned)((b - first) >> 2) & 1u, P.wait_limit);
    atomicExch(P.error, 1);
  }
}

// The same march with a row to a lane: 2 * S / 32 warps, half of them with a block of T, half with one of D.  A lane reads the
// eight 16-byte chunks of a row that it names in an order of its own, chunk (lane + i) % 8 in turn i, so that the eight lanes of
// a quarter-warp never meet in a bank whatever rows they name, and turn i of all nonzeros adds up in the same registers.  A
// nonzero is read once and not by eight lanes.  Rows of D are turned round in shared memory and leave as TMA stores.
template <int S>
__device__ __forceinline__ void band_lane(float4 (&acc)[8], const int4 *quads, int pairs, unsigned row, const char *ring, const unsigned (&chunk)[8]) {
  constexpr unsigned mask = 4u * S * 128u - 1;
  const int4 *q = quads + (row & (S - 1));
  const unsigned base = row * 128u;  // (modulo the ring, see band_row)
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  int4 e = q[0];
  for (int k = 0; k < pairs; ++k) {
    const int4 f = e;
    e = q[(k + 1 < pairs ? k + 1 : k) * S];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int off = h ? f.z : f.x;
      const float v = __int_as_float(h ? f.w : f.y);
      const char *r = ring + ((base + (unsigned)(off & ~1)) & mask);
      float4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const float4 *>(r + chunk[i]);
      if (!(off & 1)) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          acc[i].x = fmaf(v, x[i].x, acc[i].x); acc[i].y = fmaf(v, x[i].y, acc[i].y);
          acc[i].z = fmaf(v, x[i].z, acc[i].z); acc[i].w = fmaf(v, x[i].w, acc[i].w);
        }
      }
    }
  }
}

template <int S>
__global__ void __launch_bounds__(2 * S, S == 64 ? 2 : 1)
band_lane_kernel(const __grid_constant__ CUtensorMap tm_c, const __grid_constant__ CUtensorMap tm_d, const BandParams P) {
  constexpr unsigned kRing = 4u * S * 128u;
  constexpr int kHalf = S / 32;  // warps with T, and warps with D
  extern __shared__ char dyn[];
  __shared__ unsigned long long full[4];
  char *c_ring = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(dyn) + 127) & ~(uintptr_t)127);
  char *t_ring = c_ring + kRing, *stage = t_ring + kRing;  // stage: 32 rows of D per warp
  const unsigned bytes_f = (unsigned)P.pairs_f * S * 16, bytes_a = P.same ? 0u : (unsigned)P.pairs_a * S * 16;
  char *f_ring = stage + S * 128, *a_ring = P.same ? f_ring : f_ring + kBandSlots * bytes_f;
  const unsigned step_a = P.same ? bytes_f : bytes_a;
  const int tid = threadIdx.x, warp = __shfl_sync(kFull, tid >> 5, 0), lane = tid & 31;  // (known to be uniform)
  const int seg = blockIdx.x / P.chunks, col0 = (blockIdx.x - seg * P.chunks) * 32;
  const int jb = P.block_begin + seg * P.seg_blocks, je = min(P.block_end, jb + P.seg_blocks);
  const int first = max(0, jb - 2), end = min(P.blocks, je + 2);  // blocks of C that the segment reads
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(&full[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto load = [&](int b) {  // the first warp, see elect_one
    if (elect_one()) {
      unsigned long long *bar = &full[b & 3];
      mbar_expect_tx(bar, S * 128 + bytes_f + bytes_a);
      tma_load_2d(c_ring + (size_t)(b & 3) * (S * 128), &tm_c, col0, b * S, bar);
      bulk_load(f_ring + (b % kBandSlots) * bytes_f, P.quads_f + (size_t)b * P.pairs_f * S, bytes_f, bar);
      if (bytes_a) bulk_load(a_ring + (b % kBandSlots) * bytes_a, P.quads_a + (size_t)b * P.pairs_a * S, bytes_a, bar);
    }
    __syncwarp();
  };
  unsigned chunk[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) chunk[i] = ((lane + i) & 7) * 16;
  int issued = first;
  if (warp == 0)
    for (; issued < min(end, jb + 1); ++issued) load(issued);
  int landed = first;  // blocks that have arrived
  bool ok = true;
  for (int s = jb - 1; s <= je + 1; ++s) {
    if (warp == 0 && s + 2 >= issued && s + 2 < end) { load(s + 2); issued = s + 3; }
    for (; ok && landed < min(end, s + 2); ++landed)
      ok = __all_sync(kFull, mbar_wait(&full[landed & 3], (unsigned)((landed - first) >> 2) & 1u, P.wait_limit));  // (the warp leaves as one)
    float4 acc[8];
    if (warp < kHalf) {
      if (ok && s >= 0 && s < P.blocks && s <= je) {
        const unsigned row = (unsigned)(s * S + warp * 32 + lane);
        band_lane<S>(acc, reinterpret_cast<const int4 *>(f_ring + (s % kBandSlots) * bytes_f), P.pairs_f, row, c_ring, chunk);
        char *o = t_ring + ((row * 128u) & (kRing - 1));
#pragma unroll
        for (int i = 0; i < 8; ++i) *reinterpret_cast<float4 *>(o + chunk[i]) = acc[i];
      }
    } else if (ok && s - 2 >= jb) {
      const int row0 = (s - 2) * S + (warp - kHalf) * 32;
      band_lane<S>(acc, reinterpret_cast<const int4 *>(a_ring + ((s - 2) % kBandSlots) * step_a), P.same ? P.pairs_f : P.pairs_a,
                   (unsigned)(row0 + lane), t_ring, chunk);
      char *o = stage + (warp - kHalf) * 4096;
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the rows before have left the buffer
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) *reinterpret_cast<float4 *>(o + lane * 128 + chunk[i]) = acc[i];
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (row0 < P.m && elect_one())
        asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"((unsigned long long)&tm_d),
                     "r"(smem_u32(o)), "r"(col0), "r"(row0) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    if (__syncthreads_or(!ok)) { ok = false; break; }
  }
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if (!ok && warp == 0) {
    // a wait ran out: no copy may outlive the CTA, so wait (again with a limit) for those in flight
    for (int b = max(first, issued - 4); b < issued; ++b)
      mbar_wait(&full[b & 3], (unsigned)((b - first) >> 2) & 1u, P.wait_limit);
    if (lane == 0) atomicExch(P.error, 1);
  }
}

}  // namespace

static_assert(kBandSmemMax <= 227 * 1024 - 64, "with the four barriers, what a CTA has");

int band_make_map(CUtensorMap *out, const float *c, long long rows, int n_cols, int block) {
  return tc_make_map(out, c, rows, n_cols, block, n_cols, false);
}

size_t band_smem(int block, int pairs_f, int pairs_a, bool same) {
  return 1024 + (size_t)block * (2 * 4 * 128 + kBandSlots * 16 * (size_t)(pairs_f + (same ? 0 : pairs_a)));
}

// What the kernel with a row to a lane takes on top: 32 rows of D per warp.
static size_t lane_smem(int block, int pairs_f, int pairs_a, bool same) { return band_smem(block, pairs_f, pairs_a, same) - 896 + (size_t)block * 128; }
constexpr size_t kBandSmemTwo = (228 * 1024) / 2 - 1024 - 64;  // of a CTA where two share an SM

// The kernel with a row to a lane takes 30 % fewer wavefronts of shared memory but has 8 warps on an SM, which is enough where two
// CTAs share it (or one with blocks of 128), and where they march: with no more than two blocks of rows to a CTA the latency of
// a block counts, and the 16 warps of the other kernel are ahead (10 000 rows, 12 within 40, 96 columns: 12.5 us and 12.7; 5 003
// rows, 64 columns: 9.1 and 9.9; 30 000 rows, 64 columns: 16.5 and 14.2; two operators of 12 nonzeros, one CTA per SM: 118 and 119).
int band_threads(int block, const BandParams &p, int sm_count) {
  const size_t smem = lane_smem(block, p.pairs_f, p.pairs_a, p.same);
  const bool two = block == 64 && smem <= kBandSmemTwo;
  if (smem > kBandSmemMax || (block == 64 && !two)) return kBandThreads;
  const long long blocks = (p.m + block - 1) / block, chunks = (p.n_cols + 31) / 32;
  return blocks * chunks > 2LL * sm_count * (two ? 2 : 1) ? 2 * block : kBandThreads;
}

template <int S>
static cudaError_t launch(const CUtensorMap &tm_c, const CUtensorMap &tm_d, BandParams &p, int sm_count, cudaStream_t s) {
  p.chunks = (p.n_cols + 31) / 32;
  p.blocks = (p.m + S - 1) / S;
  const int n = p.block_end - p.block_begin;
  if (n <= 0) return cudaSuccess;
  const bool lanes = band_threads(S, p, sm_count) != kBandThreads;
  const size_t smem = lanes ? lane_smem(S, p.pairs_f, p.pairs_a, p.same) : band_smem(S, p.pairs_f, p.pairs_a, p.same);
  const long long resident = (long long)sm_count * (S == 64 && smem <= (lanes ? kBandSmemTwo : 112 * 1024) ? 2 : 1);
  p.seg_blocks = tf::segment_length(n, p.chunks, resident, 3, 1);  // a segment of n blocks of D takes n + 3 steps
  // (the limit is the kernel's, not the call's: the same for all operators, so that threads with different plans don't lower it
  // for one another)
  const void *f = lanes ? (const void *)band_lane_kernel<S> : (const void *)band_march_kernel<S>;
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kBandSmemMax);
  if (e != cudaSuccess) return e;
  const long long ctas = (long long)((n + p.seg_blocks - 1) / p.seg_blocks) * p.chunks;
  if (lanes) band_lane_kernel<S><<<(unsigned)ctas, 2 * S, smem, s>>>(tm_c, tm_d, p);
  else band_march_kernel<S><<<(unsigned)ctas, kBandThreads, smem, s>>>(tm_c, p);
  return cudaGetLastError();
}

cudaError_t launch_band_march(const CUtensorMap &tm_c, const CUtensorMap &tm_d, int block, BandParams &p, int sm_count, cudaStream_t s) {
  return block == 64 ? launch<64>(tm_c, tm_d, p, sm_count, s) : launch<128>(tm_c, tm_d, p, sm_count, s);
}

}  // namespace tfk
