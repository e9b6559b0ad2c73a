// What the kernels share that run tcgen05.mma on CTA pairs (row_gemm.cu, spmm_gemm.cu): the even CTA issues the products of
// both, cta_group::2, TF32 operands, fp32 accumulators in tensor memory.
#pragma once
#include "gemm_tc.cuh"

namespace tfk {

__device__ __forceinline__ unsigned pair_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on the barrier of the even CTA of the pair.  What goes with the arrival is shared memory that the tensor cores read
// through the async proxy: fence.proxy.async has completed the writes there before, each in its own SM.  (A release at
// cluster scope would order the thread's other accesses too and costs a splitting warp half of its time: N = K = 256,
// 2.1 M rows: 1 410 us with it, 1 228 with one thread of the odd CTA that passes local arrivals on, 1 075 like this, as
// CUTLASS's ClusterBarrier::arrive has it.)
__device__ __forceinline__ void pair_arrive_leader(unsigned long long *bar) {
  asm volatile(
      "{\n\t.reg .b32 a;\n\t"
      "mapa.shared::cluster.u32 a, %0, 0;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait that also leaves when another role of the CTA has given up.  CLUSTER: threads of the other CTA arrive too.
template <bool CLUSTER = false>
__device__ __forceinline__ bool pair_wait(unsigned long long *bar, unsigned parity, int &dead, int limit) {
  const unsigned a = smem_u32(bar);
  for (int i = 0; i < limit; ++i) {
    unsigned done;
    if (CLUSTER)
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(a), "r"(parity) : "memory");
    else
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(a), "r"(parity) : "memory");
    if (done) return true;
    if (*reinterpret_cast<volatile int *>(&dead)) return false;
  }
  dead = 1;
  return false;
}
__device__ __forceinline__ unsigned pair_idesc(int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(2 * kTcRows >> 4) << 24);
}
__device__ __forceinline__ void pair_mma(unsigned d, unsigned long long da, unsigned long long db, unsigned idesc, unsigned acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
}
// Both CTAs' barriers at this offset are arrived on when the products issued so far have been computed.
__device__ __forceinline__ void pair_commit(unsigned long long *bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)), "h"((unsigned short)3) : "memory");
}

// x = hi + lo for the tensor core, which reads the first eleven bits of either.  hi is rounded to them by the addition (its last bits
// need not be cleared); a NaN may be lost there, but not in lo.  lo is a power of two or has at most twelve bits: if the last of
// them is set, lo / 2048 carries into the bit before (it is at least one unit there and less than two), if not, what it adds
// is cut off again, so that lo is rounded like hi.  (Clearing hi, rounding lo like hi and looking for NaNs first took
// eight instructions of the half-rate integer pipe, which bounded the splitting, instead of two.)
constexpr float kRoundLow = 1.f + 1.f / 2048;
__device__ __forceinline__ void split_pair(float x, float round_low, float &hi, float &lo) {
  const unsigned h = __float_as_uint(x) + 0x1000u;
  hi = __uint_as_float(h);
  lo = (x - __uint_as_float(h & 0xffffe000u)) * round_low;
}

// 32 columns of a warp's 32 tensor-memory lanes.  The registers hold them after tcgen05.wait::ld only: tmem_loaded keeps the
// compiler from using them before.
__device__ __forceinline__ void tmem_load32(float (&v)[32], unsigned taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
        "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
        "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_loaded(float (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+f"(v[i]));
}

}  // namespace tfk
