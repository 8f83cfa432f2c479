// Device helpers shared by the tcgen05 GEMM kernels: shared-memory
// addresses, bounded mbarrier waits, TMA 2-D tile loads, shared-memory matrix
// descriptors (128-byte swizzle) and the kind::f16 instruction descriptor.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include <cstdint>

namespace fcc {
namespace tc5 {

constexpr long long WAIT_CLK = 4000000000ll;  // every mbarrier wait gives up after about 2 s of SM clocks

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Bounded wait on an mbarrier phase; false after WAIT_CLK.  The limit is
// counted on the SM clock: a wait that is not satisfied at once is the normal
// case in every pipeline here, and reading %globaltimer in it costs more than
// the wait itself.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (it == 0) t0 = clock64();
    else if ((it & 15) == 0 && clock64() - t0 > WAIT_CLK) return false;
  }
}

// True in one lane of a converged warp.  Roles that issue TMA loads or MMAs
// are entered through this and not through a comparison of the lane number:
// their operands sit in uniform registers, and only here does the compiler
// know that one thread runs the code.
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok));
  return ok != 0;
}

// Whether an mbarrier phase has completed, without waiting.
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* tm, int32_t x, int32_t y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle,
// 8-row groups 1024 bytes apart (SBO), fixed version bits 46-48 = 0b001.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;             // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;   // stride byte offset
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;             // SWIZZLE_128B
  return d;
}

// Instruction descriptor, kind::f16: D F32, A and B BF16, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}


__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// ---- pairs of CTAs (a cluster of two on neighbouring SMs, cta_group::2)
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of a CTA's copy of a shared variable
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// a load into this CTA signalled on a barrier of the pair's other CTA or its own
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* tm, int32_t x, int32_t y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// the barrier at this offset in both CTAs
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void mma_bf16_pair(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// One MMA (K = 16) of the calling CTA; acc = 0 overwrites the accumulator.
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}

// 32 columns of the warp's 32 TMEM lanes (wait::ld before the values are used).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}

// 16 and 8 columns likewise.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// Waits for the loads issued so far; the values named pass through it, so no
// use of them can be scheduled ahead of the wait.
template <int N>
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[N]) {
  static_assert(N % 8 == 0, "eight registers at a time");
#pragma unroll
  for (int q = 0; q < N; q += 8)
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[q]), "+r"(r[q + 1]), "+r"(r[q + 2]), "+r"(r[q + 3]), "+r"(r[q + 4]), "+r"(r[q + 5]),
                   "+r"(r[q + 6]), "+r"(r[q + 7]));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

// (double)f * 2^e (negated if neg) by integer exponent arithmetic; FP32
// subnormals and results below the FP64 normal range give 0
__device__ __forceinline__ double f32_to_f64_scaled(float f, int e, bool neg) {
  const uint32_t b = __float_as_uint(f);
  const int ex = (int)((b >> 23) & 0xFF);
  if (ex == 0) return 0.0;
  int ne = ex - 127 + 1023 + e;
  if (ne <= 0) return 0.0;
  if (ne > 2046) ne = 2047;
  const unsigned long long sign = (unsigned long long)((b >> 31) ^ (neg ? 1u : 0u)) << 63;
  const unsigned long long bits = sign | ((unsigned long long)ne << 52) | ((unsigned long long)(b & 0x7FFFFFu) << 29);
  return __longlong_as_double((long long)bits);
}

// Output tile of linear block index lin on a tm x tn tile grid, walked in
// groups of 8 tile rows (row fastest inside a group) so that the CTAs resident
// at the same time share A and B panels in L2.
// (32-bit arithmetic: a 64-bit division takes the FP64 pipe, at 1/64 rate here)
__device__ __forceinline__ void grouped_tile(uint32_t lin, uint32_t tm, uint32_t tn, uint32_t& mt, uint32_t& nt) {
  constexpr uint32_t GM = 8;
  const uint32_t per_group = GM * tn;
  const uint32_t g = lin / per_group;
  const uint32_t first = g * GM;
  const uint32_t gm = tm - first < GM ? tm - first : GM;
  const uint32_t r = lin - g * per_group;
  mt = first + r % gm;
  nt = r / gm;
}

}  // namespace tc5
}  // namespace fcc
