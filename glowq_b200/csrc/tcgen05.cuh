// Device primitives of the tensor-core kernels (sm_100a): bounded mbarrier waits, TMA, tcgen05.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace glowq {

// Polls of one wait before the kernel gives up (status 3), measured as about a quarter of a second: warps that run ahead of the
// dependency wait sit in these waits until the kernels before are complete, which are launches of this library as well.
constexpr uint32_t kGemmSpin = 1u << 20;

__device__ __forceinline__ uint32_t sm_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void g_mbar_init(uint32_t a, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void g_mbar_arrive(uint32_t a) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ void g_mbar_expect_tx(uint32_t a, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
template <uint32_t kLimit = kGemmSpin>
__device__ __forceinline__ bool g_mbar_wait(uint32_t a, uint32_t parity, volatile int* abort_flag, uint32_t* status) {
  uint32_t spins = 0;
  for (;;) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(a), "r"(parity)
                 : "memory");
    if (ok) return true;
    if ((++spins & 63u) == 0 && *abort_flag) return false;
    if (spins > kLimit) {
      *abort_flag = 1;
      atomicExch(status, 3u);
      return false;
    }
  }
}
// the same with cluster-scope acquire: the arrivals come from the peer CTA as well
__device__ __forceinline__ bool g_mbar_wait_cluster(uint32_t a, uint32_t parity, volatile int* abort_flag, uint32_t* status) {
  uint32_t spins = 0;
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((++spins & 63u) == 0 && *abort_flag) return false;
    if (spins > kGemmSpin) {
      *abort_flag = 1;
      atomicExch(status, 3u);
      return false;
    }
  }
}
__device__ __forceinline__ void g_tma_2d(uint32_t dst, const CUtensorMap* tmap, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(tmap), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// K-major, 128-byte-swizzled operand tile: rows of 128 B, 8-row atoms 1024 B apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(1) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
}
__device__ __forceinline__ uint64_t mk64(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ bool g_mbar_try_once(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(a), "r"(parity)
               : "memory");
  return ok != 0;
}
// Waits of a whole warp that issues tcgen05.mma: one elected lane asks, and a vote gives the answer to all, so that every branch is
// uniform in the source.  With the wait under `lane == 0` a step of eight MMAs takes 506 clocks to issue, so 171 (N = 16, one warp per
// SM, barriers open; 78 without any wait).  Supposed reason: behind a branch that may diverge the MMAs' operands are not kept uniform.
__device__ __forceinline__ uint32_t g_mbar_test_elected(uint32_t a, uint32_t parity) {   // does not suspend
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred e, p;\n\telect.sync _|e, 0xffffffff;\n\tmov.u32 %0, 0;\n\t"
      "@e mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@e selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(a), "r"(parity)
      : "memory");
  return r;
}
__device__ __forceinline__ uint32_t g_mbar_try_elected(uint32_t a, uint32_t parity) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred e, p;\n\telect.sync _|e, 0xffffffff;\n\tmov.u32 %0, 0;\n\t"
      "@e mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@e selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(a), "r"(parity)
      : "memory");
  return r;
}
template <bool kSpin>   // kSpin: the warp stays awake
__device__ __forceinline__ bool g_mbar_wait_warp(uint32_t a, uint32_t parity, volatile int* abort_flag, uint32_t* status) {
  uint32_t spins = 0;
  while (!__any_sync(0xffffffffu, kSpin ? g_mbar_test_elected(a, parity) : g_mbar_try_elected(a, parity))) {
    ++spins;
    if ((spins & 63u) == 0 && __any_sync(0xffffffffu, *abort_flag)) return false;
    if (spins > (kSpin ? 4 : 1) * kGemmSpin) {
      *abort_flag = 1;
      atomicExch(status, 3u);
      return false;
    }
  }
  return true;
}
// ---- CTA pairs: barriers of the peer CTA are reached through shared::cluster addresses.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {  // shared::cta -> shared::cluster of `rank`
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void g_mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
      "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
        "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
        "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}

// Eight packed words -> 64 fp16 weights half_rn((n - z) * scale) in the order of K.  Byte i of a word holds codes 2i, 2i + 1: as the low
// bytes of two halves with exponent byte 0x64 and the other nibble masked off they are (1024 + n, 1024 + 16 n'), in the order the MMA
// wants them; one FMA with zc = (-(1024 + z), -(64 + z)) leaves the exact (n - z, n' - z), and the product with the scale (s2: twice)
// rounds once.  In three passes over all 32 registers: as one expression per register the launch of the 13B gate/up shape at 16 tokens
// executes 19.3 million instructions instead of 17.1 and takes 31.2 us instead of 29.3 (supposedly moves into the consecutive registers
// that tcgen05.st takes).
// SCALED false: the exact integers n - z.
template <bool SCALED = true>
__device__ __forceinline__ void dequant_words(uint32_t (&v)[32], const uint32_t (&w)[16], int first, uint32_t zc, uint32_t s2) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) v[4 * j + i] = prmt(w[first + j], 0x64646464u, 0x4040u + 0x0101u * i) & 0x64F0640Fu;
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = hfma2(v[j], 0x2C003C00u, zc);
  if (SCALED) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = hmul2(v[j], s2);
  }
}

}  // namespace glowq
