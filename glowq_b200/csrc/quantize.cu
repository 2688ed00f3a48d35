// RTN uint4 quantiser and packer: fp16 weights -> packed codes, zero points and scales in one pass over the weight.
//
// Same fp16 arithmetic as the pure-torch quantiser of cuda_w4a16/linear.py (every operation rounds to fp16):
//   scale = (max - min) / 15, zero = clamp(rint(-min / scale), 0, 15), code = clamp(rint(w / scale + zero), 0, 15)
// per (row, 128-column group); columns past IC count as zero; zero-point nibbles past the last group hold 8.
//
// Bound: HBM (2.6 bytes per weight), then issue slots.  A half warp holds one group in registers (16 lanes x 8 columns = one 16-byte
// load and one packed word per lane), a warp takes the eight groups of one zero-point word: four loads in flight per lane, the minimum
// and maximum travel as ONE half2 {-min, max}, and codes, scales and the zero word leave as whole segments.  The weight is read once
// and nothing intermediate is written (the torch expression is about thirty elementwise kernels).
// A warp's eight groups are divided once, a group per quad of lanes, and the quotients of its weights are paired fp32 operations; with
// every half warp dividing for each of its four groups in turn, and for groups past the end of a row too, 13824 x 5120 took 64 us and
// 18944 x 3584 (28 groups) 89; now 42 (4.2 TB/s; a copy's 28) and 46.  5120 x 5120: 26 -> 18.  Six blocks an SM: a few bytes of spill
// in the path that divides, 43 us where five without took 45.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "common.cuh"

namespace glowq {
namespace {

constexpr int kQThreads = 256;
constexpr int kQIters = 4;      // passes of two groups: the eight groups of a zero-point word

__device__ __forceinline__ uint32_t hmax2_nan(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.NaN.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t hmin2_nan(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("min.NaN.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// rint(clamp(x, 0, 15)) in the low four bits of each half: 1024 + x rounds to an integer (the fp16 ulp is 1 there).  A
// NaN (0 / 0 of an all-zero group) becomes 0, as torch's conversion to uint8 has it.
__device__ __forceinline__ uint32_t code_bits(uint32_t x) {
  uint32_t r;
  asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(0u));
  asm("min.f16x2 %0, %1, %2;" : "=r"(r) : "r"(r), "r"(0x4B804B80u));
  return hadd2(r, 0x64006400u);
}
// code_bits(q + z) where neither is NaN: the sum as a fused multiply-add by one that takes the lower clamp along.
__device__ __forceinline__ uint32_t sum_code_bits(uint32_t q, uint32_t z) {
  uint32_t r;
  asm("fma.rn.relu.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(q), "r"(0x3C003C00u), "r"(z));
  asm("min.f16x2 %0, %1, %2;" : "=r"(r) : "r"(r), "r"(0x4B804B80u));
  return hadd2(r, 0x64006400u);
}
// Two products or fused multiply-adds in one instruction, each rounded like the single one.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__global__ void __launch_bounds__(kQThreads, 6) quantize_kernel(const __half* __restrict__ w, int32_t* __restrict__ qweight,
                                                             int32_t* __restrict__ qzeros, __half* __restrict__ scales, int OC,
                                                             int IC, int G, int words, long long w_stride, int vec_ok,
                                                             int64_t* __restrict__ gid) {
  const int lane = threadIdx.x & 31, hsel = lane >> 4, s16 = lane & 15;
  // (32 bits: the entry point refuses more than 2^32 - 8 items, so that the last block's eight fit as well)
  const uint32_t item = blockIdx.x * (kQThreads / 32) + (threadIdx.x >> 5);
  const uint32_t row_u = item / static_cast<uint32_t>(words);
  if (row_u >= static_cast<uint32_t>(OC)) return;   // whole warps leave together
  const int row = static_cast<int>(row_u), zw_i = static_cast<int>(item - row_u * static_cast<uint32_t>(words));
  const __half* wrow = w + static_cast<size_t>(row) * w_stride;
  uint4 v[kQIters];
#pragma unroll
  for (int i = 0; i < kQIters; ++i) {
    const int k = (zw_i * 8 + 2 * i + hsel) * 128 + s16 * 8;
    v[i] = make_uint4(0, 0, 0, 0);
    if (vec_ok) {                        // IC is a multiple of 8 and the rows are 16-byte aligned
      if (k < IC) v[i] = ldg_stream_v4(wrow + k);
    } else {
      __align__(16) __half t[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) t[e] = k + e < IC ? wrow[k + e] : __float2half(0.f);
      v[i] = *reinterpret_cast<const uint4*>(t);
    }
  }
  // {-min, max} of the eight groups as one half2 each: a half warp's four passes change places while they are reduced (five shuffles,
  // not sixteen), after which the four lanes of a quad hold one group, pass `mine` of their half warp.
  uint32_t mm[kQIters];
#pragma unroll
  for (int i = 0; i < kQIters; ++i) {
    const uint32_t hi2 = hmax2_nan(hmax2_nan(v[i].x, v[i].y), hmax2_nan(v[i].z, v[i].w));
    const uint32_t lo2 = hmin2_nan(hmin2_nan(v[i].x, v[i].y), hmin2_nan(v[i].z, v[i].w));
    mm[i] = hmax2_nan(prmt(lo2, hi2, 0x5410) ^ 0x8000u, prmt(lo2, hi2, 0x7632) ^ 0x8000u);
  }
  const bool b3 = lane & 8, b2 = lane & 4;
  const int mine = (b2 ? 2 : 0) + (b3 ? 1 : 0);
  const uint32_t m01 = hmax2_nan(b3 ? mm[1] : mm[0], __shfl_xor_sync(0xffffffffu, b3 ? mm[0] : mm[1], 8));
  const uint32_t m23 = hmax2_nan(b3 ? mm[3] : mm[2], __shfl_xor_sync(0xffffffffu, b3 ? mm[2] : mm[3], 8));
  uint32_t m = hmax2_nan(b2 ? m23 : m01, __shfl_xor_sync(0xffffffffu, b2 ? m01 : m23, 4));
  m = hmax2_nan(m, __shfl_xor_sync(0xffffffffu, m, 2));
  m = hmax2_nan(m, __shfl_xor_sync(0xffffffffu, m, 1));
  const int gl = 2 * mine + hsel, g_own = zw_i * 8 + gl;
  const float2 mf = __half22float2(*reinterpret_cast<const __half2*>(&m));   // {-min, max}
  const float diff = __half2float(__float2half_rn(mf.y + mf.x));
  // (the lower clamp of the scale, 1e-8, rounds to zero in fp16: it only turns -0 into +0)
  const uint32_t sbits = __half_as_ushort(__float2half_rn(__fdiv_rn(diff, 15.f))) & (diff == 0.f ? 0u : 0xFFFFu);
  const float sc_own = __half2float(__ushort_as_half(static_cast<unsigned short>(sbits)));
  const uint32_t zq = pack2(__fdiv_rn(mf.x, sc_own), 0.f);
  const uint32_t z = code_bits(zq) & 0xFu;
  // (the zero point that is added keeps a NaN, 0 / 0, although the stored one is 0)
  const uint32_t zh = (zq & 0x7FFFu) > 0x7C00u ? 0x7FFFu : static_cast<uint32_t>(__half_as_ushort(__uint2half_rn(z)));
  const uint32_t own = sbits | (zh << 16);
  const float r_own = __frcp_rn(sc_own);
  // w / scale rounded to fp32 and then to fp16, as the division of two halves is.  With r the correctly rounded
  // reciprocal, one residual step on w * r gives the correctly rounded quotient (Markstein, IBM J. Res. Dev. 34,
  // 1990); where a group's scale is zero, infinity or NaN the warp divides.  (Not for groups past the end, which are not stored.)
  const auto codes = [&](auto plain) {
#pragma unroll
    for (int i = 0; i < kQIters; ++i) {
      const int g = zw_i * 8 + 2 * i + hsel, from = hsel * 16 + (i & 1) * 8 + (i >> 1) * 4;
      const uint32_t sz = __shfl_sync(0xffffffffu, own, from);
      const float sc = __half2float(__ushort_as_half(static_cast<unsigned short>(sz & 0xFFFFu)));
      const uint32_t z2 = prmt(sz, sz, 0x3232);
      const uint32_t* vw = &v[i].x;
      uint32_t c[4];
      if constexpr (plain.value) {
        const float r = __shfl_sync(0xffffffffu, r_own, from);
        const float2 rr = make_float2(r, r), ss = make_float2(-sc, -sc);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(vw + e));
          const float2 q0 = mul2(f, rr), q1 = fma2(fma2(q0, ss, f), rr, q0);
          c[e] = sum_code_bits(pack2(q1.x, q1.y), z2);   // byte 0: column 2e, byte 2: column 2e + 1 (in its low four bits)
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(vw + e));
          c[e] = code_bits(hadd2(pack2(__fdiv_rn(f.x, sc), __fdiv_rn(f.y, sc)), z2));
        }
      }
      const uint32_t c01 = prmt(c[0], c[1], 0x6240), c23 = prmt(c[2], c[3], 0x6240);
      const uint32_t word = prmt(c01, c23, 0x5410) | (prmt(c01, c23, 0x7632) << 4);
      if (g < G) qweight[static_cast<size_t>(row) * (static_cast<size_t>(G) * 16) + g * 16 + s16] = static_cast<int32_t>(word);
    }
  };
  if (__all_sync(0xffffffffu, (sbits != 0u && sbits < 0x7C00u) || g_own >= G))
    codes(std::true_type{});
  else
    codes(std::false_type{});
  if (gid != nullptr && row == 0) {   // the module's group index of every column: a launch or two less than made on their own
    for (int k = zw_i * 1024 + lane; k < min(IC, zw_i * 1024 + 1024); k += 32) gid[k] = k >> 7;
  }
  const uint32_t zword = __reduce_or_sync(0xffffffffu, (g_own < G ? z : 8u) << (4 * gl));
  if (lane == 0) qzeros[static_cast<size_t>(row) * words + zw_i] = static_cast<int32_t>(zword);
  if ((lane & 3) == 0 && g_own < G) scales[static_cast<size_t>(row) * G + g_own] = __ushort_as_half(static_cast<unsigned short>(sbits));
}

}  // namespace

cudaError_t launch_quantize(const __half* w, int32_t* qweight, int32_t* qzeros, __half* scales, int64_t* gid, int OC, int IC,
                            long long w_stride, cudaStream_t stream) {
  const int G = (IC - 1) / 128 + 1, words = (G + 7) / 8;
  const long long items = static_cast<long long>(OC) * words;
  const long long blocks = (items + kQThreads / 32 - 1) / (kQThreads / 32);
  const int vec_ok = (IC & 7) == 0 && (w_stride & 7) == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0;
  quantize_kernel<<<static_cast<unsigned>(blocks), kQThreads, 0, stream>>>(w, qweight, qzeros, scales, OC, IC, G, words, w_stride,
                                                                          vec_ok, gid);
  return cudaGetLastError();
}

}  // namespace glowq
