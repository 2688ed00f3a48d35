// RTN uint4 quantiser and packer: fp16 weights -> packed codes, zero points and scales in one pass over the weight.
//
// Same fp16 arithmetic as the pure-torch quantiser of cuda_w4a16/linear.py (every operation rounds to fp16):
//   scale = (max - min) / 15, zero = clamp(rint(-min / scale), 0, 15), code = clamp(rint(w / scale + zero), 0, 15)
// per (row, 128-column group); columns past IC count as zero; zero-point nibbles past the last group hold 8.
//
// Bound: HBM (2.6 bytes per weight).  A half warp holds one group in registers (16 lanes x 8 columns = one 16-byte load
// and one packed word per lane), a warp takes the eight groups of one zero-point word: four loads in flight per lane,
// the minimum and maximum travel as ONE half2 {-min, max} through four shuffles, and codes, scales and the zero word
// leave as whole segments.  The weight is read once and nothing intermediate is written (the torch expression is about
// thirty elementwise kernels).  Measured on B200: 13824 x 5120 in 66 us (2.8 TB/s), 5120 x 5120 in 29 us (2.4 TB/s): the
// arithmetic (two conversions, a quotient and a rounding per weight) is what is left above the copy's 28 us.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

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
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__global__ void __launch_bounds__(kQThreads) quantize_kernel(const __half* __restrict__ w, int32_t* __restrict__ qweight,
                                                             int32_t* __restrict__ qzeros, __half* __restrict__ scales, int OC,
                                                             int IC, int G, int words, long long w_stride, int vec_ok) {
  const int lane = threadIdx.x & 31, hsel = lane >> 4, s16 = lane & 15;
  const long long item = static_cast<long long>(blockIdx.x) * (kQThreads / 32) + (threadIdx.x >> 5);
  if (item >= static_cast<long long>(OC) * words) return;   // whole warps leave together
  const int row = static_cast<int>(item / words), zw_i = static_cast<int>(item - static_cast<long long>(row) * words);
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
  uint32_t zword = 0, my_scale = 0;
#pragma unroll
  for (int i = 0; i < kQIters; ++i) {
    const int g = zw_i * 8 + 2 * i + hsel;
    // {-min, max} of the group as one half2
    const uint32_t hi2 = hmax2_nan(hmax2_nan(v[i].x, v[i].y), hmax2_nan(v[i].z, v[i].w));
    constexpr uint32_t kSign = 0x80008000u;
    const uint32_t lo2 = hmax2_nan(hmax2_nan(v[i].x ^ kSign, v[i].y ^ kSign), hmax2_nan(v[i].z ^ kSign, v[i].w ^ kSign));
    uint32_t mm = hmax2_nan(prmt(lo2, hi2, 0x5410), prmt(lo2, hi2, 0x7632));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) mm = hmax2_nan(mm, __shfl_xor_sync(0xffffffffu, mm, o));
    const float2 mf = __half22float2(*reinterpret_cast<const __half2*>(&mm));   // {-min, max}
    const float diff = __half2float(__float2half_rn(mf.y + mf.x));
    // (the lower clamp of the scale, 1e-8, rounds to zero in fp16: it only turns -0 into +0)
    const uint32_t sbits = __half_as_ushort(__float2half_rn(__fdiv_rn(diff, 15.f))) & (diff == 0.f ? 0u : 0xFFFFu);
    const float sc = __half2float(__ushort_as_half(static_cast<unsigned short>(sbits)));
    const uint32_t zq = pack2(__fdiv_rn(mf.x, sc), 0.f);
    const uint32_t z = code_bits(zq) & 0xFu;
    zword |= (g < G ? z : 8u) << (4 * (2 * i + hsel));
    // w / scale rounded to fp32 and then to fp16, as the division of two halves is.  With r the correctly rounded
    // reciprocal, one residual step on w * r gives the correctly rounded quotient (Markstein, IBM J. Res. Dev. 34,
    // 1990); a scale of zero, infinity or NaN divides.
    // (the zero point that is added keeps a NaN, 0 / 0, although the stored one is 0)
    const uint32_t zh = (zq & 0x7FFFu) > 0x7C00u ? 0x7FFFu : static_cast<uint32_t>(__half_as_ushort(__uint2half_rn(z)));
    const uint32_t z2 = zh * 0x00010001u;
    const float r = __frcp_rn(sc);
    const bool plain = sbits != 0u && sbits < 0x7C00u;   // the same for the half warp's 16 lanes
    const uint32_t* vw = &v[i].x;
    uint32_t word = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(vw + e));
      uint32_t q;
      if (plain) {
        const float q0 = f.x * r, q1 = f.y * r;
        q = pack2(fmaf(fmaf(-q0, sc, f.x), r, q0), fmaf(fmaf(-q1, sc, f.y), r, q1));
      } else {
        q = pack2(__fdiv_rn(f.x, sc), __fdiv_rn(f.y, sc));
      }
      const uint32_t c = code_bits(hadd2(q, z2));          // bits 0..3: column 2e, bits 16..19: column 2e + 1
      word |= ((c & 0xFu) | ((c >> 12) & 0xF0u)) << (8 * e);
    }
    if (g < G) qweight[static_cast<size_t>(row) * (static_cast<size_t>(G) * 16) + g * 16 + s16] = static_cast<int32_t>(word);
    // lane l < 8 keeps the scale of group l of the word (group 2 i + h comes from half warp h)
    const uint32_t from = __shfl_sync(0xffffffffu, sbits, (lane & 1) * 16);
    if ((lane >> 1) == i) my_scale = from;
  }
  zword |= __shfl_xor_sync(0xffffffffu, zword, 16);
  if (lane == 0) qzeros[static_cast<size_t>(row) * words + zw_i] = static_cast<int32_t>(zword);
  const int gs = zw_i * 8 + lane;
  if (lane < 8 && gs < G) scales[static_cast<size_t>(row) * G + gs] = __ushort_as_half(static_cast<unsigned short>(my_scale));
}

}  // namespace

cudaError_t launch_quantize(const __half* w, int32_t* qweight, int32_t* qzeros, __half* scales, int OC, int IC,
                            long long w_stride, cudaStream_t stream) {
  const int G = (IC + 127) / 128, words = (G + 7) / 8;
  const long long items = static_cast<long long>(OC) * words;
  const long long blocks = (items + kQThreads / 32 - 1) / (kQThreads / 32);
  if (blocks > 0x7FFFFFFFll) return cudaErrorInvalidValue;
  const int vec_ok = (IC & 7) == 0 && (w_stride & 7) == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0;
  quantize_kernel<<<static_cast<unsigned>(blocks), kQThreads, 0, stream>>>(w, qweight, qzeros, scales, OC, IC, G, words, w_stride,
                                                                          vec_ok);
  return cudaGetLastError();
}

}  // namespace glowq
