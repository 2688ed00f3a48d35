// Corrected W4A16 product for decode batches (9 tokens and more) with the dequantised weights in TENSOR MEMORY.
//
//   D[128 output columns, N tokens] += W[128, 128 k] . X[N, 128 k]^T      (one quantisation group of K per step)
//
// The weights are the MMA's A operand: the dequant warps turn packed rows into half_rn((code - zero) * scale) in registers
// and write them to tensor memory (tcgen05.st), the activations are the B operand by TMA, the accumulator is D^T in tensor
// memory.  What bounds the form with the weights as a shared-memory operand is shared-memory bandwidth: the fp16 tile is
// written and read back (and a 128-row activation tile read, however few tokens there are) for 4 bits of weight, about
// 900 clocks per 8 KB of packed weights.  Here only the packed bytes and N token rows pass through shared memory.
//   warp 0   activation producer (one thread): TMA of N x 128 activations per step; in the correction steps (64 columns of the
//            rank each) N x 64 of r and the 128 x 64 tile of L, both fp16 shared-memory operands.
//   warp 2   packed-weight producer (one thread): TMA of 128 rows x 64 B per step, running ahead of everything.
//   warp 1   allocates tensor memory and issues tcgen05.mma (A from tensor memory; from shared memory in the correction
//            steps) and the commits that release the stages.
//   warps 3. dequantise in TEAMS of four warps that take alternate steps - a thread owns one weight row, which is its
//            tensor-memory lane - and are the epilogue afterwards: lane = output column, so a token's 32 outputs of a
//            warp are one contiguous store.
// Small token tiles (N <= 64) run two CTAs per SM (256 tensor-memory columns each) with two teams, so that one CTA's
// prologue and epilogue hide behind the other's steps; larger ones one CTA with four teams, as a CTA PAIR (cta_group::2)
// that computes 256 output columns x N tokens, each CTA holding half of the activation rows.
// K may be sliced over CTAs; the CTA that completes a tile's count adds the fp32 slots in slice order (deterministic).
// Every mbarrier wait is bounded; on expiry a status word is set and the CTA drains and frees its tensor memory.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "../../include/glowq_w4a16.h"
#include "common.cuh"
#include "params.h"
#include "tcgen05.cuh"

namespace glowq {

int tensor_map_2d_ex(CUtensorMap* out, CUtensorMapDataType dtype, const void* ptr, uint64_t dim0, uint64_t dim1,
                     uint64_t stride_bytes, uint32_t box0, uint32_t box1, int swizzle);

namespace {

constexpr int kRows = 128;                    // weight rows (output columns) per CTA
constexpr int kPStage = kRows * 64;           // packed stage: 128 rows x 128 codes
constexpr int kA16 = kRows * 128;             // fp16 tile of a correction step: 128 rows x 64 columns
constexpr int kMaxS = 8, kMaxP = 8;
constexpr int kA16Slots = 2;

struct TsMember {
  const __half* scales;
  const int32_t* qzeros;
  const __half* bias;
  void* out;
  int OC, nu, sstride, zstride, out_stride, lr_separate, out_vec_ok, tile_begin;
  float alpha;
};
struct TsParams {
  uint32_t* status;
  uint32_t* tile_ctr;   // arrivals of a sliced tile's K slices, zero between launches
  float* slots;         // [ksplit][sliced tile][token][128] fp32
  int M, G, out_fp32, n_members;
  int N;                // tokens per tile (multiple of 16)
  int ns, np;           // ring depths: stages (an activation tile and a tensor-memory A tile each), packed weights
  int a_col;            // first tensor-memory column of the A tiles
  int ksplit, full_tiles, n_tail, n_x;   // items: full_tiles whole tiles, then n_tail tiles of ksplit K slices each
  TsMember mem[kMaxMembers];
};
struct alignas(64) TsMaps {
  CUtensorMap x, r;
  CUtensorMap w[kMaxMembers], l[kMaxMembers];
};

template <int TEAMS>
struct TsCfg {
  static constexpr int kDequantWarps = 4 * TEAMS;
  static constexpr int kCtrlWarps = 3;
  static constexpr int kThreads = 32 * (kCtrlWarps + kDequantWarps);
  static constexpr int kCtas = TEAMS == 2 ? 2 : 1;            // per SM
  static constexpr int kTmemCols = TEAMS == 2 ? 256 : 512;
  static constexpr int kSmem = TEAMS == 2 ? 112 * 1024 : 226 * 1024;
};

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
      "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

// The MMAs of one step and the commit that releases its stage, issued by one elected lane of a converged warp.  The whole
// warp runs the issuing loop, and the step is one block, so that descriptors and addresses stay in uniform registers,
// which these instructions read: a loop under `lane == 0` moves every operand of every MMA over first (the gate/up launch
// of the 13B shapes at 16 tokens: 38.6 us so, 34.4 with an elected lane per MMA, 33.0 with the step as one block).
// `bar`, `peer`: released in this CTA and, in a pair, in the other one.  b_lo / b_hi: descriptor words of the activation
// tile, whose second 64 columns lie `sub16` further; accumulate 0: the first MMA overwrites D.
#define GLOWQ_TS_MMA(CG, A, B, P) "@e tcgen05.mma.cta_group::" CG ".kind::f16 [%0], " A ", " B ", %5, " P ";\n\t"
#define GLOWQ_TS_COMMIT(CG, R) "@e tcgen05.commit.cta_group::" CG ".mbarrier::arrive::one.shared::cluster.b64 [" R "];\n\t"
#define GLOWQ_TS_STEP(CG, LAST)                                                                                              \
  "{\n\t.reg .pred e, p, t;\n\t.reg .b32 a<8>, l<8>;\n\t.reg .b64 b<8>;\n\t"                                                 \
  "setp.ne.b32 p, %6, 0;\n\tsetp.eq.b32 t, 0, 0;\n\telect.sync _|e, 0xffffffff;\n\t"                                         \
  "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\tadd.u32 a4, %1, 32;\n\tadd.u32 a5, %1, 40;\n\t"       \
  "add.u32 a6, %1, 48;\n\tadd.u32 a7, %1, 56;\n\tadd.u32 l1, %2, 2;\n\tadd.u32 l2, %2, 4;\n\tadd.u32 l3, %2, 6;\n\t"         \
  "add.u32 l4, %2, %4;\n\tadd.u32 l5, l4, 2;\n\tadd.u32 l6, l4, 4;\n\tadd.u32 l7, l4, 6;\n\t"                                \
  "mov.b64 b0, {%2, %3};\n\tmov.b64 b1, {l1, %3};\n\tmov.b64 b2, {l2, %3};\n\tmov.b64 b3, {l3, %3};\n\t"                     \
  "mov.b64 b4, {l4, %3};\n\tmov.b64 b5, {l5, %3};\n\tmov.b64 b6, {l6, %3};\n\tmov.b64 b7, {l7, %3};\n\t"                     \
  GLOWQ_TS_MMA(CG, "[%1]", "b0", "p") GLOWQ_TS_MMA(CG, "[a1]", "b1", "t") GLOWQ_TS_MMA(CG, "[a2]", "b2", "t")                \
  GLOWQ_TS_MMA(CG, "[a3]", "b3", "t") GLOWQ_TS_MMA(CG, "[a4]", "b4", "t") GLOWQ_TS_MMA(CG, "[a5]", "b5", "t")                \
  GLOWQ_TS_MMA(CG, "[a6]", "b6", "t") GLOWQ_TS_MMA(CG, "[a7]", "b7", "t") LAST "}"
template <bool PAIR>
__device__ __forceinline__ void umma_ts_step(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, uint32_t sub16, uint32_t idesc,
                                             uint32_t accumulate, uint32_t bar, uint32_t peer) {
  if constexpr (PAIR)
    asm volatile(GLOWQ_TS_STEP("2", GLOWQ_TS_COMMIT("2", "%7") GLOWQ_TS_COMMIT("2", "%8"))::"r"(d), "r"(a), "r"(b_lo), "r"(b_hi),
                 "r"(sub16), "r"(idesc), "r"(accumulate), "r"(bar), "r"(peer)
                 : "memory");
  else
    asm volatile(GLOWQ_TS_STEP("1", GLOWQ_TS_COMMIT("1", "%7"))::"r"(d), "r"(a), "r"(b_lo), "r"(b_hi), "r"(sub16), "r"(idesc),
                 "r"(accumulate), "r"(bar)
                 : "memory");
}
// One 16-column MMA with both operands in shared memory (correction steps).
template <bool PAIR>
__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (PAIR)
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void umma_commit_elect(uint32_t bar) {
  if constexpr (PAIR)
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t" GLOWQ_TS_COMMIT("2", "%0") "}" ::"r"(bar) : "memory");
  else
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t" GLOWQ_TS_COMMIT("1", "%0") "}" ::"r"(bar) : "memory");
}
// A poll that does not block (mbarrier.try_wait may suspend the thread while the phase is open).
template <bool CLUSTER>
__device__ __forceinline__ bool test_bar(uint32_t a, uint32_t parity) {   // CLUSTER: arrivals come from the peer CTA too
  uint32_t ok;
  if constexpr (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(a), "r"(parity)
                 : "memory");
  return ok != 0;
}
__device__ __forceinline__ void arrive_release_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// One ring position: index and phase parity (by <= depth).
struct Ring {
  uint32_t i, ph;
  __device__ __forceinline__ void step(uint32_t by, uint32_t depth) {
    i += by;
    if (i >= depth) {
      i -= depth;
      ph ^= 1;
    }
  }
};

template <int TEAMS, bool PAIR>
__global__ void __launch_bounds__(TsCfg<TEAMS>::kThreads, TsCfg<TEAMS>::kCtas)
gemm_tmem_kernel(const __grid_constant__ TsParams p, const __grid_constant__ TsMaps tm) {
  using C = TsCfg<TEAMS>;
  constexpr int kCG = PAIR ? 2 : 1;
  extern __shared__ unsigned char smem[];
  __shared__ int s_abort;
  __shared__ uint32_t s_tmem_base, s_last;
  const uint32_t smem0 = (sm_u32(smem) + 1023u) & ~1023u;
  // barriers in the first 1 KB.  full: a stage's A tile is in tensor memory and its activations have landed (ONE barrier
  // for the issuing warp to poll per step: the dequant warps, the copies' bytes and, in a pair, the peer's relay);
  // land: the peer's own copies; cfull / cempty: the fp16 tiles of the correction steps.
  const uint32_t full = smem0, empty = smem0 + 64, land = smem0 + 128, pfull = smem0 + 192, pempty = smem0 + 256,
                 cfull = smem0 + 320, cempty = smem0 + 336, accum = smem0 + 352;
  const int NB = p.N / kCG;                                  // activation rows this CTA holds
  const uint32_t sub = static_cast<uint32_t>(NB) * 128;      // one 64-column half of an activation tile
  const uint32_t a16 = smem0 + 1024, ring = a16 + kA16Slots * kA16, pring = ring + p.ns * 2 * sub;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t crank = PAIR ? cluster_ctarank() : 0u;

  const int item = static_cast<int>(blockIdx.x) / kCG;
  int tile_lin = item, zslice = 0, ks = 1;
  if (item >= p.full_tiles) {
    const int r = item - p.full_tiles, t = r / p.ksplit;
    tile_lin = p.full_tiles + t;
    zslice = r - t * p.ksplit;
    ks = p.ksplit;
  }
  const int by = tile_lin / p.n_x, bx = tile_lin - by * p.n_x;
  int mi = 0;
#pragma unroll
  for (int i = 1; i < kMaxMembers; ++i)
    if (i < p.n_members && bx >= p.mem[i].tile_begin) mi = i;
  const TsMember& mb = p.mem[mi];
  const int n0 = (bx - mb.tile_begin) * (kRows * kCG) + static_cast<int>(crank) * kRows;
  const int m0 = by * p.N;
  const int nk_all = p.G + mb.nu;
  const int it0 = ks > 1 ? static_cast<int>(static_cast<long long>(nk_all) * zslice / ks) : 0;
  const int nk = ks > 1 ? static_cast<int>(static_cast<long long>(nk_all) * (zslice + 1) / ks) : nk_all;
  const int nkp = max(it0, min(nk, p.G));    // steps [it0, nkp) are packed weights, [nkp, nk) the correction

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < p.ns; ++i) {
      g_mbar_init(full + 8 * i, 4 * kCG + 1 + (PAIR ? 1 : 0));
      g_mbar_init(empty + 8 * i, 1);
      g_mbar_init(land + 8 * i, 1);
    }
    for (int i = 0; i < p.np; ++i) {
      g_mbar_init(pfull + 8 * i, 1);
      g_mbar_init(pempty + 8 * i, 4);
    }
    for (int i = 0; i < kA16Slots; ++i) {
      g_mbar_init(cfull + 8 * i, PAIR && crank == 0 ? 2 : 1);
      g_mbar_init(cempty + 8 * i, 1);
    }
    g_mbar_init(accum, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sm_u32(&s_tmem_base)),
                   "r"(C::kTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sm_u32(&s_tmem_base)),
                   "r"(C::kTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR) cluster_sync_all();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // Only now: a CTA of the next kernel that shares this SM must not take the tensor memory this one still asks for.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem = s_tmem_base;
  volatile int* abort_flag = &s_abort;
  auto drain = [&](uint32_t bars, int depth, int issued) {   // after a failed wait: let copies in flight land (bounded)
    for (int j = (issued > depth ? issued - depth : 0); j < issued; ++j) {
      uint32_t spins = 0;
      while (!g_mbar_try_once(bars + 8 * (j % depth), (j / depth) & 1) && ++spins < kGemmSpin) {
      }
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      Ring b{0, 0}, c{0, 0};
      int issued = 0, cissued = 0;
      bool ok = true;
      const int tok0 = m0 + static_cast<int>(crank) * NB;
      const uint32_t landed = PAIR && crank != 0 ? land : full;
      asm volatile("griddepcontrol.wait;" ::: "memory");   // activations and r come from the kernels before
      for (int it = it0; it < nk; ++it) {
        if (!(ok = g_mbar_wait(empty + 8 * b.i, b.ph ^ 1, abort_flag, p.status))) break;
        const uint32_t dst = ring + b.i * 2 * sub;
        if (it < nkp) {
          const uint32_t bar = landed + 8 * b.i;
          g_mbar_expect_tx(bar, 2 * sub);
          g_tma_2d(dst, &tm.x, it * 128, tok0, bar);
          g_tma_2d(dst + sub, &tm.x, it * 128 + 64, tok0, bar);
          ++issued;
        } else {
          if (!(ok = g_mbar_wait(cempty + 8 * c.i, c.ph ^ 1, abort_flag, p.status))) break;
          const uint32_t bar = cfull + 8 * c.i;
          g_mbar_expect_tx(bar, sub + kA16);
          g_tma_2d(dst, &tm.r, (it - p.G) * 64, tok0, bar);
          g_tma_2d(a16 + c.i * kA16, &tm.l[mi], (it - p.G) * 64, n0, bar);
          ++cissued;
          c.step(1, kA16Slots);
        }
        b.step(1, p.ns);
      }
      if (!ok) {
        drain(landed, p.ns, issued);
        drain(cfull, kA16Slots, cissued);
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    if (lane == 0) {
      Ring s{0, 0};
      int issued = 0;
      bool ok = true;
      for (int it = it0; it < nkp; ++it) {
        if (!(ok = g_mbar_wait(pempty + 8 * s.i, s.ph ^ 1, abort_flag, p.status))) break;
        g_mbar_expect_tx(pfull + 8 * s.i, kPStage);
        g_tma_2d(pring + s.i * kPStage, &tm.w[mi], it * 16, n0, pfull + 8 * s.i);
        ++issued;
        s.step(1, p.np);
      }
      if (!ok) drain(pfull, p.np, issued);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (crank == 0) {   // the whole warp: see umma_ts_step
      Ring b{0, 0}, c{0, 0};
      // instruction descriptor: fp32 accumulate, fp16 operands, K-major, M = 128 (256 over a pair), N tokens
      const uint32_t idesc = (1u << 4) | ((static_cast<uint32_t>(p.N) >> 3) << 17) | (static_cast<uint32_t>(kRows * kCG >> 4) << 24);
      const uint64_t desc0 = smem_desc_sw128(ring), desc_a0 = smem_desc_sw128(a16);
      const uint32_t hi = static_cast<uint32_t>(desc0 >> 32), lo0 = static_cast<uint32_t>(desc0);
      const uint32_t a_lo0 = static_cast<uint32_t>(desc_a0);
      const uint32_t pe = PAIR ? 1u : 0u;
      const uint32_t peer_empty = map_to_cta(empty, pe), peer_cempty = map_to_cta(cempty, pe), peer_accum = map_to_cta(accum, pe);
      auto commit = [&](uint32_t own, uint32_t peer) {
        umma_commit_elect<PAIR>(own);
        if (PAIR) umma_commit_elect<PAIR>(peer);
      };
      // After a failed wait the MMAs go on without waiting (their results are void, the status word is set): every
      // stage is still released, and the warp stays converged for the elections.
      bool ok = true;
      auto wait_slow = [&](uint32_t bar, uint32_t ph) {
        if (lane == 0)   // (one lane: a wait that the whole warp executes is 32 barrier operations)
          ok = ok && (PAIR ? g_mbar_wait_cluster(bar, ph, abort_flag, p.status) : g_mbar_wait(bar, ph, abort_flag, p.status));
        __syncwarp();
      };
      uint32_t acc = 0;
      bool ready = false;   // lane 0's poll
      for (int it = it0; it < nkp; ++it) {
        if (!__any_sync(0xffffffffu, ready)) wait_slow(full + 8 * b.i, b.ph);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t cur = b.i;
        b.step(1, p.ns);
        if (lane == 0) ready = test_bar<PAIR>(full + 8 * b.i, b.ph);   // answered while this stage's MMAs are issued
        __syncwarp();
        umma_ts_step<PAIR>(tmem, tmem + p.a_col + cur * 64, lo0 + cur * ((2 * sub) >> 4), hi, sub >> 4, idesc, acc, empty + 8 * cur,
                           peer_empty + 8 * cur);
        acc = 1;
      }
      if (mb.lr_separate) acc = 0;   // the first MMA overwrites its accumulator
      const uint32_t d = tmem + (mb.lr_separate ? p.N : 0);
      for (int it = nkp; it < nk; ++it) {
        wait_slow(cfull + 8 * c.i, c.ph);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t lo = lo0 + b.i * ((2 * sub) >> 4), la = a_lo0 + c.i * (kA16 >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          umma_ss<PAIR>(d, mk64(la + k * 2, hi), mk64(lo + k * 2, hi), idesc, acc);
          acc = 1;
        }
        commit(cempty + 8 * c.i, peer_cempty + 8 * c.i);
        commit(empty + 8 * b.i, peer_empty + 8 * b.i);
        c.step(1, kA16Slots);
        b.step(1, p.ns);
      }
      commit(accum, peer_accum);
    }
    if (PAIR && lane == 0 && crank == 1) {   // relay: this CTA's copies of a stage have landed
      const uint32_t full0 = map_to_cta(full, 0), cfull0 = map_to_cta(cfull, 0);
      Ring b{0, 0}, c{0, 0};
      bool ok = true;
      for (int it = it0; it < nk; ++it) {
        if (it < nkp) {
          ok = ok && g_mbar_wait(land + 8 * b.i, b.ph, abort_flag, p.status);
          arrive_release_cluster(full0 + 8 * b.i);
          b.step(1, p.ns);
        } else {
          ok = ok && g_mbar_wait(cfull + 8 * c.i, c.ph, abort_flag, p.status);
          arrive_release_cluster(cfull0 + 8 * c.i);
          c.step(1, kA16Slots);
        }
      }
    }
    __syncwarp();
  } else {
    // ================================================================ dequant warps, then epilogue
    const int dw = warp - C::kCtrlWarps, team = dw >> 2, q = warp & 3;   // q: the tensor-memory lanes this warp reaches
    const int rloc = q * 32 + lane, row = n0 + rloc;
    const bool rvalid = row < mb.OC;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16);
    bool ok = true;
    {
      const __half* srow = mb.scales + static_cast<size_t>(rvalid ? row : 0) * mb.sstride;
      const int32_t* zrow = mb.qzeros + static_cast<size_t>(rvalid ? row : 0) * mb.zstride;
      const uint32_t prow = static_cast<uint32_t>(rloc) * 64, psw = (static_cast<uint32_t>(rloc) >> 1) & 3u;
      const uint32_t full0 = PAIR ? map_to_cta(full, 0) : full;
      Ring a{0, 0}, s{0, 0};
      a.step(team, p.ns);
      s.step(team, p.np);
      uint32_t nx_s = 0, nx_z = 0;
      auto fetch = [&](int g) {   // rows past the end multiply by zero
        nx_s = nx_z = 0;
        if (rvalid && g < nkp) {
          nx_s = __half_as_ushort(__ldg(srow + g));
          nx_z = (static_cast<uint32_t>(__ldg(zrow + (g >> 3))) >> ((g & 7) * 4)) & 0xFu;
        }
      };
      fetch(it0 + team);
      for (int it = it0 + team; it < nkp; it += TEAMS) {
        const uint32_t s2 = nx_s * 0x00010001u;
        // -(1024 + z) and -(64 + z): the fp16 ulp is 1 at 1024 and 1/16 at 64
        const uint32_t zc = 0xD400E400u | (nx_z * 0x00100001u);
        // both polls go out together (an answer takes about a hundred clocks); after a failed wait the stores go on:
        // tensor memory is held to the end and the status word is set
        const bool have_p = test_bar<false>(pfull + 8 * s.i, s.ph), have_e = test_bar<false>(empty + 8 * a.i, a.ph ^ 1);
        if (!have_p) ok = ok && g_mbar_wait(pfull + 8 * s.i, s.ph, abort_flag, p.status);
        __syncwarp();
        fetch(it + TEAMS);
        const uint32_t src = pring + s.i * kPStage + prow;
        const uint32_t dst = lane_base + p.a_col + a.i * 64;
        uint32_t w[16];
#pragma unroll
        for (int j = 0; j < 4; ++j)   // (the box lands with its 16-byte chunks XORed within 64 bytes: no bank conflicts)
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(w[4 * j]), "=r"(w[4 * j + 1]), "=r"(w[4 * j + 2]), "=r"(w[4 * j + 3])
                       : "r"(src + ((static_cast<uint32_t>(j) ^ psw) << 4)));
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t v[32];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            // byte i of the word holds codes 2i, 2i + 1: as the low bytes of two halves with exponent byte 0x64 and the
            // other nibble masked off they are (1024 + n, 1024 + 16 n'), in the order the MMA wants them; one FMA leaves
            // the exact (n - z, n' - z) and the product with the scale rounds once
#pragma unroll
            for (int i = 0; i < 4; ++i)
              v[4 * j + i] = hmul2(hfma2(prmt(w[8 * half + j], 0x64646464u, 0x4040u + 0x0101u * i) & 0x64F0640Fu, 0x2C003C00u, zc), s2);
          }
          if (half == 0) {   // the MMAs that read this stage's A tile before are done
            if (!have_e) ok = ok && g_mbar_wait(empty + 8 * a.i, a.ph ^ 1, abort_flag, p.status);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          tmem_st32(dst + half * 32, v);
          if (half == 0 && lane == 0) g_mbar_arrive(pempty + 8 * s.i);   // the packed rows are in registers
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if (PAIR)
            arrive_release_cluster(full0 + 8 * a.i);
          else
            g_mbar_arrive(full + 8 * a.i);
        }
        a.step(TEAMS, p.ns);
        s.step(TEAMS, p.np);
      }
    }

    // ---- epilogue
    if (lane == 0) ok = ok && g_mbar_wait(accum, 0, abort_flag, p.status);
    ok = __all_sync(0xffffffffu, ok);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // With a separate correction accumulator, a K slice that lies wholly in one phase never writes the other's.
    const bool sep = mb.lr_separate != 0, has_main = it0 < p.G || !sep, has_lr = sep && nk > p.G;
    const int ntok = min(p.N, p.M - m0);
    const size_t slot_floats = static_cast<size_t>(p.N) * kRows;
    const int sl_tile = (tile_lin - p.full_tiles) * kCG + static_cast<int>(crank);
    float* slot = p.slots + (static_cast<size_t>(zslice) * (p.n_tail * kCG) + sl_tile) * slot_floats + rloc;
    const float bias = (rvalid && mb.bias) ? __half2float(mb.bias[row]) : 0.f;
    for (int t0 = team * 16; t0 < ntok; t0 += 16 * TEAMS) {
      uint32_t acc[16], lr[16];
      tmem_ld16(lane_base + t0, acc);
      if (sep) tmem_ld16(lane_base + p.N + t0, lr);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (!ok) continue;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (t0 + j < ntok) {
          float v = has_main ? __uint_as_float(acc[j]) : 0.f;
          if (has_lr) v = fmaf(mb.alpha, __uint_as_float(lr[j]), v);
          if (ks > 1) {
            __stcg(slot + static_cast<size_t>(t0 + j) * kRows, v);
          } else if (rvalid) {
            const size_t idx = static_cast<size_t>(m0 + t0 + j) * mb.out_stride + row;
            if (p.out_fp32)
              static_cast<float*>(mb.out)[idx] = v + bias;
            else
              static_cast<__half*>(mb.out)[idx] = __float2half_rn(v + bias);
          }
        }
      }
    }
    if (ks > 1) {
      // the CTA that completes the tile's count adds the slots in slice order
      asm volatile("bar.sync 1, %0;" ::"n"(C::kDequantWarps * 32) : "memory");
      const int et = threadIdx.x - 32 * C::kCtrlWarps;
      if (et == 0) {
        __threadfence();   // (cumulative over the CTA's stores, which the barrier ordered before it)
        uint32_t* ctr = p.tile_ctr + sl_tile;
        const bool last = atomicAdd(ctr, 1u) == static_cast<uint32_t>(ks - 1);
        if (last) {
          *ctr = 0u;
          __threadfence();
        }
        s_last = last ? 1u : 0u;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(C::kDequantWarps * 32) : "memory");
      if (s_last != 0u) {
        const float* base = p.slots + static_cast<size_t>(sl_tile) * slot_floats;
        const size_t zs = static_cast<size_t>(p.n_tail) * kCG * slot_floats;
        for (int i = et; i < ntok * (kRows / 4); i += C::kDequantWarps * 32) {
          const int tok = i >> 5, c4 = (i & 31) * 4, col = n0 + c4;
          const float* src = base + static_cast<size_t>(tok) * kRows + c4;
          float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int z0 = 0; z0 < ks; z0 += 4) {
            float4 u[4];
#pragma unroll
            for (int z = 0; z < 4; ++z)
              u[z] = z0 + z < ks ? __ldcg(reinterpret_cast<const float4*>(src + (z0 + z) * zs)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int z = 0; z < 4; ++z) {
              s.x += u[z].x;
              s.y += u[z].y;
              s.z += u[z].z;
              s.w += u[z].w;
            }
          }
          float v[4] = {s.x, s.y, s.z, s.w};
          if (mb.bias) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col + j < mb.OC) v[j] += __half2float(mb.bias[col + j]);
          }
          const size_t idx = static_cast<size_t>(m0 + tok) * mb.out_stride + col;
          if (mb.out_vec_ok && col + 4 <= mb.OC) {
            if (p.out_fp32) {
              *reinterpret_cast<float4*>(static_cast<float*>(mb.out) + idx) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
              const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
              *reinterpret_cast<uint2*>(static_cast<__half*>(mb.out) + idx) =
                  make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col + j < mb.OC) {
                if (p.out_fp32)
                  static_cast<float*>(mb.out)[idx + j] = v[j];
                else
                  static_cast<__half*>(mb.out)[idx + j] = __float2half_rn(v[j]);
              }
          }
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR) cluster_sync_all();  // neither CTA retires while the other's MMAs or arrivals may still touch it
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::kTmemCols) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::kTmemCols) : "memory");
  }
}

inline int cdiv(int a, int b) { return (a + b - 1) / b; }
inline bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool pdl_enabled() {
  static const bool on = [] {
    const char* v = std::getenv("GLOWQ_PDL");
    return !(v && v[0] == '0');
  }();
  return on;
}

template <int TEAMS, bool PAIR>
cudaError_t launch(const TsParams& p, const TsMaps& tm, int items, cudaStream_t stream) {
  using C = TsCfg<TEAMS>;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tmem_kernel<TEAMS, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem);
    if (e != cudaSuccess) return e;
    attr_done[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(items * (PAIR ? 2 : 1), 1, 1);
  cfg.blockDim = dim3(C::kThreads, 1, 1);
  cfg.dynamicSmemBytes = C::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (PAIR) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = 2;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, gemm_tmem_kernel<TEAMS, PAIR>, p, tm);
}

int env_or(const char* name, int dflt) {
  const char* v = std::getenv(name);
  return (v && *v) ? std::atoi(v) : dflt;
}

}  // namespace

// Members' products and corrections of a group call (r is in g.r_buf).  `slots` .. `slots + slot_bytes`: scratch for K
// slices; `tile_ctr`: n_ctr zeroed counters.
int gemm_tmem_forward(const glowq_w4a16_group_t& g, bool any_corr, bool any_separate, uint32_t* status, uint32_t* tile_ctr,
                      int n_ctr, float* slots, size_t slot_bytes, int sms, cudaStream_t stream, cudaError_t* cuda_err) {
  static const int env_f = env_or("GLOWQ_TS_F", -1), env_ks = env_or("GLOWQ_TS_KS", 0);   // tuning overrides
  const int G = cdiv(g.IC, kGroup);
  // tokens per tile: equal tiles of at most n_max tokens (a correction with its own accumulator doubles the columns)
  const int n_y = cdiv(g.M, any_separate ? 128 : 256);
  TsParams p{};
  p.N = cdiv(cdiv(g.M, n_y), 16) * 16;
  const bool two = p.N <= 64;            // two CTAs per SM
  const bool pair = !two;
  const int cg = pair ? 2 : 1, nb_rows = p.N / cg;
  const int d_cols = any_separate ? 2 * p.N : p.N;
  const int cols = two ? 256 : 512;
  {
    // stages: what tensor memory leaves beside the accumulators, as far as shared memory holds them and a few packed tiles
    const int smem = (two ? TsCfg<2>::kSmem : TsCfg<4>::kSmem) - 2048 - kA16Slots * kA16, bst = nb_rows * 256;
    p.ns = std::min({kMaxS, (cols - d_cols) / 64, (smem - (two ? 3 : 4) * kPStage) / bst});
    p.np = std::min(kMaxP, (smem - p.ns * bst) / kPStage);
    p.a_col = cols - p.ns * 64;
  }
  p.status = status;
  p.tile_ctr = tile_ctr;
  p.slots = slots;
  p.M = g.M;
  p.G = G;
  p.out_fp32 = g.out_dtype == GLOWQ_OUT_F32;
  p.n_members = g.n_members;
  TsMaps tm;
  std::memset(&tm, 0, sizeof(tm));
  int rc;
  if ((rc = tensor_map_2d_ex(&tm.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.x, g.IC, g.M, static_cast<uint64_t>(g.x_stride) * 2, 64,
                             nb_rows, 1)))
    return rc;
  tm.r = tm.x;
  if (any_corr && (rc = tensor_map_2d_ex(&tm.r, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.r_buf, g.rank, g.M,
                                         static_cast<uint64_t>(g.rank) * 2, 64, nb_rows, 1)))
    return rc;
  int n_x = 0, nu = 0;
  for (int i = 0; i < g.n_members; ++i) {
    const auto& m = g.members[i];
    const bool corr = any_corr && m.L && m.alpha != 0.f;
    if ((rc = tensor_map_2d_ex(&tm.w[i], CU_TENSOR_MAP_DATA_TYPE_INT32, m.qweight, static_cast<uint64_t>(G) * 16, m.OC,
                               static_cast<uint64_t>(m.weight_stride_i32) * 4, 16, kRows, 3)))
      return rc;
    tm.l[i] = tm.w[i];
    if (corr && (rc = tensor_map_2d_ex(&tm.l[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, m.L, g.rank, m.OC,
                                       static_cast<uint64_t>(m.L_stride) * 2, 64, kRows, 1)))
      return rc;
    TsMember& d = p.mem[i];
    d.scales = static_cast<const __half*>(m.scales);
    d.qzeros = m.qzeros;
    d.bias = static_cast<const __half*>(m.bias);
    d.out = m.out;
    d.OC = m.OC;
    d.nu = corr ? cdiv(g.rank, 64) : 0;
    nu = std::max(nu, d.nu);
    d.sstride = m.scale_stride;
    d.zstride = m.zero_stride_i32;
    d.out_stride = m.out_stride;
    d.alpha = m.alpha;
    d.lr_separate = corr && m.alpha != 1.f;
    d.out_vec_ok = al16(m.out) && (static_cast<size_t>(m.out_stride) * (p.out_fp32 ? 4 : 2)) % 16 == 0;
    d.tile_begin = n_x;
    n_x += cdiv(m.OC, kRows * cg);
  }
  p.n_x = n_x;
  const int total = n_x * n_y, units = sms / cg, resident = (two ? 2 * sms : sms) / cg;   // work items per SM (pair), resident at once
  const size_t item_bytes = static_cast<size_t>(cg) * p.N * kRows * 4;
  // Work partition: f rounds of whole tiles, the rest cut into ks slices of K.  Cost in microseconds, fitted on B200: an
  // SM takes 0.33 per step while two CTAs share it (0.5 alone; one CTA per SM: 1.0), 2.5 per wave of items for prologue
  // and epilogue, and the slices of a tile are added through memory.  Measured at 16 tokens on the 13B shapes: q/k/v
  // 31.5 us whole, 21.7 in two slices, 28.0 in four; o_proj 24.8 / 17.5 / 13.3, 12.7 in six; gate/up 35.5 whole, 41.4 in two
  // slices, 33.8 with one round whole and the other 68 tiles in two slices.
  p.full_tiles = total;
  p.n_tail = 0;
  p.ksplit = 1;
  const int nk = G + nu;
  double best = 1e30;
  for (int f = 0; f <= total / units; ++f) {
    if (env_f >= 0 && f != env_f) continue;
    const int full = f * units, tail = total - full;
    for (int ks = 1; ks <= 16 && (ks == 1 || ks * 4 <= nk); ++ks) {
      if (env_ks > 0 && ks != env_ks) continue;
      if (ks > 1 && (tail == 0 || tail * cg > n_ctr || static_cast<size_t>(tail) * ks * item_bytes > slot_bytes)) break;
      const int items = full + tail * ks;
      const double load = static_cast<double>(f) * nk + static_cast<double>(cdiv(tail * ks, units)) * nk / ks;
      const double cost = load * (two ? (items > units ? 0.33 : 0.5) : 1.0) + 2.5 * cdiv(items, resident) +
                          (ks > 1 ? 1.5 + 0.006 * p.N * ks : 0.0);
      if (cost < best) {
        best = cost;
        p.ksplit = ks;
        p.full_tiles = ks > 1 ? full : total;
        p.n_tail = ks > 1 ? tail : 0;
      }
    }
  }
  const int items = p.full_tiles + p.n_tail * p.ksplit;
  const cudaError_t e = two ? launch<2, false>(p, tm, items, stream) : launch<4, true>(p, tm, items, stream);
  if (e != cudaSuccess) {
    *cuda_err = e;
    return GLOWQ_ERR_CUDA;
  }
  return GLOWQ_OK;
}

}  // namespace glowq
