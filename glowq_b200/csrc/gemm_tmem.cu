// Corrected W4A16 product for decode batches (9 to 64 tokens; 2 to 8 in an exact form, see EXACT) with the dequantised weights in
// TENSOR MEMORY.
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
//   warps 3. dequantise in kTeams of four warps that take alternate steps - a thread owns one weight row, which is its
//            tensor-memory lane - and are the epilogue afterwards: lane = output column, so a token's 32 outputs of a
//            warp are one contiguous store.
// Two CTAs share an SM (256 tensor-memory columns and two teams each), so that one CTA's prologue and epilogue hide behind
// the other's steps.
//   r = X . R^T is computed inside the launch by the lowest block indices (placed first): a CTA multiplies 128 rows of R with a
// slice of K - the correction steps' loop with R in the place of L and X in the place of r - and parks an fp32 slot; once all
// slices of an R tile have arrived, its CTAs add each a share of its elements (one also the shares of those that left early) in a
// fixed order, round to fp16 and write r_buf.  The activation producers poll the count of finished shares before their first
// correction step.  As a launch of its own in front, r cost 6 to 11 microseconds per group.
// K may be sliced over CTAs; the CTA of a tile's last slice adds the others' fp32 slots in slice order (deterministic).
// A CTA waits for CTAs with lower block indices only (r, the earlier slices of its tile), which are placed before it: a launch
// gets through on any number of SMs.  Every wait is bounded; on expiry a status word is set, and the CTA drains and frees its
// tensor memory.
//
// Measured (B200, corrected group calls of the 13B shapes, microseconds at 16 / 32 / 64 tokens; before: MMAs issued by a lane that
// had waited alone, an epilogue of one token at a time, two slots in flight): q/k/v 19.2 / 20.5 / 23.3 (23.6 / 24.3 / 28.7), o_proj
// 11.2 / 12.3 / 16.1 (15.5 / 16.1 / 21.6), gate/up 29.5 / 30.1 / 33.8 (36.7 / 37.5 / 42.3), down_proj 18.1 / 19.8 / 23.7 (22.8 /
// 23.7 / 29.0).  Left: five to six microseconds of dependent chain per launch, and 0.3 to 0.4 per step and SM for the
// issue slots of the dequant warps, where the packed bytes alone would take 0.19 at the measured copy rate.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "../../include/glowq_w4a16.h"
#include "common.cuh"
#include "params.h"
#include "tcgen05.cuh"

namespace glowq {

int plan_prefetch(const glowq_w4a16_group_t& g, const unsigned char** ptr, unsigned* bytes);
int tensor_map_2d_ex(CUtensorMap* out, CUtensorMapDataType dtype, const void* ptr, uint64_t dim0, uint64_t dim1,
                     uint64_t stride_bytes, uint32_t box0, uint32_t box1, int swizzle);

namespace {

constexpr int kRows = 128;                    // weight rows (output columns) per CTA
constexpr int kPStage = kRows * 64;           // packed stage: 128 rows x 128 codes
constexpr int kA16 = kRows * 128;             // fp16 tile of a correction step: 128 rows x 64 columns
constexpr int kMaxS = 8, kMaxP = 8, kMaxC = 8;
constexpr int kA16Slots = 2;                  // fp16 tiles in flight; a CTA of r, which has no packed tiles, takes their room too
constexpr int kTeams = 2;
constexpr int kDequantWarps = 4 * kTeams, kCtrlWarps = 3, kThreads = 32 * (kCtrlWarps + kDequantWarps);
constexpr int kTmemCols = 256;                // per CTA: two share an SM
constexpr int kSmemBytes = 112 * 1024;
constexpr int kSlotsAhead = 4;                // slots of a tile that a thread has in flight (two 16-byte loads each)
constexpr int kMaxRCtas = 48;                 // CTAs that compute r
// Polls of a count of finished CTAs: some seconds, because another stream's kernel may hold the SMs that the rest of the CTAs
// of r need (they are placed first, so that nothing of this launch does).
constexpr unsigned kCountSpin = 1u << 22;
constexpr unsigned kDrainSpin = 1u << 18;     // polls (tens of milliseconds) for one of this CTA's own copies or MMAs
// Polls (some tens of microseconds) that a CTA of r spends on the others' arrival before it leaves the adding to them.
constexpr unsigned kShareSpin = 64;
// Words of the counters of r: per R tile 64 bits, of which 0..15 count the K slices that have arrived and 16 + z says that the CTA
// of slice z left before all had; then finished shares and exits.
enum : int { kRCnt = 0, kRFlag = 64, kRExit = 65 };
constexpr unsigned kArrivals = 0xFFFFu;
static_assert(kMaxRCtas <= 48 && kMaxRTiles * kRTileRows / kRows * 2 <= kRFlag, "the words of an R tile's count");

struct TsMember {
  const __half* scales;
  const int32_t* qzeros;
  const __half* bias;
  void* out;
  int OC, nu, sstride, zstride, out_stride, lr_separate, tile_begin;
  float alpha;
};
struct TsParams {
  uint32_t* status;
  uint32_t* tile_ctr;   // arrivals of a sliced tile's K slices, zero between launches
  uint32_t* r_ctr;      // counters of r (kRCnt ..), zero between launches
  float* r_slots;       // [CTA of r][token][128] fp32
  __half* r_buf;
  int n_r, r_slices, rank, nkr;   // CTAs of r (the lowest block indices; 0: r is ready), K slices of an R tile, 64-column steps of K
  float* slots;         // [ksplit][sliced tile][token / 4][128][4] fp32
  int M, G, out_fp32, n_members;
  int N;                // tokens per tile (multiple of 16)
  int ns, np;           // ring depths: stages (an activation tile and a tensor-memory A tile each), packed weights
  int a_col;            // first tensor-memory column of the A tiles
  int ksplit, full_tiles, n_tail, n_x;   // items: full_tiles whole tiles, then n_tail tiles of ksplit K slices each
  // head of the call that follows (weights of a streaming launch, which starts on them): every CTA asks L2 for its share
  int n_pf;
  const unsigned char* pf_ptr[kMaxPrefetch];
  unsigned pf_bytes[kMaxPrefetch];
  TsMember mem[kMaxMembers];
};
struct alignas(64) TsMaps {
  CUtensorMap x, r, R;
  CUtensorMap w[kMaxMembers], l[kMaxMembers];
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
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

// The MMAs of one step and the commit that releases its stage, issued by one elected lane of a converged warp.  The whole
// warp runs the issuing loop, and the step is one block, meant to leave descriptors and addresses where these instructions read
// them.  The gate/up launch of the 13B shapes at 16 tokens: 38.6 us with a loop under `lane == 0`, 34.4 with an elected lane per
// MMA, 33.0 with the step as one block.
// `bar`: the stage's release.  b_lo / b_hi: descriptor words of the activation tile, whose second 64 columns lie `sub16`
// further; accumulate 0: the first MMA overwrites D.
#define GLOWQ_TS_MMA(A, B, P) "@e tcgen05.mma.cta_group::1.kind::f16 [%0], " A ", " B ", %5, " P ";\n\t"
#define GLOWQ_TS_STEP                                                                                                        \
  "{\n\t.reg .pred e, p, t;\n\t.reg .b32 a<8>, l<8>;\n\t.reg .b64 b<8>;\n\t"                                                 \
  "setp.ne.b32 p, %6, 0;\n\tsetp.eq.b32 t, 0, 0;\n\telect.sync _|e, 0xffffffff;\n\t"                                         \
  "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\tadd.u32 a4, %1, 32;\n\tadd.u32 a5, %1, 40;\n\t"       \
  "add.u32 a6, %1, 48;\n\tadd.u32 a7, %1, 56;\n\tadd.u32 l1, %2, 2;\n\tadd.u32 l2, %2, 4;\n\tadd.u32 l3, %2, 6;\n\t"         \
  "add.u32 l4, %2, %4;\n\tadd.u32 l5, l4, 2;\n\tadd.u32 l6, l4, 4;\n\tadd.u32 l7, l4, 6;\n\t"                                \
  "mov.b64 b0, {%2, %3};\n\tmov.b64 b1, {l1, %3};\n\tmov.b64 b2, {l2, %3};\n\tmov.b64 b3, {l3, %3};\n\t"                     \
  "mov.b64 b4, {l4, %3};\n\tmov.b64 b5, {l5, %3};\n\tmov.b64 b6, {l6, %3};\n\tmov.b64 b7, {l7, %3};\n\t"                     \
  GLOWQ_TS_MMA("[%1]", "b0", "p") GLOWQ_TS_MMA("[a1]", "b1", "t") GLOWQ_TS_MMA("[a2]", "b2", "t")                \
  GLOWQ_TS_MMA("[a3]", "b3", "t") GLOWQ_TS_MMA("[a4]", "b4", "t") GLOWQ_TS_MMA("[a5]", "b5", "t")                \
  GLOWQ_TS_MMA("[a6]", "b6", "t") GLOWQ_TS_MMA("[a7]", "b7", "t")                                                                                     \
  "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t}"
__device__ __forceinline__ void umma_ts_step(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, uint32_t sub16, uint32_t idesc,
                                             uint32_t accumulate, uint32_t bar) {
  asm volatile(GLOWQ_TS_STEP::"r"(d), "r"(a), "r"(b_lo), "r"(b_hi), "r"(sub16), "r"(idesc), "r"(accumulate), "r"(bar) : "memory");
}
// One 16-column MMA with both operands in shared memory (correction steps), and a commit on its own.
__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit_elect(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
      : "memory");
}
// A poll that does not block (mbarrier.try_wait may suspend the thread while the phase is open).
__device__ __forceinline__ bool test_bar(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(a), "r"(parity)
               : "memory");
  return ok != 0;
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kDequantWarps * 32) : "memory"); }

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

// One share of the sum over an R tile's slots, added in a fixed order: a lane takes up to 12 slots of four elements, all in flight, and
// where there are more, two or four lanes share them.
struct ShareArgs {
  const float* base;
  __half* r_buf;
  size_t slot_floats;
  int r_slices, rank, n0, units;
};
__device__ __forceinline__ void add_share(const ShareArgs& a, int share, int et) {
  constexpr int kSlots = kMaxRCtas / 4;
  const int log = a.r_slices <= kSlots ? 0 : a.r_slices <= 2 * kSlots ? 1 : 2;   // log2 of the lanes per four elements
  const int part = (a.r_slices + (1 << log) - 1) >> log, zq = (et & ((1 << log) - 1)) * part, per = (kDequantWarps * 32) >> log;
  for (int i0 = 0; i0 < a.units; i0 += a.r_slices * per) {   // (the same number of rounds for all lanes: they exchange sums)
    const int i = i0 + share * per + (et >> log);
    const int tok = i >> 5, c4 = (i & 31) * 4, col = a.n0 + c4;
    const float* src = a.base + static_cast<size_t>(tok) * kRows + c4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f), u[kSlots];
#pragma unroll
    for (int z = 0; z < kSlots; ++z)
      u[z] = (i < a.units && z < part && zq + z < a.r_slices) ? __ldcg(reinterpret_cast<const float4*>(src + (zq + z) * a.slot_floats))
                                                              : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int z = 0; z < kSlots; ++z) {
      s.x += u[z].x;
      s.y += u[z].y;
      s.z += u[z].z;
      s.w += u[z].w;
    }
    for (int o = 1; o < (1 << log); o <<= 1) {
      s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
      s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
      s.z += __shfl_xor_sync(0xffffffffu, s.z, o);
      s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
    }
    if ((et & ((1 << log) - 1)) == 0 && i < a.units && col < a.rank) {   // the rank is a multiple of 8
      const __half2 lo = __floats2half2_rn(s.x, s.y), hi = __floats2half2_rn(s.z, s.w);
      *reinterpret_cast<uint2*>(a.r_buf + static_cast<size_t>(tok) * a.rank + col) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
}
// The shares of the CTAs in `left`, which could not wait.  Rare, and out of line: with this loop in the kernel the half-corrected
// Qwen2.5-7B step at 64 tokens took 548 us, 514 with the call.
__device__ __noinline__ void add_shares(ShareArgs a, unsigned long long left, int et) {
  for (; left != 0; left &= left - 1) add_share(a, __ffsll(left) - 1, et);
}

// EXACT (up to 8 tokens): the weights enter the product as the exact integers code - zero, every step has an accumulator of its own per
// team, and the team that dequantised a step adds scale x accumulator to fp32 sums in registers - the precision of the weight-streaming
// kernel.  Else they are rounded to fp16 with their scale first, as the reference rounds them.  The exact form spills: 48 bytes a
// thread, 46 thousand of 16.1 million instructions in the launch of the 13B gate/up shape at 8 tokens (29.6 us).
template <bool EXACT>
__global__ void __launch_bounds__(kThreads, 2)
gemm_tmem_kernel(const __grid_constant__ TsParams p, const __grid_constant__ TsMaps tm) {
  extern __shared__ unsigned char smem[];
  __shared__ int s_abort;
  __shared__ unsigned long long s_word;
  __shared__ uint32_t s_tmem_base;
  const uint32_t smem0 = (sm_u32(smem) + 1023u) & ~1023u;
  // barriers in the first 1 KB.  full: a stage's A tile is in tensor memory and its activations have landed (ONE barrier
  // for the issuing warp to poll per step: the dequant warps and the copies' bytes); cfull / cempty: the fp16 tiles of the
  // correction steps.
  const uint32_t full = smem0, empty = smem0 + 64, pfull = smem0 + 128, pempty = smem0 + 192, cfull = smem0 + 256,
                 cempty = smem0 + 320, accum = smem0 + 384;
  const uint32_t sub = static_cast<uint32_t>(p.N) * 128;      // one 64-column half of an activation tile
  const uint32_t ring = smem0 + 1024, a16 = ring + p.ns * 2 * sub, pring = a16 + kA16Slots * kA16;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const bool r_cta = static_cast<int>(blockIdx.x) < p.n_r;
  int tile_lin = 0, zslice, ks = 1, mi = 0, n0, m0 = 0, it0 = 0, nk, nkp;
  if (r_cta) {
    const int rt = static_cast<int>(blockIdx.x) / p.r_slices;
    zslice = static_cast<int>(blockIdx.x) - rt * p.r_slices;
    n0 = rt * kRows;
    it0 = p.nkr * zslice / p.r_slices;
    nk = p.nkr * (zslice + 1) / p.r_slices;
    nkp = it0;
  } else {
    const int item = static_cast<int>(blockIdx.x) - p.n_r;
    tile_lin = item;
    zslice = 0;
    if (item >= p.full_tiles) {
      const int r = item - p.full_tiles, t = r / p.ksplit;
      tile_lin = p.full_tiles + t;
      zslice = r - t * p.ksplit;
      ks = p.ksplit;
    }
    const int by = tile_lin / p.n_x, bx = tile_lin - by * p.n_x;
#pragma unroll
    for (int i = 1; i < kMaxMembers; ++i)
      if (i < p.n_members && bx >= p.mem[i].tile_begin) mi = i;
    n0 = (bx - p.mem[mi].tile_begin) * kRows;
    m0 = by * p.N;
    const int nk_all = p.G + p.mem[mi].nu;
    if (ks > 1) it0 = nk_all * zslice / ks;
    nk = ks > 1 ? nk_all * (zslice + 1) / ks : nk_all;
    nkp = max(it0, min(nk, p.G));   // steps [it0, nkp) are packed weights, [nkp, nk) the correction
  }
  const TsMember& mb = p.mem[mi];
  const int u0 = r_cta ? 0 : p.G;   // fp16 step it covers columns 64 (it - u0) .. of its operands
  constexpr int kAccs = EXACT ? kTeams : 1;   // accumulators in front of the correction's own
  const bool sep = !r_cta && (EXACT || mb.lr_separate != 0);
  const uint32_t cdepth = r_cta ? static_cast<uint32_t>(min(kMaxC, kA16Slots + p.np * kPStage / kA16)) : kA16Slots;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < p.ns; ++i) {
      g_mbar_init(full + 8 * i, 5);   // the four warps of a team and the copies
      g_mbar_init(empty + 8 * i, 1);
    }
    for (int i = 0; i < p.np; ++i) {
      g_mbar_init(pfull + 8 * i, 1);
      g_mbar_init(pempty + 8 * i, 4);
    }
    for (int i = 0; i < kMaxC; ++i) {
      g_mbar_init(cfull + 8 * i, 1);
      g_mbar_init(cempty + 8 * i, 1);
    }
    g_mbar_init(accum, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sm_u32(&s_tmem_base)), "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // Only now: a CTA of the next kernel that shares this SM must not take the tensor memory this one still asks for.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem = s_tmem_base;
  volatile int* abort_flag = &s_abort;
  // A thread that issues copies or MMAs stays until the last of them are done, also when a wait of the CTA has run out and
  // nobody else waits for them any more.  (Bounded: a step that was announced and never issued does not complete.)
  auto drain = [&](uint32_t bars, int depth, int issued) {
    for (int j = (issued > depth ? issued - depth : 0); j < issued; ++j) {
      uint32_t spins = 0;
      while (!g_mbar_try_once(bars + 8 * (j % depth), (j / depth) & 1) && ++spins < kDrainSpin) {
      }
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      Ring b{0, 0}, c{0, 0}, ca{0, 0};
      int issued = 0, cissued = 0;
      bool ok = true;
      const CUtensorMap* const tb = r_cta ? &tm.x : &tm.r;
      const CUtensorMap* const ta = r_cta ? &tm.R : &tm.l[mi];
      // one fp16 tile (L, R: constant) and the announcement of its step's bytes
      auto load_a = [&](int it) {
        const uint32_t bar = cfull + 8 * ca.i;
        g_mbar_expect_tx(bar, sub + kA16);
        g_tma_2d(a16 + ca.i * kA16, ta, (it - u0) * 64, n0, bar);
        ca.step(1, cdepth);
        ++cissued;
      };
      const int na0 = min(nk - nkp, static_cast<int>(cdepth));
      for (int j = 0; j < na0; ++j) load_a(nkp + j);
      asm volatile("griddepcontrol.wait;" ::: "memory");   // activations (and a ready r) come from the kernels before
      for (int it = it0; it < nkp; ++it) {
        // (nothing is issued once a wait of this CTA has failed: the other warps no longer wait for these copies)
        if (!(ok = g_mbar_wait(empty + 8 * b.i, b.ph ^ 1, abort_flag, p.status) && *abort_flag == 0)) break;
        const uint32_t dst = ring + b.i * 2 * sub, bar = full + 8 * b.i;
        g_mbar_expect_tx(bar, 2 * sub);
        g_tma_2d(dst, &tm.x, it * 128, m0, bar);
        g_tma_2d(dst + sub, &tm.x, it * 128 + 64, m0, bar);
        ++issued;
        b.step(1, p.ns);
      }
      if (ok && !r_cta && p.n_r > 0 && nkp < nk) {   // r of this launch
        uint32_t spins = 0;
        while (ld_acquire_u32(p.r_ctr + kRFlag) != static_cast<uint32_t>(p.n_r)) {
          __nanosleep(32);
          if (++spins > kCountSpin || *abort_flag) {
            *abort_flag = 1;
            atomicExch(p.status, 1u);
            ok = false;
            break;
          }
        }
        asm volatile("fence.proxy.async;" ::: "memory");   // written by plain stores, read by the copies below
      }
      for (int it = nkp; ok && it < nk; ++it) {
        if (!(ok = g_mbar_wait(empty + 8 * b.i, b.ph ^ 1, abort_flag, p.status) && *abort_flag == 0)) break;
        if (it - nkp >= na0) {
          if (!(ok = g_mbar_wait(cempty + 8 * c.i, c.ph ^ 1, abort_flag, p.status))) break;
          load_a(it);
        }
        g_tma_2d(ring + b.i * 2 * sub, tb, (it - u0) * 64, m0, cfull + 8 * c.i);
        c.step(1, cdepth);
        b.step(1, p.ns);
      }
      drain(full, p.ns, issued);
      drain(cfull, cdepth, cissued);
    }
    __syncwarp();
  } else if (warp == 2) {
    if (lane == 0) {
      Ring s{0, 0};
      int issued = 0;
      for (int it = it0; it < nkp; ++it) {
        if (!g_mbar_wait(pempty + 8 * s.i, s.ph ^ 1, abort_flag, p.status) || *abort_flag != 0) break;
        g_mbar_expect_tx(pfull + 8 * s.i, kPStage);
        g_tma_2d(pring + s.i * kPStage, &tm.w[mi], it * 16, n0, pfull + 8 * s.i);
        ++issued;
        s.step(1, p.np);
      }
      drain(pfull, p.np, issued);
    }
    __syncwarp();
    if (EXACT)
      for (int r = 0; r < p.n_pf; ++r)   // this CTA's copies are all issued
        for (uint32_t at = (blockIdx.x + lane * gridDim.x) * kPrefetchSlice; at < p.pf_bytes[r]; at += 32 * gridDim.x * kPrefetchSlice)
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.pf_ptr[r] + at), "r"(min(kPrefetchSlice, p.pf_bytes[r] - at))
                       : "memory");
  } else if (warp == 1) {
    {   // the whole warp: see umma_ts_step
      Ring b{0, 0}, c{0, 0};
      // instruction descriptor: fp32 accumulate, fp16 operands, K-major, M = 128, N tokens
      const uint32_t idesc = (1u << 4) | ((static_cast<uint32_t>(p.N) >> 3) << 17) | (static_cast<uint32_t>(kRows >> 4) << 24);
      const uint64_t desc0 = smem_desc_sw128(ring), desc_a0 = smem_desc_sw128(a16);
      const uint32_t hi = static_cast<uint32_t>(desc0 >> 32), lo0 = static_cast<uint32_t>(desc0);
      const uint32_t a_lo0 = static_cast<uint32_t>(desc_a0);
      // After a failed wait the MMAs go on without waiting (their results are void, the status word is set): every
      // stage is still released, and the warp stays converged for the elections.
      bool ok = true;
      auto wait_slow = [&](uint32_t bar, uint32_t ph) {
        if (ok) ok = g_mbar_wait_warp<false>(bar, ph, abort_flag, p.status);
      };
      uint32_t acc = 0;
      uint32_t ready = 0;   // the elected lane's poll
      for (int it = it0; it < nkp; ++it) {
        if (!__any_sync(0xffffffffu, ready)) wait_slow(full + 8 * b.i, b.ph);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t cur = b.i;
        b.step(1, p.ns);
        ready = g_mbar_test_elected(full + 8 * b.i, b.ph);   // answered while this stage's MMAs are issued
        if (EXACT) acc = 0;
        umma_ts_step(EXACT ? tmem + ((it - it0) & 1) * p.N : tmem, tmem + p.a_col + cur * 64, lo0 + cur * ((2 * sub) >> 4), hi, sub >> 4,
                     idesc, acc, empty + 8 * cur);
        acc = 1;
      }
      if (sep) acc = 0;   // the first MMA overwrites its accumulator
      const uint32_t d = tmem + (sep ? kAccs * p.N : 0);
      for (int it = nkp; it < nk; ++it) {
        wait_slow(cfull + 8 * c.i, c.ph);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t lo = lo0 + b.i * ((2 * sub) >> 4), la = a_lo0 + c.i * (kA16 >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          umma_ss(d, mk64(la + k * 2, hi), mk64(lo + k * 2, hi), idesc, acc);
          acc = 1;
        }
        umma_commit_elect(cempty + 8 * c.i);
        umma_commit_elect(empty + 8 * b.i);
        c.step(1, cdepth);
        b.step(1, p.ns);
      }
      umma_commit_elect(accum);
      if (lane == 0) drain(accum, 1, 1);
    }
    __syncwarp();
  } else {
    // ================================================================ dequant warps, then epilogue
    const int dw = warp - kCtrlWarps, team = dw >> 2, q = warp & 3;   // q: the tensor-memory lanes this warp reaches
    const int rloc = q * 32 + lane, row = n0 + rloc;
    const bool rvalid = row < mb.OC;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16);
    bool ok = true;
    float xacc[8];   // EXACT: this row's sums of the team's steps
#pragma unroll
    for (int j = 0; j < 8; ++j) xacc[j] = 0.f;
    {
      const __half* srow = mb.scales + static_cast<size_t>(rvalid ? row : 0) * mb.sstride;
      const int32_t* zrow = mb.qzeros + static_cast<size_t>(rvalid ? row : 0) * mb.zstride;
      const uint32_t prow = static_cast<uint32_t>(rloc) * 64, psw = (static_cast<uint32_t>(rloc) >> 1) & 3u;
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
      // EXACT: the sums of the team's step before (its MMAs are done, or nearly) are added before the next one's may overwrite them
      Ring before = a;
      float scale_before = 0.f;
      auto add_step = [&] {
        if (!test_bar(empty + 8 * before.i, before.ph)) ok = ok && g_mbar_wait(empty + 8 * before.i, before.ph, abort_flag, p.status);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t d[8];
        tmem_ld8(lane_base + team * p.N, d);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) xacc[j] = fmaf(scale_before, __uint_as_float(d[j]), xacc[j]);
      };
      for (int it = it0 + team; it < nkp; it += kTeams) {
        const uint32_t s2 = nx_s * 0x00010001u;
        const float scale = __half2float(__ushort_as_half(static_cast<unsigned short>(nx_s)));
        // -(1024 + z) and -(64 + z): the fp16 ulp is 1 at 1024 and 1/16 at 64
        const uint32_t zc = 0xD400E400u | (nx_z * 0x00100001u);
        // both polls go out together (an answer takes about a hundred clocks); after a failed wait the stores go on:
        // tensor memory is held to the end and the status word is set
        // A parity wait tells a phase from the one before it only, and the other team used this packed stage last.  When
        // this team starts step s, the MMAs of step s - 2 - ns are done; a ring shorter than ns + 2 may still wait for the
        // landing of step s - np, whose phase has the parity tested here one turn earlier - so that use is awaited first.
        if (p.np < p.ns + kTeams) ok = ok && g_mbar_wait(pempty + 8 * s.i, s.ph ^ 1, abort_flag, p.status);
        const bool have_p = test_bar(pfull + 8 * s.i, s.ph), have_e = test_bar(empty + 8 * a.i, a.ph ^ 1);
        if (!have_p) ok = ok && g_mbar_wait(pfull + 8 * s.i, s.ph, abort_flag, p.status);
        __syncwarp();
        fetch(it + kTeams);
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
          dequant_words<!EXACT>(v, w, 8 * half, zc, s2);
          if (half == 0) {   // the MMAs that read this stage's A tile before are done
            if (!have_e) ok = ok && g_mbar_wait(empty + 8 * a.i, a.ph ^ 1, abort_flag, p.status);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          tmem_st32(dst + half * 32, v);
          if (half == 0 && lane == 0) g_mbar_arrive(pempty + 8 * s.i);   // the packed rows are in registers
        }
        if (EXACT && it >= it0 + kTeams) add_step();
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) g_mbar_arrive(full + 8 * a.i);
        if (EXACT) {
          before = a;
          scale_before = scale;
        }
        a.step(kTeams, p.ns);
        s.step(kTeams, p.np);
      }
      if (EXACT && it0 + team < nkp) add_step();
    }
    if (EXACT && !r_cta) {   // the first team has the tokens: the other's sums go through the packed ring, which is free by now
      const uint32_t at = pring + rloc * 4;
      epi_sync();
      if (team == 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + j * (kRows * 4)), "f"(xacc[j]) : "memory");
      }
      epi_sync();
      if (team == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float v;
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at + j * (kRows * 4)) : "memory");
          xacc[j] += v;
        }
      }
    }

    // ---- epilogue.  Of a sliced tile, the CTAs of all slices but the last park fp32 slots; the last one - which holds the
    // correction steps, so that it is the late one - adds them, in slice order, to its own accumulators and stores.  (Its
    // block index is the highest of the tile's: the others are resident or done.)
    const int et = threadIdx.x - 32 * kCtrlWarps;
    const int ntok = min(p.N, p.M - m0);
    const size_t slot_floats = static_cast<size_t>(p.N) * kRows;
    const int sl_tile = tile_lin - p.full_tiles;
    const size_t slice_v4 = static_cast<size_t>(p.n_tail) * (slot_floats / 4);
    float4* const slot0 = reinterpret_cast<float4*>(p.slots + (r_cta ? 0 : sl_tile * slot_floats)) + rloc;
    const bool park = r_cta || zslice < ks - 1, finish = ks > 1 && zslice == ks - 1;
    auto await_count = [&](uint32_t* ctr, uint32_t n) {   // one thread; acquires the slots of the CTAs that counted
      uint32_t spins = 0;
      while (ld_acquire_u32(ctr) != n) {
        if (++spins > kCountSpin || *abort_flag) {
          atomicExch(p.status, 1u);
          break;
        }
      }
    };
    if (finish) {
      // The counters and slots are the previous launch's until it is complete, and a short slice gets here without having
      // waited for an MMA.
      if (et == 0) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        await_count(p.tile_ctr + sl_tile, static_cast<uint32_t>(ks - 1));
        p.tile_ctr[sl_tile] = 0u;
      }
      epi_sync();
    }
    // With a separate correction accumulator, a K slice that lies wholly in one phase never writes the other's.
    const bool has_main = it0 < p.G || !sep, has_lr = sep && nk > p.G;
    const float bias = (rvalid && !park && mb.bias) ? __half2float(mb.bias[row]) : 0.f;
    // Eight tokens at a time, alternately by the teams; four slots in flight (their tokens past the last one are not used).
    bool waited = false;
    for (int t0 = team * 8; t0 < ntok; t0 += 8 * kTeams) {
      float sum[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[j] = bias;
      float4* const at = slot0 + (t0 >> 2) * kRows;
      if (finish) {
        for (int z = 0; z < ks - 1; z += kSlotsAhead) {
          float4 u[kSlotsAhead][2];
#pragma unroll
          for (int k = 0; k < kSlotsAhead; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              u[k][h] = z + k < ks - 1 ? __ldcg(at + (z + k) * slice_v4 + h * kRows) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int k = 0; k < kSlotsAhead; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              sum[4 * h] += u[k][h].x;
              sum[4 * h + 1] += u[k][h].y;
              sum[4 * h + 2] += u[k][h].z;
              sum[4 * h + 3] += u[k][h].w;
            }
        }
      }
      if (!waited) {   // the first batch of slots is on its way while the last MMAs run
        if (lane == 0) ok = ok && g_mbar_wait(accum, 0, abort_flag, p.status);
        ok = __all_sync(0xffffffffu, ok);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        waited = true;
      }
      uint32_t acc[8], lr[8];
      if (!EXACT || r_cta) tmem_ld8(lane_base + t0, acc);
      if (has_lr) tmem_ld8(lane_base + kAccs * p.N + t0, lr);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (!ok) continue;
      if (EXACT && !r_cta) {
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j] += xacc[j];
      } else if (has_main) {
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j] += __uint_as_float(acc[j]);
      }
      if (has_lr) {
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j] = fmaf(mb.alpha, __uint_as_float(lr[j]), sum[j]);
      }
      const int n = ntok - t0;
      if (r_cta) {
        float* o = p.r_slots + blockIdx.x * slot_floats + static_cast<size_t>(t0) * kRows + rloc;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < n) __stcg(o + j * kRows, sum[j]);
      } else if (park) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          __stcg(at + zslice * slice_v4 + h * kRows, make_float4(sum[4 * h], sum[4 * h + 1], sum[4 * h + 2], sum[4 * h + 3]));
      } else if (rvalid) {
        const size_t idx = static_cast<size_t>(m0 + t0) * mb.out_stride + row;
        if (p.out_fp32) {
          float* o = static_cast<float*>(mb.out) + idx;
#pragma unroll
          for (int j = 0; j < 8; ++j, o += mb.out_stride)
            if (j < n) *o = sum[j];
        } else {
          __half* o = static_cast<__half*>(mb.out) + idx;
#pragma unroll
          for (int j = 0; j < 8; ++j, o += mb.out_stride)
            if (j < n) *o = __float2half_rn(sum[j]);
        }
      }
    }
    if (park) {
      epi_sync();
      const int rt = n0 / kRows;
      if (et == 0) {
        __threadfence();   // (cumulative over the CTA's stores, which the barrier ordered before it)
        if (!r_cta) atomicAdd(p.tile_ctr + sl_tile, 1u);
      }
      if (r_cta) {
        // Once all K slices of this R tile have arrived, every CTA adds its share of the elements.  No CTA depends on another
        // one being resident: it polls for a little while and then leaves, which the word of the count records unless all have
        // arrived by then.  Once they have, the word no longer changes, and the first of the CTAs that stayed - the last to
        // arrive always does - adds the shares of those that left.
        const ShareArgs sa{p.r_slots + static_cast<size_t>(rt) * p.r_slices * slot_floats, p.r_buf, slot_floats, p.r_slices, p.rank,
                           n0, ntok * (kRows / 4)};
        if (et == 0) {
          unsigned long long* const ctr = reinterpret_cast<unsigned long long*>(p.r_ctr + kRCnt) + rt;
          atomicAdd(ctr, 1ull);
          unsigned long long v;
          for (unsigned spins = 0; ((v = ld_acquire_u64(ctr)) & kArrivals) != static_cast<unsigned>(p.r_slices); ++spins)
            if (spins >= kShareSpin && atomicCAS(ctr, v, v | 1ull << (16 + zslice)) == v) break;
          s_word = v;
        }
        epi_sync();
        const bool stayed = (s_word & kArrivals) == static_cast<unsigned>(p.r_slices);
        int done = 0;
        if (stayed) {
          add_share(sa, zslice, et);
          done = 1;
          if (unsigned long long left = s_word >> 16; left != 0 && zslice == __ffsll(~left) - 1) {
            add_shares(sa, left, et);
            done += __popcll(left);
          }
        }
        asm volatile("fence.proxy.async;" ::: "memory");   // read by other CTAs' copies
        epi_sync();
        if (et == 0 && done != 0) {
          __threadfence();
          atomicAdd(p.r_ctr + kRFlag, static_cast<unsigned>(done));
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (p.n_r > 0 && threadIdx.x == 0) {   // the last CTA leaves the counters of r at zero
    if (atomicAdd(p.r_ctr + kRExit, 1u) == gridDim.x - 1) {
      for (int i = 0; i * p.r_slices < p.n_r; ++i) reinterpret_cast<unsigned long long*>(p.r_ctr + kRCnt)[i] = 0u;
      p.r_ctr[kRFlag] = 0u;
      p.r_ctr[kRExit] = 0u;
    }
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

inline int cdiv(int a, int b) { return (a + b - 1) / b; }
inline bool pdl_enabled() {
  static const bool on = [] {
    const char* v = std::getenv("GLOWQ_PDL");
    return !(v && v[0] == '0');
  }();
  return on;
}

template <bool EXACT>
cudaError_t launch(const TsParams& p, const TsMaps& tm, int ctas, cudaStream_t stream) {
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tmem_kernel<EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_done[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, gemm_tmem_kernel<EXACT>, p, tm);
}

inline int tile_tokens(int M) { return cdiv(M, 16) * 16; }   // tokens of the one tile (M <= 64)
// K slices of an R tile: about four 64-column steps each, at most kMaxRCtas CTAs in all.
inline int r_slices_for(int IC, int rank) { return std::max(1, std::min(cdiv(cdiv(IC, 64), 4), kMaxRCtas / cdiv(rank, kRows))); }

}  // namespace

// fp32 slots of r at the beginning of the scratch (M <= 64).
size_t gemm_tmem_r_bytes(int M, int IC, int rank) {
  return static_cast<size_t>(cdiv(rank, kRows)) * r_slices_for(IC, rank) * tile_tokens(M) * kRows * 4;
}

namespace {
// Rings, CTAs of r and the partition into work items of a group call; no CUDA calls.
struct TmemPlan {
  int N, ns, np;               // tokens per tile, ring depths
  int n_r, r_slices;           // CTAs of r, K slices of an R tile
  int ksplit, full_tiles, n_tail;
  int nk_min;                  // K steps of the shortest member
  int total, nk;               // tiles, K steps of the longest member
  size_t off_slots;            // in the workspace: K slices' slots (those of r are at kWsSlotsOffset)
};
TmemPlan make_tmem_plan(const glowq_w4a16_group_t& g, bool exact, bool compute_r, bool any_corr, bool any_separate, int sms) {
  TmemPlan pl{};
  pl.N = tile_tokens(g.M);
  {
    // stages: what tensor memory leaves beside the accumulators (a correction with its own doubles them), as far as shared
    // memory holds them and a few packed tiles
    const int smem = kSmemBytes - 2048 - kA16Slots * kA16, bst = pl.N * 256;
    pl.ns = std::min({kMaxS, (kTmemCols - (exact ? kTeams + 1 : any_separate ? 2 : 1) * pl.N) / 64, (smem - 3 * kPStage) / bst});
    pl.np = std::min(kMaxP, (smem - pl.ns * bst) / kPStage);
  }
  pl.off_slots = kWsSlotsOffset;
  if (compute_r) {
    pl.r_slices = r_slices_for(g.IC, g.rank);
    pl.n_r = cdiv(g.rank, kRows) * pl.r_slices;
    pl.off_slots += gemm_tmem_r_bytes(g.M, g.IC, g.rank);
  }
  const size_t slot_bytes = g.workspace_bytes > pl.off_slots ? g.workspace_bytes - pl.off_slots : 0;
  int total = 0, nk = 0, nk_min = 1 << 30;   // K steps of the longest and of the shortest member
  for (int i = 0; i < g.n_members; ++i) {
    const bool corr = any_corr && g.members[i].L && g.members[i].alpha != 0.f;
    const int steps = cdiv(g.IC, kGroup) + (corr ? cdiv(g.rank, 64) : 0);
    total += cdiv(g.members[i].OC, kRows);
    nk = std::max(nk, steps);
    nk_min = std::min(nk_min, steps);
  }
  pl.nk_min = nk_min;
  pl.nk = nk;
  pl.total = total;
  const int units = sms, resident = 2 * sms;
  const size_t item_bytes = static_cast<size_t>(pl.N) * kRows * 4;
  // Work partition: f rounds of whole tiles, the rest cut into ks slices of K.  Microseconds, fitted on B200 to every partition of 108
  // group calls (the one taken is 1.2 % slower than the best on average): a step of an SM while two CTAs share it, or of a CTA alone; r,
  // which the last steps wait for; a second wave of items (the CTAs of r take slots, but are gone before a whole tile is done); the
  // slices of a tile, which go through memory.  (The exact form's partitions of 808 calls: 1.0 % slower than the best, 21 % at worst.)
  const double r_us = compute_r ? 3.9 + 0.052 * pl.N : 0.0;
  pl.full_tiles = total;
  pl.n_tail = 0;
  pl.ksplit = 1;
  double best = 1e30;
  for (int f = 0; f <= total / units; ++f) {
    const int full = f * units, tail = total - full;
    // (a member is cut by its own steps: a slice without any would add what nothing wrote)
    for (int ks = 1; ks <= std::min(16, nk_min) && (ks == 1 || ks * 4 <= nk); ++ks) {
      if (ks > 1 && (tail == 0 || tail > kTileCtrWords || static_cast<size_t>(tail) * ks * item_bytes > slot_bytes)) break;
      const int items = full + tail * ks;
      const double load = static_cast<double>(f) * nk + static_cast<double>(cdiv(tail * ks, units)) * nk / ks;
      const double cost = std::max(load * (items > units ? 0.283 + 0.0012 * pl.N : 0.492 + 0.0012 * pl.N), r_us) +
                          5.1 * (cdiv(items, f > 0 ? resident : std::max(units, resident - pl.n_r)) - 1) +
                          (ks > 1 ? 1.0 + 0.0122 * pl.N * ks + 0.0129 * pl.N : 0.0);
      if (cost < best) {
        best = cost;
        pl.ksplit = ks;
        pl.full_tiles = ks > 1 ? full : total;
        pl.n_tail = ks > 1 ? tail : 0;
      }
    }
  }
  return pl;
}
}  // namespace

// The K slices' slots that a call takes where it has the room: any members of so many columns in all, with and without a correction
// (and r), planned for `sms` SMs.
size_t gemm_tmem_slot_bytes(int M, int IC, int OC_total, int rank, int n_members, int sms) {
  size_t most = 0;
  glowq_w4a16_group_t g{};
  g.M = M;
  g.IC = IC;
  g.workspace_bytes = ~static_cast<size_t>(0);
  g.n_members = std::min(n_members, OC_total);
  for (int narrow = 0; narrow < g.n_members; ++narrow) {   // members that end within a tile: one tile more each
    for (int i = 0; i < g.n_members; ++i) {
      g.members[i].OC = i == 0 ? OC_total - narrow : i <= narrow ? 1 : 0;
      g.members[i].L = &g;
      g.members[i].alpha = 1.f;
    }
    for (int corr = 0; corr <= (rank > 0 ? 2 : 0); ++corr) {   // none, r at hand, r of this launch
      g.rank = corr ? rank : 0;
      const TmemPlan pl = make_tmem_plan(g, true, corr == 2, corr > 0, false, sms);
      most = std::max(most, static_cast<size_t>(pl.n_tail) * pl.ksplit * pl.N * kRows * 4);
    }
  }
  return most;
}

// Microseconds of a call of 2 to 8 tokens in the exact form, as its partition has it.  Fitted on B200 together with the streaming
// kernel's estimate (see takes_gemm): a step of an SM that two CTAs share, of a CTA alone; r; a second wave; K slices.
double gemm_tmem_exact_us(const glowq_w4a16_group_t& g, bool compute_r, bool any_corr, int sms) {
  const TmemPlan pl = make_tmem_plan(g, true, compute_r, any_corr, false, sms);
  constexpr double kShared = 0.226, kAlone = 0.356;
  const int ks = pl.ksplit, f = ks > 1 ? pl.full_tiles / sms : 0, slices = ks > 1 ? pl.n_tail * ks : pl.total;
  const int per_sm = cdiv(slices, sms), items = f * sms + slices;
  const double steps = static_cast<double>(pl.nk) / ks;   // of an item that is not a whole tile beside slices
  double body;
  if (f == 0) {
    body = per_sm / 2 * 2 * steps * kShared + per_sm % 2 * steps * kAlone;
  } else {   // whole tiles in pairs, an odd one beside the slices
    const double cut = per_sm * steps, nk = pl.nk;
    body = f / 2 * 2 * nk * kShared;
    if (f % 2 == 0)
      body += cut * kShared;
    else
      body += cut < nk ? 2 * cut * kShared + (nk - cut) * kAlone : (nk + cut) * kShared;
  }
  const double slots = ks > 1 ? 0.455 : 0.0, start = 3.898;
  double us = start + std::max(body, compute_r ? 3.258 : 0.0) + slots + (ks > 1 ? 0.869 * slices / sms : 0.0) +
              2.196 * (cdiv(items, f > 0 ? 2 * sms : std::max(sms, 2 * sms - pl.n_r)) - 1);
  if (compute_r && items + pl.n_r > 2 * sms) us = std::max(us, start + 0.304 + 1.77 * steps * kShared + slots);   // items behind r's CTAs
  return us;
}

// (host arithmetic: see glowq_internal_workspace_map)
void gemm_tmem_workspace_map(const glowq_w4a16_group_t& g, bool exact, bool compute_r, bool any_corr, bool any_separate, int sms,
                             WorkspaceMap* map) {
  const TmemPlan pl = make_tmem_plan(g, exact, compute_r, any_corr, any_separate, sms);
  map->kernel = 1;
  map->ksplit = pl.ksplit;
  map->whole_tiles = pl.full_tiles;
  map->sliced_tiles = pl.n_tail;
  map->r_ctas = pl.n_r;
  map->shortest = pl.nk_min;
  map->ctr_begin = kWsTileCtrOffset;
  map->ctr_end = kWsTileCtrOffset + static_cast<size_t>(pl.n_tail) * 4;
  map->slots_begin = kWsSlotsOffset;
  map->slots_end = pl.off_slots + static_cast<size_t>(pl.n_tail) * pl.ksplit * pl.N * kRows * 4;
}

// Members' products and corrections of a group call of up to 64 tokens.  compute_r: r into g.r_buf as well (else it is
// there); the workspace must hold gemm_tmem_r_bytes for it behind kWsSlotsOffset.
int gemm_tmem_forward(const glowq_w4a16_group_t& g, bool exact, bool compute_r, bool any_corr, bool any_separate, int sms,
                      cudaStream_t stream, cudaError_t* cuda_err) {
  const int G = cdiv(g.IC, kGroup);
  const TmemPlan pl = make_tmem_plan(g, exact, compute_r, any_corr, any_separate, sms);
  unsigned char* const ws = static_cast<unsigned char*>(g.workspace);
  TsParams p{};
  p.N = pl.N;
  p.ns = pl.ns;
  p.np = pl.np;
  p.a_col = kTmemCols - p.ns * 64;
  if (compute_r) {
    p.r_slices = pl.r_slices;
    p.n_r = pl.n_r;
    p.nkr = cdiv(g.IC, 64);
    p.rank = g.rank;
    p.r_buf = static_cast<__half*>(g.r_buf);
    p.r_ctr = reinterpret_cast<uint32_t*>(ws + kWsHeaderBytes);
    p.r_slots = reinterpret_cast<float*>(ws + kWsSlotsOffset);
  }
  p.status = reinterpret_cast<uint32_t*>(ws) + WS_STATUS;
  p.tile_ctr = reinterpret_cast<uint32_t*>(ws + kWsTileCtrOffset);
  p.slots = reinterpret_cast<float*>(ws + pl.off_slots);
  p.ksplit = pl.ksplit;
  p.full_tiles = pl.full_tiles;
  p.n_tail = pl.n_tail;
  p.M = g.M;
  p.G = G;
  p.out_fp32 = g.out_dtype == GLOWQ_OUT_F32;
  p.n_pf = exact ? plan_prefetch(g, p.pf_ptr, p.pf_bytes) : 0;
  p.n_members = g.n_members;
  TsMaps tm;
  std::memset(&tm, 0, sizeof(tm));
  int rc;
  if ((rc = tensor_map_2d_ex(&tm.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.x, g.IC, g.M, static_cast<uint64_t>(g.x_stride) * 2, 64,
                             p.N, 1)))
    return rc;
  tm.r = tm.x;
  tm.R = tm.x;
  if (compute_r && (rc = tensor_map_2d_ex(&tm.R, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.R, g.IC, g.rank,
                                          static_cast<uint64_t>(g.R_stride) * 2, 64, kRows, 1)))
    return rc;
  if (any_corr && (rc = tensor_map_2d_ex(&tm.r, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.r_buf, g.rank, g.M,
                                         static_cast<uint64_t>(g.rank) * 2, 64, p.N, 1)))
    return rc;
  int n_x = 0;
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
    d.sstride = m.scale_stride;
    d.zstride = m.zero_stride_i32;
    d.out_stride = m.out_stride;
    d.alpha = m.alpha;
    d.lr_separate = corr && m.alpha != 1.f;
    d.tile_begin = n_x;
    n_x += cdiv(m.OC, kRows);
  }
  p.n_x = n_x;
  const int ctas = p.n_r + p.full_tiles + p.n_tail * p.ksplit;
  const cudaError_t e = exact ? launch<true>(p, tm, ctas, stream) : launch<false>(p, tm, ctas, stream);
  if (e != cudaSuccess) {
    *cuda_err = e;
    return GLOWQ_ERR_CUDA;
  }
  return GLOWQ_OK;
}

}  // namespace glowq
