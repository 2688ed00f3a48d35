// Corrected W4A16 product for prompts (65 tokens and more): CTA pairs, dequantised weights in TENSOR MEMORY.
//
//   D[256 output columns, N tokens] += W[256, 128 k] . X[N, 128 k]^T      (one quantisation group of K per step)
//
// A cluster of two CTAs works on one tile (cta_group::2 MMAs, M = 256).  Each CTA dequantises 128 weight rows - its half of the
// MMA's A operand - in registers and writes them to its tensor memory (tcgen05.st); each holds half of the tile's tokens as the B
// operand in shared memory (TMA, 128-byte swizzle), which the MMA reads from both.  The accumulator is the transposed output tile:
// a CTA's 128 output columns are its tensor-memory lanes.
//   warp 0      activation producer (one thread): TMA of N/2 x 128 activations per step, of r in the correction steps
//   warp 1      tensor memory; CTA 0's issues tcgen05.mma and the commits that release the stages of both CTAs; a thread of CTA 1's
//               hands out the items
//   warp 2      weight producer (one thread): TMA of 128 rows x 64 B of packed codes, or of 32 columns of an fp16 operand (L, R)
//   warp 3      scales and zero points: from memory into shared memory beside the packed stage, in the form the arithmetic takes
//   warps 4-7   epilogue: accumulators as MMA fragments, transposed by stmatrix, stored by the copy engine
//   warps 8-15  dequantise, in two teams of four warps that take alternate steps (a thread owns one weight row); two thirds of the pass
//               that adds K slices' slots or the correction's accumulator are theirs as well
// r = X . R^T is the first items of the launch: R in the place of the weights (fp16 rows go to tensor memory as they are), the
// output goes to r_buf; the producers wait for the count of finished r tiles before their first correction step.
//   What bounds it: 256 tokens, the MMAs (1024 clocks a step; measured 1030) and the epilogue that only the next steps' dequantisation
// runs under; narrower tiles, tensor memory's writes and the chain from a stage's release to its next MMAs (about 1000 clocks a step
// whatever the width, also with four teams).  Long runs are bound by the 1 kW limit.  Corrected group calls at 211, 2048 and
// 4096 tokens, us (behind the stroke before the elected waits, the dequantisation in place, the shared sums and the fitted plans, same
// minute): 14B gate/up 69, 601, 1217 / 72, 641, 1244; 14B down_proj 49, 310, 640 / 64, 351, 657; 3B q/k/v 25, 69, 123 / 28, 75, 136.
//   Items are taken in order from a ticket (or are the clusters themselves where they are few): a CTA waits for items in front of
// its own only, so a launch gets through on any number of SMs.  K may be sliced; the CTAs of a tile's last slice add the other
// slices' fp32 slots in slice order (deterministic).  Every wait is bounded; on expiry a status word is set and the CTAs drain.
#include <algorithm>
#include <cmath>
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

constexpr int kRows = 128;                 // weight rows (output columns) per CTA
constexpr int kPStage = kRows * 64;        // weight stage: 128 rows x 64 bytes
constexpr int kMeta = 2 * kRows * 4;       // per weight stage and row: the scale twice (half2), the zero-point constants
constexpr int kNP = 4;                     // weight stages per team: an fp16 step of 128 columns takes all four.  (With two the producer,
                                           // which takes the steps in order, feeds one team at a time; 14B down_proj, 777 tokens: 220 -> 194 us.)
constexpr int kMaxB = 8;                   // activation stages at most
constexpr int kOStage = 2048;              // output stage of a warp: 32 tokens x 32 fp16 columns, or 16 x 32 fp32
constexpr int kMaxO = 8;                   // output stages at most
constexpr int kTeams = 2;                  // of four dequant warps
constexpr int kTmemCols = 512;
constexpr int kThreads = 32 * (8 + 4 * kTeams);
constexpr int kConsumers = 2 * (1 + 1 + 1 + 4 * kTeams + 4) + 1;   // arrivals that give the item slot back: two CTAs, and the MMA warp
constexpr int kAhead = 12;                 // the next item is asked for when this many steps of one are still to be loaded
constexpr int kSmemMax = 227 * 1024 - 512;
constexpr unsigned kCountSpin = 1u << 22;  // polls of a count of finished CTAs (seconds)
constexpr unsigned kSumGoSpin = 1u << 25;  // polls for the end of such a wait, longer than it: 8 s at a quarter of a microsecond
static_assert(kSumGoSpin >= 8 * kCountSpin, "a poll of a count is a trip to memory, up to eight times a poll of a barrier");
constexpr unsigned kDrainSpin = 1u << 18;  // polls for one of this CTA's own copies or MMAs
enum : int { kCTicket = 72, kCFlag = 73, kCExit = 74 };   // words of the counters in front of the slots, zero between launches

struct PtMember {
  const __half* scales;
  const int32_t* qzeros;
  const __half* bias;
  void* out;
  int OC, sstride, zstride, out_stride, tile_begin, corr, svec, out_tma;
  float alpha;
};
struct PtParams {
  uint32_t* status;
  uint32_t* ctr;          // counters (kCTicket ..)
  int tickets;            // items by ticket (0: every cluster has one)
  uint32_t* tile_ctr;     // [r tiles, then sliced tiles][2 CTAs] arrivals of K slices
  float *slots, *r_slots; // [slice][tile][token / 4][256][4]
  int M, G, N, rank, out_fp32, n_members;
  int n_items, n_r, r_x, r_slices, r_tiles;     // items; r items, column tiles, K slices and tiles of r
  int ctr_base;           // tile counters of r in front of those of the sliced tiles
  int n_tiles, n_x, n_y, band, full_tiles, n_tail, ksplit;
  int sep;                // a correction with a factor other than 1: an accumulator of its own
  int nbuf, nb, na, no;   // accumulators, activation stages, A stages (64 columns each, behind the accumulators), output stages
  PtMember mem[kMaxMembers];
};
struct alignas(64) PtMaps {
  CUtensorMap x, r, R, r_out;
  CUtensorMap w[kMaxMembers], l[kMaxMembers], out[kMaxMembers];
};

enum : uint32_t { kValid = 1u, kIsR = 2u, kCorr = 4u };
struct Tile {          // eight words in shared memory
  uint32_t flags;      // kValid, kIsR, kCorr (this CTA's rows are corrected), member
  int n0, m0, it0, nk, z, ks, ctr;
  __device__ __forceinline__ bool is_r() const { return flags & kIsR; }
  __device__ __forceinline__ bool corr() const { return flags & kCorr; }
  __device__ __forceinline__ int mi() const { return static_cast<int>(flags >> 8); }
};

// Work of one item for the CTA `rank` of its pair.
__device__ __forceinline__ Tile decode(const PtParams& p, uint32_t ticket, int rank) {
  Tile t{};
  // (a ticket that no launch could have reached - a workspace that was not zero - ends the launch)
  if (ticket >= static_cast<uint32_t>(p.n_items)) return t;
  int item = static_cast<int>(ticket), mi = 0;
  t.flags = kValid;
  if (item < p.n_r) {
    const int tile = item / p.r_slices, y = tile / p.r_x;
    t.z = item - tile * p.r_slices;
    t.ks = p.r_slices;
    t.n0 = (2 * (tile - y * p.r_x) + rank) * kRows;
    t.m0 = y * p.N;
    t.it0 = p.G * t.z / t.ks;
    t.nk = p.G * (t.z + 1) / t.ks;
    t.ctr = tile;
    t.flags |= kIsR | kCorr;
    return t;
  }
  item -= p.n_r;
  int tile = item;
  t.z = 0;
  t.ks = 1;
  t.ctr = 0;
  if (item >= p.full_tiles) {
    const int r = item - p.full_tiles, k = r / p.ksplit;
    tile = p.full_tiles + k;
    t.z = r - k * p.ksplit;
    t.ks = p.ksplit;
    t.ctr = p.ctr_base + k;
  }
  // token tiles in bands; within a band, column tile by column tile
  const int per = p.n_x * p.band, b = tile / per, rem = tile - b * per, rows = min(p.band, p.n_y - b * p.band);
  const int x = rem / rows, y = b * p.band + rem - x * rows;
  const int ct = 2 * x + rank, other = 2 * x + 1 - rank;
  int mo = 0;
#pragma unroll
  for (int i = 1; i < kMaxMembers; ++i) {
    if (i < p.n_members && ct >= p.mem[i].tile_begin) mi = i;
    if (i < p.n_members && other >= p.mem[i].tile_begin) mo = i;
  }
  t.n0 = (ct - p.mem[mi].tile_begin) * kRows;
  t.m0 = y * p.N;
  const bool corr = p.mem[mi].corr != 0 && ct < p.n_tiles, any = corr || (p.mem[mo].corr != 0 && other < p.n_tiles);
  const int nk = p.G + (any ? (p.rank + 127) >> 7 : 0);
  t.it0 = nk * t.z / t.ks;
  t.nk = nk * (t.z + 1) / t.ks;
  t.flags |= (corr ? kCorr : 0u) | static_cast<uint32_t>(mi) << 8;
  return t;
}
// 64-column halves of step `it`
__device__ __forceinline__ int halves(const PtParams& p, int it) { return it < p.G || p.rank - (it - p.G) * 128 > 64 ? 2 : 1; }

__device__ __forceinline__ void tmem_st32p(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
      "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16p(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16p(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// 32 lanes x 32 columns as MMA fragments: v[8 i + 2 m] and v[8 i + 2 m + 1] are columns 8 i + 2 (lane % 4) and the next of lane
// 8 m + lane / 4.
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, uint32_t (&v)[32]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[4 * h]), "=r"(v[4 * h + 1]), "=r"(v[4 * h + 2]), "=r"(v[4 * h + 3]), "=r"(v[4 * h + 8]), "=r"(v[4 * h + 9]),
          "=r"(v[4 * h + 10]), "=r"(v[4 * h + 11]), "=r"(v[4 * h + 16]), "=r"(v[4 * h + 17]), "=r"(v[4 * h + 18]),
          "=r"(v[4 * h + 19]), "=r"(v[4 * h + 24]), "=r"(v[4 * h + 25]), "=r"(v[4 * h + 26]), "=r"(v[4 * h + 27])
        : "r"(taddr + (static_cast<uint32_t>(16 * h) << 16)));
}
__device__ __forceinline__ void lds_v4(uint32_t* w, uint32_t addr) {
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr));
}

// The MMAs of one step (eight of 16 columns, or the first four) and the commit that releases its stages in both CTAs, issued by
// one elected lane of a converged warp, as one block (see umma_ts_step of the one-CTA form, where it was measured).
#define GLOWQ_PT_MMA(E, A, B, P) "@" E " tcgen05.mma.cta_group::2.kind::f16 [%0], " A ", " B ", %5, " P ";\n\t"
__device__ __forceinline__ void pair_step(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, uint32_t sub16, uint32_t idesc,
                                          uint32_t accumulate, uint32_t both_halves, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred e, f, p, t;\n\t.reg .b32 a<8>, l<8>;\n\t.reg .b64 b<8>;\n\t.reg .b16 m;\n\t"
      "setp.ne.b32 p, %6, 0;\n\tsetp.eq.b32 t, 0, 0;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.and.b32 f, %8, 0, e;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\tadd.u32 a4, %1, 32;\n\tadd.u32 a5, %1, 40;\n\t"
      "add.u32 a6, %1, 48;\n\tadd.u32 a7, %1, 56;\n\tadd.u32 l1, %2, 2;\n\tadd.u32 l2, %2, 4;\n\tadd.u32 l3, %2, 6;\n\t"
      "add.u32 l4, %2, %4;\n\tadd.u32 l5, l4, 2;\n\tadd.u32 l6, l4, 4;\n\tadd.u32 l7, l4, 6;\n\t"
      "mov.b64 b0, {%2, %3};\n\tmov.b64 b1, {l1, %3};\n\tmov.b64 b2, {l2, %3};\n\tmov.b64 b3, {l3, %3};\n\t"
      "mov.b64 b4, {l4, %3};\n\tmov.b64 b5, {l5, %3};\n\tmov.b64 b6, {l6, %3};\n\tmov.b64 b7, {l7, %3};\n\tmov.b16 m, 3;\n\t"
      GLOWQ_PT_MMA("e", "[%1]", "b0", "p") GLOWQ_PT_MMA("e", "[a1]", "b1", "t") GLOWQ_PT_MMA("e", "[a2]", "b2", "t")
      GLOWQ_PT_MMA("e", "[a3]", "b3", "t") GLOWQ_PT_MMA("f", "[a4]", "b4", "t") GLOWQ_PT_MMA("f", "[a5]", "b5", "t")
      GLOWQ_PT_MMA("f", "[a6]", "b6", "t") GLOWQ_PT_MMA("f", "[a7]", "b7", "t")
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%7], m;\n\t}" ::"r"(d),
      "r"(a), "r"(b_lo), "r"(b_hi), "r"(sub16), "r"(idesc), "r"(accumulate), "r"(bar), "r"(both_halves)
      : "memory");
}
__device__ __forceinline__ void pair_commit(uint32_t bar) {   // both CTAs' barriers, once all MMAs issued so far are done
  asm volatile(
      "{\n\t.reg .pred e;\n\t.reg .b16 m;\n\tmov.b16 m, 3;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}" ::"r"(bar)
      : "memory");
}
// TMA of this CTA's half of the B operand; the bytes count on a barrier of CTA 0.
__device__ __forceinline__ void tma_2d_pair(uint32_t dst, const CUtensorMap* tmap, int x, int y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(tmap), "r"(x), "r"(y), "r"(cluster_bar)
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tmap, int x, int y, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(tmap), "r"(x), "r"(y), "r"(src)
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
// The same as a wait, for the places where the answer is on the path of the next MMA: the thread stays awake.
__device__ __forceinline__ bool spin_bar(uint32_t a, uint32_t parity, volatile int* abort_flag, uint32_t* status) {
  for (uint32_t spins = 0; !test_bar(a, parity);) {
    if ((++spins & 63u) == 0 && *abort_flag) return false;
    if (spins > 4 * kGemmSpin) {
      *abort_flag = 1;
      atomicExch(status, 3u);
      return false;
    }
  }
  return true;
}
// The epilogue warps go on together or leave together: none may wait at a barrier for one whose wait ran out.
__device__ __forceinline__ bool epi_vote(bool ok) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(r)
               : "r"(static_cast<uint32_t>(ok))
               : "memory");
  return r != 0;
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// Ring positions of the teams' weight stages.
static_assert(kNP == 4, "two bits per team");
struct TeamRings {
  uint32_t idx, ph;   // two bits and one bit per team
  __device__ __forceinline__ uint32_t at(uint32_t team) const { return team * kNP + ((idx >> (2 * team)) & 3u); }
  __device__ __forceinline__ uint32_t phase(uint32_t team) const { return (ph >> team) & 1u; }
  __device__ __forceinline__ void step(uint32_t team) {
    const uint32_t i = (idx >> (2 * team)) & 3u;
    idx ^= (i ^ ((i + 1) & 3u)) << (2 * team);
    ph ^= static_cast<uint32_t>(i == 3u) << team;
  }
};
struct Ring {   // one ring position: index and phase parity
  uint32_t i, ph;
  __device__ __forceinline__ void step(uint32_t depth) {
    if (++i == depth) {
      i = 0;
      ph ^= 1;
    }
  }
};

// Barriers in the first KB of shared memory.
constexpr uint32_t kBFull = 0;                    // [kMaxB] CTA 0: both CTAs' activations have landed and A tiles are written
constexpr uint32_t kBDone = 64;                   // [kMaxB] each CTA: the MMAs of the step are done
constexpr uint32_t kBPFull = 128;                 // [kTeams][kNP] weight stages
constexpr uint32_t kBPEmpty = 192;
constexpr uint32_t kBAccFull = 256;               // [2] each CTA
constexpr uint32_t kBAccEmpty = 272;              // [2] CTA 0: the epilogue warps of both CTAs
constexpr uint32_t kBSFull = 288;                 // each CTA: an item
constexpr uint32_t kBSEmpty = 320;                // CTA 1: everybody has read it, and the weight producers are nearly through with it
constexpr uint32_t kBFin = 352;                   // CTA 0: all MMAs done
constexpr uint32_t kBSumGo = 360;                 // each CTA: an item's accumulators may be merged (see merge)
constexpr uint32_t kBSumDone = 368;               // each CTA: the dequant warps have merged their part
constexpr uint32_t kBItem = 384;                  // the item (a Tile)

// The pass over an item's accumulators that comes before the output where K is sliced or the correction has an accumulator of its own:
// 16 tokens at a time from `first` on, every `step`, the correction's sums and the other slices' slots (in slice order) are added, and
// the result goes to the slot or back to the accumulator.  The dequant warps, which have nothing to do until the epilogue gives the
// accumulators back, take two thirds of it: by the four epilogue warps alone the seven slots of a sliced r tile of 224 tokens took 18 us.
constexpr int kMergers = 1 + kTeams;
struct Merge {
  uint32_t d;          // this warp's lanes of the accumulators
  float4* slot0;       // this thread's row of the tile's first slot
  size_t slice_v4;
  int ntok;
  bool park, has_main, has_lr;
  float alpha;
  __device__ __forceinline__ Merge(const PtParams& p, const Tile& t, uint32_t lane_base, uint32_t buf, int rank, int rloc) {
    const bool is_r = t.is_r();
    const size_t slot_floats = static_cast<size_t>(p.N) * (2 * kRows);
    d = lane_base + buf * static_cast<uint32_t>(p.N);
    slot0 = reinterpret_cast<float4*>(is_r ? p.r_slots + static_cast<size_t>(t.ctr) * slot_floats
                                           : p.slots + static_cast<size_t>(t.ctr - p.ctr_base) * slot_floats) +
            rank * kRows + rloc;
    slice_v4 = (is_r ? static_cast<size_t>(p.r_tiles) : static_cast<size_t>(p.n_tail)) * (slot_floats / 4);
    ntok = min(p.N, p.M - t.m0);
    park = t.z < t.ks - 1;
    has_main = t.it0 < p.G || !p.sep;
    has_lr = p.sep && !is_r && t.corr() && t.nk > p.G;
    alpha = p.mem[t.mi()].alpha;
  }
};
__device__ __forceinline__ void merge(const PtParams& p, const Tile& t, const Merge& m, int part) {
  for (int t0 = 16 * part; t0 < m.ntok; t0 += 16 * kMergers) {
    uint32_t v[16];
    tmem_ld16p(m.d + t0, v);
    if (m.has_lr) {
      uint32_t lr[16];
      tmem_ld16p(m.d + p.N + t0, lr);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int k = 0; k < 16; ++k)
        v[k] = __float_as_uint(fmaf(m.alpha, __uint_as_float(lr[k]), m.has_main ? __uint_as_float(v[k]) : 0.f));
    } else {
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (!m.has_main) {
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = 0u;
      }
    }
    float4* const at = m.slot0 + static_cast<size_t>(t0 / 4) * (2 * kRows);
    if (m.park) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        __stcg(at + t.z * m.slice_v4 + k * (2 * kRows), make_float4(__uint_as_float(v[4 * k]), __uint_as_float(v[4 * k + 1]),
                                                                    __uint_as_float(v[4 * k + 2]), __uint_as_float(v[4 * k + 3])));
      continue;
    }
    for (int z = 0; z < t.ks - 1; z += 3) {   // three slots in flight
      float4 u[3][4];
#pragma unroll
      for (int y = 0; y < 3; ++y)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          u[y][k] = z + y < t.ks - 1 ? __ldcg(at + (z + y) * m.slice_v4 + k * (2 * kRows)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int y = 0; y < 3; ++y)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          v[4 * k] = __float_as_uint(__uint_as_float(v[4 * k]) + u[y][k].x);
          v[4 * k + 1] = __float_as_uint(__uint_as_float(v[4 * k + 1]) + u[y][k].y);
          v[4 * k + 2] = __float_as_uint(__uint_as_float(v[4 * k + 2]) + u[y][k].z);
          v[4 * k + 3] = __float_as_uint(__uint_as_float(v[4 * k + 3]) + u[y][k].w);
        }
    }
    tmem_st16p(m.d + t0, v);
  }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ PtParams p, const __grid_constant__ PtMaps tm) {
  extern __shared__ unsigned char smem[];
  __shared__ int s_abort;
  __shared__ uint32_t s_tmem_base;
  const uint32_t smem0 = (sm_u32(smem) + 1023u) & ~1023u;
  const uint32_t sub = static_cast<uint32_t>(p.N) * 64;        // 64 columns of this CTA's N / 2 tokens
  const uint32_t ring = smem0 + 1024, pring = ring + p.nb * 2 * sub, meta = pring + kTeams * kNP * kPStage,
                 ostage = meta + kTeams * kNP * kMeta;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int pair = static_cast<int>(blockIdx.x >> 1);

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < kMaxB; ++i) {
      g_mbar_init(smem0 + kBFull + 8 * i, 9);    // four dequant warps of either CTA, the announcement of the copies
      g_mbar_init(smem0 + kBDone + 8 * i, 1);
    }
    for (int i = 0; i < kTeams * kNP; ++i) {
      g_mbar_init(smem0 + kBPFull + 8 * i, 2);   // the copy and the scales
      g_mbar_init(smem0 + kBPEmpty + 8 * i, 4);
    }
    for (int i = 0; i < 2; ++i) {
      g_mbar_init(smem0 + kBAccFull + 8 * i, 1);
      g_mbar_init(smem0 + kBAccEmpty + 8 * i, 8);
    }
    g_mbar_init(smem0 + kBSFull, 1);
    g_mbar_init(smem0 + kBSEmpty, kConsumers);
    g_mbar_init(smem0 + kBFin, 1);
    g_mbar_init(smem0 + kBSumGo, 1);
    g_mbar_init(smem0 + kBSumDone, 4 * kTeams);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sm_u32(&s_tmem_base)), "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();   // both CTAs' barriers and tensor memory
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem = s_tmem_base;
  volatile int* abort_flag = &s_abort;
  auto drain = [&](uint32_t bars, int depth, int issued) {   // a thread that issues copies or MMAs stays until they are done
    for (int j = (issued > depth ? issued - depth : 0); j < issued; ++j) {
      uint32_t spins = 0;
      while (!g_mbar_try_once(smem0 + bars + 8 * (j % depth), (j / depth) & 1) && ++spins < kDrainSpin) {
      }
    }
  };
  auto await = [&](uint32_t bar, uint32_t ph) { return g_mbar_wait(smem0 + bar, ph, abort_flag, p.status); };
  uint32_t sph = 0;
  auto release_item = [&] { g_mbar_arrive_cluster(map_to_cta(smem0 + kBSEmpty, 1)); };
  auto next_item = [&](Tile& t, bool one_thread, bool release) -> bool {
    bool ok = g_mbar_wait_cluster(smem0 + kBSFull, sph, abort_flag, p.status);
    if (!one_thread) ok = __all_sync(0xffffffffu, ok);
    if (!ok) return false;
    uint32_t w[8];
    lds_v4(w, smem0 + kBItem);
    lds_v4(w + 4, smem0 + kBItem + 16);
    t.flags = w[0];
    t.n0 = w[1];
    t.m0 = w[2];
    t.it0 = w[3];
    t.nk = w[4];
    t.z = w[5];
    t.ks = w[6];
    t.ctr = w[7];
    if (!one_thread) __syncwarp();
    if (release && (one_thread || lane == 0)) release_item();
    sph ^= 1;
    return t.flags & kValid;
  };
  Tile t{};   // (no member out of range when the first wait for an item runs out)

  if (warp == 0) {
    if (lane == 0) {
      asm volatile("griddepcontrol.wait;" ::: "memory");   // activations (and a ready r) come from the kernels before
      Ring b{0, 0};
      int issued = 0;
      bool ok = true, have_r = p.n_r == 0;
      const uint32_t full0 = map_to_cta(smem0 + kBFull, 0);
      while (ok && next_item(t, true, true)) {
        const int y = t.m0 + rank * (p.N >> 1);
        for (int it = t.it0; it < t.nk; ++it) {
          if (!(ok = await(kBDone + 8 * b.i, b.ph ^ 1) && *abort_flag == 0)) break;
          const int h = halves(p, it);
          if (it >= p.G && !have_r) {   // r of this launch
            uint32_t spins = 0;
            while (ld_acquire_u32(p.ctr + kCFlag) != static_cast<uint32_t>(2 * p.r_tiles)) {
              __nanosleep(32);
              if (++spins > kCountSpin || *abort_flag) {
                *abort_flag = 1;
                atomicExch(p.status, 1u);
                ok = false;
                break;
              }
            }
            if (!ok) break;
            asm volatile("fence.proxy.async;" ::: "memory");   // read by the copies below
            have_r = true;
          }
          if (rank == 0) g_mbar_expect_tx(smem0 + kBFull + 8 * b.i, 2 * h * sub);
          const uint32_t dst = ring + b.i * 2 * sub;
          const CUtensorMap* const m = it < p.G ? &tm.x : &tm.r;
          const int x = (it < p.G ? it : it - p.G) * 128;
          tma_2d_pair(dst, m, x, y, full0 + 8 * b.i);
          if (h == 2) tma_2d_pair(dst + sub, m, x + 64, y, full0 + 8 * b.i);
          ++issued;
          b.step(p.nb);
        }
      }
      drain(kBDone, p.nb, issued);
    }
    __syncwarp();
  } else if (warp == 2) {
    if (lane == 0) {
      TeamRings s{0, 0};
      uint32_t j = 0;
      bool ok = true;
      while (ok && next_item(t, true, false)) {
        const CUtensorMap* const a16 = t.is_r() ? &tm.R : &tm.l[t.mi()];
        const CUtensorMap* const a4 = &tm.w[t.mi()];
        const int ask = max(t.it0, t.nk - kAhead);   // pairs that are ahead get more of the items
        for (int it = t.it0; ok && it < t.nk; ++it, ++j) {
          if (it == ask) release_item();
          const uint32_t team = j & (kTeams - 1);
          const bool f16 = t.is_r() || it >= p.G;
          const int n = !f16 ? 1 : (t.corr() ? 2 * halves(p, it) : 0);
          for (int k = 0; k < n; ++k) {
            const uint32_t at = s.at(team);
            if (!(ok = await(kBPEmpty + 8 * at, s.phase(team) ^ 1) && *abort_flag == 0)) break;
            const uint32_t bar = smem0 + kBPFull + 8 * at, dst = pring + at * kPStage;
            g_mbar_expect_tx(bar, kPStage);
            if (f16)
              g_tma_2d(dst, a16, (t.is_r() ? it : it - p.G) * 128 + k * 32, t.n0, bar);
            else
              g_tma_2d(dst, a4, it * 16, t.n0, bar);
            s.step(team);
          }
        }
      }
      // the last copy of every stage has landed
      for (uint32_t at = 0; at < kTeams * kNP; ++at) {
        const uint32_t team = at / kNP, k = at % kNP, cur = (s.idx >> (2 * team)) & 3u;
        // (a stage of the present round, or of the round before; none at all: its barrier is in its first phase)
        const uint32_t par = k < cur ? s.phase(team) : s.phase(team) ^ 1;
        uint32_t spins = 0;
        while (!g_mbar_try_once(smem0 + kBPFull + 8 * at, par) && ++spins < kDrainSpin) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // A lane loads four rows, eight groups at a time: with one group at a time (two bytes of each row) the loads of a step
    // take 256 wavefronts, and the shared-memory loads of the dequant warps wait behind them.
    TeamRings s{0, 0};
    uint32_t j = 0;
    bool ok = true;
    while (ok && next_item(t, false, true)) {
      const int n4 = t.is_r() ? t.it0 : min(t.nk, p.G);   // steps [it0, n4) have scales
      const PtMember& mb = p.mem[t.mi()];
      const int vec = mb.svec;
      for (int it = t.it0; ok && it < n4;) {
        uint32_t sc[4][4], zw[4];
        const int g8 = it & ~7, c0 = it & 7, n = min(8 - c0, n4 - it);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = t.n0 + lane + 32 * i;
#pragma unroll
          for (int k = 0; k < 4; ++k) sc[i][k] = 0u;   // rows past the end multiply by zero
          zw[i] = 0u;
          if (row >= mb.OC) continue;
          const __half* sp = mb.scales + static_cast<size_t>(row) * mb.sstride + g8;
          zw[i] = static_cast<uint32_t>(__ldg(mb.qzeros + static_cast<size_t>(row) * mb.zstride + (g8 >> 3)));
          if (vec == 8) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(sp));
            sc[i][0] = v.x;
            sc[i][1] = v.y;
            sc[i][2] = v.z;
            sc[i][3] = v.w;
          } else if (vec == 4) {
#pragma unroll
            for (int k = 0; k < 2; ++k)
              if (g8 + 4 * k < p.G) {
                const uint2 v = __ldg(reinterpret_cast<const uint2*>(sp + 4 * k));
                sc[i][2 * k] = v.x;
                sc[i][2 * k + 1] = v.y;
              }
          } else if (vec == 2) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (g8 + 2 * k < p.G) sc[i][k] = __ldg(reinterpret_cast<const uint32_t*>(sp + 2 * k));
          } else {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (g8 + k < p.G) sc[i][k >> 1] |= static_cast<uint32_t>(__half_as_ushort(__ldg(sp + k))) << (16 * (k & 1));
          }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          if (c < c0 || c >= c0 + n || !ok) continue;
          const uint32_t team = j & (kTeams - 1), at = s.at(team);
          bool w = true;
          if (lane == 0) w = await(kBPEmpty + 8 * at, s.phase(team) ^ 1);
          if (!(ok = __all_sync(0xffffffffu, w))) continue;
          s.step(team);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            // -(1024 + z) and -(64 + z): the fp16 ulp is 1 at 1024 and 1/16 at 64
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(meta + at * kMeta + (lane + 32 * i) * 8),
                         "r"(prmt(sc[i][c >> 1], 0u, c & 1 ? 0x3232u : 0x1010u)),
                         "r"(0xD400E400u | ((zw[i] >> (4 * c)) & 0xFu) * 0x00100001u)
                         : "memory");
          __syncwarp();
          if (lane == 0) g_mbar_arrive(smem0 + kBPFull + 8 * at);
          ++j;
        }
        it += n;
      }
      // fp16 stages have none, but this warp's arrival is what keeps it in step: it must not miss a phase of a stage
      for (int it = max(t.it0, n4); ok && it < t.nk; ++it, ++j) {
        const int stages = t.corr() ? 2 * halves(p, it) : 0;
        const uint32_t team = j & (kTeams - 1);
        for (int k = 0; k < stages; ++k) {
          if (lane == 0) {
            ok = ok && await(kBPEmpty + 8 * s.at(team), s.phase(team) ^ 1);
            if (ok) g_mbar_arrive(smem0 + kBPFull + 8 * s.at(team));
          }
          s.step(team);
        }
        ok = __all_sync(0xffffffffu, ok);
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {   // the whole warp: see pair_step
      Ring b{0, 0};
      uint32_t n = 0;
      // instruction descriptor: fp32 accumulate, fp16 operands, K-major, M = 256 over the pair, N tokens
      const uint32_t idesc = (1u << 4) | ((static_cast<uint32_t>(p.N) >> 3) << 17) | (static_cast<uint32_t>(2 * kRows >> 4) << 24);
      const uint64_t desc0 = smem_desc_sw128(ring);
      const uint32_t hi = static_cast<uint32_t>(desc0 >> 32), lo0 = static_cast<uint32_t>(desc0);
      bool ok = true;
      uint32_t ready = 0;   // the elected lane's poll
      const uint32_t acol = tmem + kTmemCols - p.na * 64, stage16 = (2 * sub) >> 4, sub16 = sub >> 4, G = p.G, nb = p.nb, na = p.na;
      uint32_t ai = 0;
      while (ok && __all_sync(0xffffffffu, next_item(t, false, true))) {
        const uint32_t buf = p.nbuf == 2 ? n & 1 : 0, use = p.nbuf == 2 ? n >> 1 : n;
        ++n;
        if (!(ok = g_mbar_wait_warp<false>(smem0 + kBAccEmpty + 8 * buf, (use & 1) ^ 1, abort_flag, p.status))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t d = tmem + buf * static_cast<uint32_t>(p.N), acc = 0;
        // (what was read from shared memory is the same in all lanes: a reduction says so in the source)
        const uint32_t it0 = __reduce_or_sync(0xffffffffu, t.it0), nk = __reduce_or_sync(0xffffffffu, t.nk);
        const uint32_t last = G + ((p.rank + 127) >> 7) - 1, last_both = (p.rank & 127) == 0 || (p.rank & 127) > 64;
        const uint32_t sep_at = p.sep ? G : 0xFFFFFFFFu;
        if (it0 > sep_at) d += p.N;   // a K slice that starts behind the correction's first step
        for (uint32_t it = it0; it < nk; ++it) {
          if (it == sep_at) {
            d += p.N;
            acc = 0;
          }
          if (!__any_sync(0xffffffffu, ready) &&
              !(ok = g_mbar_wait_warp<true>(smem0 + kBFull + 8 * b.i, b.ph, abort_flag, p.status)))
            break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          pair_step(d, acol + ai * 64, lo0 + b.i * stage16, hi, sub16, idesc, acc, it < G || it != last || last_both,
                    smem0 + kBDone + 8 * b.i);
          if (++ai == na) ai = 0;
          b.step(nb);
          ready = g_mbar_test_elected(smem0 + kBFull + 8 * b.i, b.ph);
          acc = 1;
        }
        if (ok) pair_commit(smem0 + kBAccFull + 8 * buf);
      }
      asm volatile(
          "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
          "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem0 + kBFin)
          : "memory");
      if (lane == 0) drain(kBFin, 1, 1);
    } else if (lane == 0) {   // items: the cluster's own, or by ticket, until one past the end
      if (p.tickets) asm volatile("griddepcontrol.wait;" ::: "memory");   // the counters are the previous launch's until it is complete
      uint32_t item = 0, ph = 1;
      do {
        if (!await(kBSEmpty, ph)) break;
        item = p.tickets ? atomicAdd(p.ctr + kCTicket, 1u) : (ph ? pair : p.n_items);
        ph ^= 1;
        for (int c = 0; c < 2; ++c) {
          const Tile n = decode(p, item, c);
          const uint32_t at = map_to_cta(smem0 + kBItem, c);
          asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(n.flags), "r"(n.n0), "r"(n.m0), "r"(n.it0)
                       : "memory");
          asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + 16), "r"(n.nk), "r"(n.z), "r"(n.ks), "r"(n.ctr)
                       : "memory");
          asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_to_cta(smem0 + kBSFull, c)) : "memory");
        }
      } while (item < static_cast<uint32_t>(p.n_items));
    }
    __syncwarp();
  } else if (warp >= 8) {
    // ================================================================ dequant warps
    const int team = (warp - 8) >> 2, q = warp & 3;   // q: the tensor-memory lanes this warp reaches
    const int rloc = q * 32 + lane;
    const uint32_t na = p.na, nb = p.nb, dst0 = tmem + (static_cast<uint32_t>(q * 32) << 16) + kTmemCols - na * 64;
    const uint32_t prow = pring + team * kNP * kPStage + static_cast<uint32_t>(rloc) * 64, psw = (static_cast<uint32_t>(rloc) >> 1) & 3u;
    const uint32_t mrow = meta + team * kNP * kMeta + static_cast<uint32_t>(rloc) * 8;
    const uint32_t pfull = smem0 + kBPFull + 8 * team * kNP, pempty = smem0 + kBPEmpty + 8 * team * kNP;
    const uint32_t full0 = map_to_cta(smem0 + kBFull, 0);
    // this team's next step (of all tiles' together), its place in the ring of steps, that of the step na before (whose MMAs read
    // the same A stage), its A stage
    uint32_t jn = team, ai = team % na;
    const uint32_t e0 = team + 4 * nb - na;
    Ring s{0, 0}, d{team % nb, (team / nb) & 1u}, e{e0 % nb, (e0 / nb) & 1u};
    uint32_t jbase = 0, n = 0, mph = 0;
    bool ok = true;
    while (ok && next_item(t, false, true)) {
      const uint32_t buf = p.nbuf == 2 ? n & 1 : 0;
      ++n;
      const uint32_t jend = jbase + static_cast<uint32_t>(t.nk - t.it0);
      for (; jn < jend; jn += kTeams) {
        const int it = t.it0 + static_cast<int>(jn - jbase);
        const uint32_t dst = dst0 + ai * 64, dbar = smem0 + kBDone + 8 * e.i;
        // both polls go out together (an answer takes some hundred clocks)
        const bool have_p = test_bar(pfull + 8 * s.i, s.ph), have_d = jn < na || test_bar(dbar, e.ph);
        auto await_stage = [&] {   // the MMAs that read this A stage before are done
          if (!have_d) ok = ok && spin_bar(dbar, e.ph, abort_flag, p.status);
          __syncwarp();
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        };
        if (!t.is_r() && it < p.G) {
          if (!have_p) ok = ok && g_mbar_wait(pfull + 8 * s.i, s.ph, abort_flag, p.status);
          __syncwarp();
          uint32_t s2, zc, w[16];
          asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(s2), "=r"(zc) : "r"(mrow + s.i * kMeta));
#pragma unroll
          for (int k = 0; k < 4; ++k) lds_v4(w + 4 * k, prow + s.i * kPStage + ((static_cast<uint32_t>(k) ^ psw) << 4));
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t v[32];
            dequant_words(v, w, 8 * half, zc, s2);
            if (half == 0) {
              if (lane == 0) g_mbar_arrive(pempty + 8 * s.i);   // the packed rows are in registers
              await_stage();
            }
            tmem_st32p(dst + half * 32, v);   // (after a failed wait the stores go on: the status word is set)
          }
          s.step(kNP);
        } else {   // fp16 rows (L, R), or zeros beside rows that are corrected
          const int h = halves(p, it);
          await_stage();
          for (int half = 0; half < h; ++half) {
            uint32_t v[32];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              if (t.corr()) {
                ok = ok && g_mbar_wait(pfull + 8 * s.i, s.ph, abort_flag, p.status);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; ++i) lds_v4(v + 16 * k + 4 * i, prow + s.i * kPStage + ((static_cast<uint32_t>(i) ^ psw) << 4));
                __syncwarp();
                if (lane == 0) g_mbar_arrive(pempty + 8 * s.i);
                s.step(kNP);
              } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) v[16 * k + i] = 0u;
              }
            }
            tmem_st32p(dst + half * 32, v);
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) g_mbar_arrive_cluster(full0 + 8 * d.i);
#pragma unroll
        for (int k = 0; k < kTeams; ++k) {
          d.step(nb);
          e.step(nb);
          if (++ai == na) ai = 0;
        }
      }
      jbase = jend;
      if (ok && (p.sep || t.ks > 1)) {
        // (the epilogue may be waiting for the other slices, whose CTAs another stream's kernel may keep from their SMs)
        ok = g_mbar_wait<kSumGoSpin>(smem0 + kBSumGo, mph, abort_flag, p.status);
        mph ^= 1;
        if (!__all_sync(0xffffffffu, ok)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        merge(p, t, Merge(p, t, tmem + (static_cast<uint32_t>(q * 32) << 16), buf, rank, rloc), 1 + team);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) g_mbar_arrive(smem0 + kBSumDone);
      }
    }
  } else {
    // ================================================================ epilogue warps
    const int q = warp & 3, rloc = q * 32 + lane, et = static_cast<int>(threadIdx.x) - 128;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t accempty0 = map_to_cta(smem0 + kBAccEmpty, 0);
    const uint32_t ow = ostage + static_cast<uint32_t>(q * p.no) * kOStage;
    uint32_t n = 0, ob = 0, mph = 0;
    // Output stages, each warp its own, handed to the copy engine two at a time (the fence takes some hundred clocks).  Behind the
    // stores the oldest ones have been read, so that the next two stages are free: a stage has a group of its own, an empty one where
    // the warp's columns lie past the end, so that the groups still to be waited for are the last stages written.
    auto store_stages = [&](const CUtensorMap* m, int x, int y, int rows, int count, bool inside) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        uint32_t o = ob;
        for (int c = 0; c < count; ++c) {
          if (inside) tma_store_2d(m, x, y + c * rows, ow + o * kOStage);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          if (++o == static_cast<uint32_t>(p.no)) o = 0;
        }
        if (p.no >= 8)
          asm volatile("cp.async.bulk.wait_group.read 6;" ::: "memory");
        else if (p.no >= 6)
          asm volatile("cp.async.bulk.wait_group.read 4;" ::: "memory");
        else
          asm volatile("cp.async.bulk.wait_group.read 2;" ::: "memory");
      }
      __syncwarp();
      ob += count;
      if (ob >= static_cast<uint32_t>(p.no)) ob -= p.no;
    };
    auto stage_at = [&](int c) {
      uint32_t o = ob + c;
      if (o >= static_cast<uint32_t>(p.no)) o -= p.no;
      return ow + o * kOStage;
    };
    for (;;) {
      const uint32_t buf = p.nbuf == 2 ? n & 1 : 0, use = p.nbuf == 2 ? n >> 1 : n;
      ++n;
      bool go = next_item(t, false, true);
      // (everything that takes a trip to memory before the accumulator is awaited)
      const bool is_r = t.is_r();
      const PtMember& mb = p.mem[t.mi()];
      const int row = t.n0 + rloc, col0 = t.n0 + q * 32, ntok = min(p.N, p.M - t.m0);
      const bool valid = row < mb.OC;
      const bool as_f32 = p.out_fp32 && !is_r, tma = is_r || mb.out_tma, frag = tma && !as_f32;
      float bias[4];   // of this lane's column, or of the four columns of its fragments
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int c = frag ? col0 + 8 * m + (lane >> 2) : row;
        bias[m] = (go && !is_r && mb.bias && c < mb.OC) ? __half2float(mb.bias[c]) : 0.f;
      }
      const bool park = t.z < t.ks - 1, finish = t.ks > 1 && !park;
      uint32_t* const tctr = p.tile_ctr + 2 * t.ctr + rank;
      go = go && await(kBAccFull + 8 * buf, use & 1);
      if (!epi_vote(go)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (finish) {
        if (et == 0) {
          uint32_t spins = 0;
          while (ld_acquire_u32(tctr) != static_cast<uint32_t>(t.ks - 1)) {
            if (++spins > kCountSpin || *abort_flag) {
              atomicExch(p.status, 1u);
              break;
            }
          }
          *tctr = 0u;
        }
        epi_sync();
      }
      const uint32_t d = lane_base + buf * static_cast<uint32_t>(p.N);
      const CUtensorMap* const om = is_r ? &tm.r_out : &tm.out[t.mi()];
      const bool inside = col0 < (is_r ? p.rank : mb.OC);
      if (p.sep || t.ks > 1) {
        if (et == 0) g_mbar_arrive(smem0 + kBSumGo);
        merge(p, t, Merge(p, t, lane_base, buf, rank, rloc), 0);
        const bool merged = await(kBSumDone, mph);
        mph ^= 1;
        if (!epi_vote(merged)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      int pending = 0;
      for (int t0 = 0; t0 < (park ? 0 : ntok); t0 += 32) {
        uint32_t v[32];
        if (frag)
          tmem_ld_frag(d + t0, v);
        else
          tmem_ld32(d + t0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (t0 + 32 >= ntok) {   // the accumulator is read
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) g_mbar_arrive_cluster(accempty0 + 8 * buf);
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) + bias[(k >> 1) & 3]);
        // Outputs go through shared memory and the copy engine, which clips at the last token and column.
        if (frag) {
          // the fragments, transposed, are rows of 8 columns: 16-byte chunks, XORed within 64 bytes as the copy expects them
          const uint32_t r = lane & 7, m = lane >> 3, at = stage_at(pending);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
              asm("cvt.rn.f16x2.f32 %0, %1, %2;"
                  : "=r"(h[j])
                  : "f"(__uint_as_float(v[8 * i + 2 * j + 1])), "f"(__uint_as_float(v[8 * i + 2 * j])));
            asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(
                             at + (8 * i + r) * 64 + ((m ^ ((r >> 1) & 3u)) << 4)),
                         "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3])
                         : "memory");
          }
          if (++pending == 2 || t0 + 32 >= ntok) {
            store_stages(om, col0, t.m0 + t0 - 32 * (pending - 1), 32, pending, inside);
            pending = 0;
          }
        } else if (tma) {
#pragma unroll
          for (int k = 0; k < 32; ++k)
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(stage_at(k >> 4) + lane * 4 + (k & 15) * 128), "r"(v[k]) : "memory");
          store_stages(om, col0, t.m0 + t0, 16, t0 + 16 < ntok ? 2 : 1, inside);
        } else if (valid) {   // rows of any pitch and address
          float* of = static_cast<float*>(mb.out) + static_cast<size_t>(t.m0 + t0) * mb.out_stride + row;
          __half* oh = static_cast<__half*>(mb.out) + static_cast<size_t>(t.m0 + t0) * mb.out_stride + row;
#pragma unroll
          for (int k = 0; k < 32; ++k) {
            if (t0 + k < ntok) {
              if (as_f32)
                *of = __uint_as_float(v[k]);
              else
                *oh = __float2half_rn(__uint_as_float(v[k]));
              of += mb.out_stride;
              oh += mb.out_stride;
            }
          }
        }
      }
      if (park) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        epi_sync();
        if (et < 4) g_mbar_arrive_cluster(accempty0 + 8 * buf);
        if (et == 0) {
          __threadfence();   // (cumulative over the CTA's stores, which the barrier ordered before it)
          atomicAdd(tctr, 1u);
        }
      } else if (is_r) {   // r is in memory before the count says so
        if (lane == 0) {
          asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
          asm volatile("fence.proxy.async;" ::: "memory");
          __threadfence();
        }
        epi_sync();
        if (et == 0 && p.ctr != nullptr) {
          __threadfence();
          atomicAdd(p.ctr + kCFlag, 1u);
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (p.ctr != nullptr && threadIdx.x == 0) {   // the last CTA leaves the counters at zero
    if (atomicAdd(p.ctr + kCExit, 1u) == gridDim.x - 1) {
      p.ctr[kCTicket] = 0u;
      p.ctr[kCFlag] = 0u;
      p.ctr[kCExit] = 0u;
    }
  }
  cluster_sync_all();   // neither CTA gives up memory that the other's MMAs or arrivals still reach
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
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

cudaError_t launch(const PtParams& p, const PtMaps& tm, int pairs, size_t smem, cudaStream_t stream) {
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    if (e != cudaSuccess) return e;
    attr_done[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, gemm_pair_kernel, p, tm);
}

// Tiles, slices and rings of a group call; no CUDA calls.
struct PairPlan {
  int N, n_y, nbuf, nb, na, no;
  int n_tiles, n_x, ksplit, full_tiles, n_tail, nk_min;
  int r_x, r_tiles, r_slices;
  size_t off_slots, end;       // in the workspace: slots of the K slices (those of r at kWsSlotsOffset), end of all slots
};

// Microseconds of a launch's parts, fitted on B200 to 438 group calls of 65 to 4096 tokens with some twenty plans each: the plans that
// the planner takes are 0.8 % slower than the best ones on average, 11 % at worst.
// A step of N tokens (tensor-memory writes and the chain from a stage's release to its next MMAs bound narrow tiles, the MMAs the
// widest; slower the more pairs are busy); what a tile costs beside its steps; an item of r, whose fp16 rows come through four weight
// stages a step; adding up K slices, three slots of 48 tokens a trip to memory.
inline double step_us(int N, double busy) { return (N <= 192 ? 0.3571 + 0.00032 * N : 0.00189 * N) * (1.0 + 0.345 * busy); }
inline double tile_us(int N, bool two) { return two ? 3.35 : 2.83 + 0.0063 * N; }
inline double r_item_us(int N, double steps) { return 0.05 + steps * (0.816 + 0.0032 * N); }
inline double r_sum_us(int N, int ks) { return ks > 1 ? 1.27 + (0.0117 * cdiv(ks - 1, 3) + 0.0003 * (ks - 1)) * N : 0.0; }
inline double sum_us(int N, int ks, bool whole_before) {
  return ks > 1 ? (whole_before ? 1.7 : 2.03) + (0.0173 * cdiv(ks - 1, 3) + 0.0025 * (ks - 1)) * N : 0.0;
}
constexpr int kMaxRSlices = 16;
constexpr double kTicketUs = 5.6;   // the first item by ticket: nothing of it runs ahead of the kernel before
// When `items` of d microseconds each, taken in order, are done: n[i] pairs are through with their first at e[i].
double rounds_us(int items, const int (&n)[4], const double (&e)[4], double d) {
  double lo = 1e300, hi = 0.0, t = 0.0;
  int pairs = 0, k[4];
  for (int i = 0; i < 4; ++i)
    if (n[i] > 0) {
      pairs += n[i];
      lo = std::min(lo, e[i]);
      hi = std::max(hi, e[i]);
    }
  // (every pair does so many at least)
  const int all = std::max(0, items / pairs - 1 - static_cast<int>(std::ceil((hi - lo) / d)));
  std::fill(k, k + 4, all);
  for (int done = all * pairs; done < items;) {
    int b = -1;
    for (int i = 0; i < 4; ++i)
      if (n[i] > 0 && (b < 0 || e[i] + k[i] * d < e[b] + k[b] * d)) b = i;
    t = e[b] + k[b] * d;
    done += n[b];
    ++k[b];
  }
  return t;
}

// First column tile of each member; returns the tiles in all.  Members that share a pair of tiles are corrected both or neither: in one
// accumulator the correction steps of a pair would reach the rows of the other member as zeros times r, which are not zero where r
// overflowed.  (With an accumulator of its own the correction is left out of the rows that have none.)
int member_tiles(const glowq_w4a16_group_t& g, bool any_corr, bool sep, int* begin) {
  int tiles = 0;
  bool before = false;
  for (int i = 0; i < g.n_members; ++i) {
    const bool corr = any_corr && g.members[i].L && g.members[i].alpha != 0.f;
    if (corr != before && !sep) tiles = (tiles + 1) & ~1;
    before = corr;
    begin[i] = tiles;
    tiles += cdiv(g.members[i].OC, kRows);
  }
  return tiles;
}

PairPlan make_pair_plan(const glowq_w4a16_group_t& g, bool compute_r, bool any_corr, bool sep, int sms) {
  const int G = cdiv(g.IC, kGroup), nu = any_corr ? cdiv(g.rank, 128) : 0, nk = G + nu, pairs = std::max(1, sms / 2);
  PairPlan best{};
  double best_cost = 1e300;
  int begin[kMaxMembers];
  const int n_tiles = member_tiles(g, any_corr, sep, begin);
  const int n_x = cdiv(n_tiles, 2);
  const size_t room = g.workspace_bytes > kWsSlotsOffset ? g.workspace_bytes - kWsSlotsOffset : 0;
  const int max_n = sep ? 192 : 256, y0 = cdiv(g.M, max_n), y1 = std::max(y0, std::min(cdiv(g.M, 64), y0 * 2 + 2));
  int last_n = 0;
  for (int y = y0; y <= y1; ++y) {
    PairPlan pl{};
    pl.N = std::max(64, cdiv(cdiv(g.M, y), 32) * 32);   // (M = 256 over a pair: N is a multiple of 32)
    if (pl.N == last_n) continue;
    last_n = pl.N;
    pl.n_y = cdiv(g.M, pl.N);
    pl.n_tiles = n_tiles;
    pl.n_x = n_x;
    pl.nk_min = G;
    const size_t tile_bytes = static_cast<size_t>(pl.N) * (2 * kRows) * 4;
    const int total = n_x * pl.n_y, f_max = total / pairs;
    const bool two = pl.N <= 192 && !sep;
    if (compute_r) {
      pl.r_x = cdiv(g.rank, 2 * kRows);
      pl.r_tiles = pl.r_x * pl.n_y;
    }
    for (int rks = 1; rks <= (compute_r ? std::max(1, std::min({kMaxRSlices, pairs / pl.r_tiles, G / 4})) : 1); ++rks) {   // K slices of r
      const size_t r_bytes = rks > 1 ? tile_bytes * pl.r_tiles * rks : 0;
      if (rks > 1 && (2 * pl.r_tiles > kTileCtrWords || r_bytes > room)) break;
      const int n_r = pl.r_tiles * rks, ctr_room = kTileCtrWords / 2 - (rks > 1 ? pl.r_tiles : 0);
      // an item of r (pairs take one, or several one after another), the sum of its slices, the pairs that add them
      const double r_item = compute_r ? r_item_us(pl.N, static_cast<double>(G) / rks) * cdiv(n_r, pairs) : 0.0;
      const double r_ready = r_item + r_sum_us(pl.N, rks);
      const int r_pairs = std::min(n_r, pairs), r_last = r_pairs / rks, others = pairs - r_pairs;
      for (int f = std::max(0, f_max - 1); f <= f_max; ++f) {   // rounds of whole tiles, the rest in ks slices each
        const int full = f * pairs, tail = total - full;
        for (int ks = 1; ks <= std::min(16, G) && (ks == 1 || ks * 4 <= nk); ++ks) {
          if (ks > 1 && (tail == 0 || tail > ctr_room || tile_bytes * tail * ks + r_bytes > room)) break;
          const int items = n_r + (ks > 1 ? full + tail * ks : total);
          const double step = step_us(pl.N, std::min(1.0, static_cast<double>(items) / pairs)), beside = tile_us(pl.N, two);
          const double tile = nk * step + beside, slice = static_cast<double>(nk) / ks * step + beside;
          if (((ks > 1 ? f * pairs : total) * tile + (ks > 1 ? tail * ks * slice : 0.0)) / pairs >= best_cost) continue;
          // first tiles, and last slices of sliced ones, wait for r before their correction; with one accumulator a pair goes on
          // when it has added r's slices
          const double with_r = compute_r ? r_ready + nu * step + beside : 0.0, r_free = two ? r_item : r_ready;
          // (a pair asks for its next item early in one of r: those that add r's slices take tiles although they are through late)
          double cost;
          if (ks == 1) {
            const double last_r = std::max(r_free + tile, with_r);
            cost = rounds_us(total, {others, r_pairs - r_last, r_last, 0},
                             {std::max(tile, with_r), std::max(r_item + tile, with_r), last_r, 0.0}, tile);
            if (r_last > 0 && total > others) cost = std::max(cost, last_r);
          } else if (f == 0) {
            const int last = compute_r ? others / ks : 0;
            cost = std::max(with_r, rounds_us(tail * ks, {others - last, last, r_pairs - r_last, r_last},
                                              {slice, std::max(slice, with_r), r_item + slice, r_free + slice}, slice));
            if (r_last > 0 && tail * ks > others) cost = std::max(cost, r_free + slice);
            cost += sum_us(pl.N, ks, false);
          } else {
            // (slices are added up while pairs that began with r are in their tiles; short ones help where both are through together)
            const double first = std::max(tile, with_r), after_r = std::max(r_item + tile, with_r);
            const double last_r = std::max(r_free + tile, with_r);
            cost = (f - 1) * tile + 0.05 * slice +
                   std::max(r_last > 0 ? last_r : first,
                            rounds_us(tail * ks, {others, r_pairs - r_last, r_last, 0},
                                      {first + slice, after_r + slice, last_r + slice, 0.0}, slice) + sum_us(pl.N, ks, true));
          }
          // (where r is not what the launch waits for, it had better be ready early all the same: the plans differ by a few per cent)
          cost += 0.04 * r_ready + (items > pairs ? kTicketUs : 0.0) + (two ? 0.0026 * pl.N : 0.0);   // (the last epilogue)
          if (cost < best_cost) {
            best_cost = cost;
            best = pl;
            best.r_slices = rks;
            best.ksplit = ks;
            best.full_tiles = ks > 1 ? full : total;
            best.n_tail = ks > 1 ? tail : 0;
            best.nbuf = two ? 2 : 1;
            best.off_slots = kWsSlotsOffset + r_bytes;
            best.end = best.off_slots + (ks > 1 ? tile_bytes * tail * ks : 0);
          }
        }
      }
    }
  }
  const int stage = best.N * 128;
  const int left = kSmemMax - 2048 - kTeams * kNP * (kPStage + kMeta);
  // At least as many activation stages as teams (a team waits for the MMAs of every second step, and a parity wait must not be able
  // to meet the phase before the last) and as A stages (the barrier of a step is that of the step nb before, which must be done).
  best.nb = std::max(3, std::min(6, (left - (best.N > 192 ? 16 : 24) * kOStage) / stage));
  best.no = std::min(kMaxO, (left - best.nb * stage) / (4 * kOStage));
  best.na = std::min({4, (kTmemCols - std::max(best.nbuf, sep ? 2 : 1) * best.N) / 64, best.nb});
  return best;
}

}  // namespace

// (host arithmetic: see glowq_internal_workspace_map)
void gemm_pair_workspace_map(const glowq_w4a16_group_t& g, bool compute_r, bool any_corr, bool any_separate, int sms, WorkspaceMap* map) {
  const PairPlan pl = make_pair_plan(g, compute_r, any_corr, any_separate, sms);
  map->kernel = 2;
  map->ksplit = pl.ksplit;
  map->whole_tiles = pl.full_tiles;
  map->sliced_tiles = pl.n_tail;
  map->r_ctas = 2 * pl.r_tiles * pl.r_slices;
  map->shortest = pl.nk_min;
  const int ctrs = 2 * ((pl.r_slices > 1 ? pl.r_tiles : 0) + pl.n_tail);
  if (ctrs > 0) {
    map->ctr_begin = kWsTileCtrOffset;
    map->ctr_end = kWsTileCtrOffset + static_cast<size_t>(ctrs) * 4;
  }
  map->slots_begin = kWsSlotsOffset;
  map->slots_end = pl.end;
}

// Members' products and corrections of a group call.  compute_r: r into g.r_buf as well (else it is there).  r_only: nothing
// but r (workspaces without room for the counters that order r and the members in one launch).
int gemm_pair_forward(const glowq_w4a16_group_t& g, bool compute_r, bool r_only, bool any_corr, bool any_separate, int sms,
                      cudaStream_t stream, cudaError_t* cuda_err) {
  const int G = cdiv(g.IC, kGroup);
  const PairPlan pl = make_pair_plan(g, compute_r, any_corr, any_separate, sms);
  unsigned char* const ws = static_cast<unsigned char*>(g.workspace);
  PtParams p{};
  p.status = reinterpret_cast<uint32_t*>(ws) + WS_STATUS;
  const bool have_ctr = g.workspace_bytes >= kWsRllOffset;
  p.ctr = have_ctr ? reinterpret_cast<uint32_t*>(ws + kWsHeaderBytes) : nullptr;
  p.tile_ctr = reinterpret_cast<uint32_t*>(ws + kWsTileCtrOffset);
  p.r_slots = reinterpret_cast<float*>(ws + kWsSlotsOffset);
  p.slots = reinterpret_cast<float*>(ws + pl.off_slots);
  p.M = g.M;
  p.G = G;
  p.N = pl.N;
  p.rank = g.rank;
  p.out_fp32 = g.out_dtype == GLOWQ_OUT_F32;
  p.n_members = g.n_members;
  p.nbuf = pl.nbuf;
  p.nb = pl.nb;
  p.na = pl.na;
  p.no = pl.no;
  p.sep = any_separate;
  p.n_x = pl.n_x;
  p.n_y = pl.n_y;
  p.n_tiles = pl.n_tiles;
  p.band = 8;
  p.full_tiles = pl.full_tiles;
  p.n_tail = pl.n_tail;
  p.ksplit = pl.ksplit;
  p.r_x = std::max(1, pl.r_x);
  p.r_slices = pl.r_slices;
  if (compute_r) {
    p.r_tiles = pl.r_tiles;
    p.n_r = pl.r_tiles * pl.r_slices;
    p.ctr_base = pl.r_slices > 1 ? pl.r_tiles : 0;
  }
  p.n_items = p.n_r + (r_only ? 0 : pl.full_tiles + pl.n_tail * pl.ksplit);
  PtMaps tm;
  std::memset(&tm, 0, sizeof(tm));
  int rc;
  if ((rc = tensor_map_2d_ex(&tm.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.x, g.IC, g.M, static_cast<uint64_t>(g.x_stride) * 2, 64,
                             p.N / 2, 1)))
    return rc;
  tm.r = tm.R = tm.r_out = tm.x;
  if (compute_r && (rc = tensor_map_2d_ex(&tm.r_out, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.r_buf, g.rank, g.M,
                                          static_cast<uint64_t>(g.rank) * 2, 32, 32, 3)))
    return rc;
  if (compute_r && (rc = tensor_map_2d_ex(&tm.R, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.R, g.IC, g.rank,
                                          static_cast<uint64_t>(g.R_stride) * 2, 32, kRows, 3)))
    return rc;
  if (any_corr && (rc = tensor_map_2d_ex(&tm.r, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, g.r_buf, g.rank, g.M,
                                         static_cast<uint64_t>(g.rank) * 2, 64, p.N / 2, 1)))
    return rc;
  int begin[kMaxMembers];
  member_tiles(g, any_corr, any_separate, begin);
  for (int i = 0; i < g.n_members; ++i) {
    const auto& m = g.members[i];
    const bool corr = any_corr && m.L && m.alpha != 0.f;
    if ((rc = tensor_map_2d_ex(&tm.w[i], CU_TENSOR_MAP_DATA_TYPE_INT32, m.qweight, static_cast<uint64_t>(G) * 16, m.OC,
                               static_cast<uint64_t>(m.weight_stride_i32) * 4, 16, kRows, 3)))
      return rc;
    tm.l[i] = tm.w[i];
    if (corr && (rc = tensor_map_2d_ex(&tm.l[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, m.L, g.rank, m.OC,
                                       static_cast<uint64_t>(m.L_stride) * 2, 32, kRows, 3)))
      return rc;
    PtMember& d = p.mem[i];
    const size_t pitch = static_cast<size_t>(m.out_stride) * (p.out_fp32 ? 4 : 2);
    d.out_tma = ((reinterpret_cast<uintptr_t>(m.out) | pitch) & 15u) == 0;
    tm.out[i] = tm.x;
    if (d.out_tma &&
        (rc = tensor_map_2d_ex(&tm.out[i], p.out_fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, m.out, m.OC,
                               g.M, pitch, 32, p.out_fp32 ? 16 : 32, p.out_fp32 ? 0 : 3)))
      return rc;
    d.scales = static_cast<const __half*>(m.scales);
    d.qzeros = m.qzeros;
    d.bias = static_cast<const __half*>(m.bias);
    d.out = m.out;
    d.OC = m.OC;
    d.corr = corr;
    // groups per load of the scales: what divides a row, its pitch and the address
    d.svec = 8;
    while (d.svec > 1 && ((G | m.scale_stride) % d.svec != 0 || reinterpret_cast<uintptr_t>(m.scales) % (2 * d.svec) != 0)) d.svec >>= 1;
    d.sstride = m.scale_stride;
    d.zstride = m.zero_stride_i32;
    d.out_stride = m.out_stride;
    d.alpha = m.alpha;
    d.tile_begin = begin[i];
  }
  const int pairs = std::max(1, sms / 2);
  p.tickets = have_ctr && p.n_items > pairs;
  const size_t smem = 2048 + static_cast<size_t>(p.nb) * p.N * 128 + kTeams * kNP * (kPStage + kMeta) + 4 * p.no * kOStage;
  const cudaError_t e = launch(p, tm, p.tickets ? pairs : p.n_items, smem, stream);
  if (e != cudaSuccess) {
    *cuda_err = e;
    return GLOWQ_ERR_CUDA;
  }
  return GLOWQ_OK;
}

}  // namespace glowq
