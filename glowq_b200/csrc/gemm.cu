// Group calls on the tensor cores: what they accept, the scratch they use, and which kernel takes them.
//
//   Y[M, OC] = X[M, IC] . dequant(Q)^T  +  alpha * r[M, rank] . L[OC, rank]^T  (+ bias),     r = X . R^T
//
// Up to 64 tokens one CTA per 128 output columns (gemm_tmem.cu; up to 8 in its exact form), above a CTA pair per 256 (gemm_pair.cu).
// Both keep the dequantised weights in tensor memory, and both compute r inside the group launch.  The line lies where the first ends: two CTAs
// share an SM's tensor memory there, which leaves an accumulator 64 tokens (13B gate/up 45 us at 64 tokens; the pair form, whose
// tiles have 64 tokens at least, takes 14B gate/up at 65 tokens from 67 to 63 us).
#include <algorithm>

#include "../../include/glowq_w4a16.h"
#include "params.h"

namespace glowq {

// r = x . R^T for calls of up to 64 tokens whose workspace has no room for the slots of the in-launch form (r_product.cu).
size_t r_product_slot_bytes(int M, int IC, int rank);
cudaError_t launch_r_product(const __half* x, const __half* R, __half* r_buf, float* slots, uint32_t* ctr, int M, int IC,
                             int rank, int x_stride, int R_stride, cudaStream_t stream);
size_t gemm_tmem_r_bytes(int M, int IC, int rank);
size_t gemm_tmem_slot_bytes(int M, int IC, int OC_total, int rank, int n_members, int sms);
int gemm_tmem_forward(const glowq_w4a16_group_t& g, bool exact, bool compute_r, bool any_corr, bool any_separate, int sms,
                      cudaStream_t stream, cudaError_t* cuda_err);
int gemm_pair_forward(const glowq_w4a16_group_t& g, bool compute_r, bool r_only, bool any_corr, bool any_separate, int sms,
                      cudaStream_t stream, cudaError_t* cuda_err);
void gemm_tmem_workspace_map(const glowq_w4a16_group_t& g, bool exact, bool compute_r, bool any_corr, bool any_separate, int sms,
                             WorkspaceMap* map);
void gemm_pair_workspace_map(const glowq_w4a16_group_t& g, bool compute_r, bool any_corr, bool any_separate, int sms, WorkspaceMap* map);

namespace {
inline bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline int cdiv(int a, int b) { return (a + b - 1) / b; }
}  // namespace

bool gemm_supported(const glowq_w4a16_group_t& g) {
  if (g.group_size != kGroup || g.M < 1) return false;
  if (!al16(g.x) || (g.x_stride & 7) || (g.IC & 7)) return false;
  const int G = (g.IC + kGroup - 1) / kGroup;
  for (int i = 0; i < g.n_members; ++i) {
    const auto& m = g.members[i];
    if (m.weight_stride_i32 < G * 16 || (m.weight_stride_i32 & 3) || !al16(m.qweight)) return false;
    if (g.r_mode != GLOWQ_R_NONE && m.L && (!al16(m.L) || (m.L_stride & 7))) return false;
  }
  if (g.r_mode != GLOWQ_R_NONE && ((g.rank & 7) || !al16(g.r_buf))) return false;
  if (g.r_mode == GLOWQ_R_COMPUTE && (!al16(g.R) || (g.R_stride & 7))) return false;
  return true;
}

// Scratch behind kWsSlotsOffset, planned for 148 SMs so that its size does not depend on the device.  The kernels' planners take the
// slices that the room allows.
constexpr int kPlanSms = 148;
constexpr int kTmemMaxM = 64;                  // tokens up to which a CTA of its own takes a tile (gemm_tmem.cu)
constexpr int kTmemSlices = 304;               // its K slices at most (two CTAs per SM), a tile of 32 or 64 tokens x 128 fp32 each
constexpr int kMaxTailSlots = 64;              // slots of 256 x 256 fp32 above 256 tokens
constexpr size_t kSlotBytes = 128 * 128 * 4;   // a 128 x 128 block of partial sums

// Slots of r: up to 16 K slices of its 128 x 128 blocks.
inline size_t r_slot_bytes(int M, int IC, int rank) {
  const int tiles = cdiv(rank, 128) * cdiv(M, 128);
  if (tiles > 64) return 0;
  const int ks = std::max(1, std::min({16, cdiv(IC, 64) / 4, 128 / tiles}));
  return ks > 1 ? static_cast<size_t>(ks) * tiles * kSlotBytes : 0;
}
// Slots of the members' K slices where the tiles do not fill the SMs (9 to 256 tokens; the one-CTA form's are counted below).
inline size_t main_slot_bytes(int M, int OC_total, int n_members) {
  // (up to 8 tokens only the one-CTA form comes here)
  const int m_tiles = cdiv(M, 128);
  if (M <= 8 || M > 256 || cdiv(OC_total, 256) * m_tiles * 2 > kPlanSms) return 0;
  const int tiles = (cdiv(OC_total, 128) + n_members) * m_tiles;
  return static_cast<size_t>(std::min(8 * tiles, 2 * kPlanSms + tiles)) * std::min(128, cdiv(M, 32) * 32) * 128 * 4;
}

size_t gemm_workspace_bytes(int M, int IC, int OC_total, int rank, int n_members) {
  size_t slots = std::max(rank > 0 ? r_slot_bytes(M, IC, rank) : 0, main_slot_bytes(M, OC_total, n_members));
  // r in a launch of its own (up to 64 tokens); up to 128 the room serves the pairs' slots, which for long rows it lets slice K finer
  if (rank > 0 && M <= 128) slots = std::max(slots, r_product_slot_bytes(M, IC, rank));
  // K slices of the one-CTA form: what its plan takes up to 8 tokens (304 slots for every call were 11.0 MB for a layer of the 13B shapes,
  // now 8.8); above, unless whole tiles fill the SMs and the last round of them is nearly full too
  const int tmem_tiles = cdiv(OC_total, 128), tmem_rest = tmem_tiles % kPlanSms;
  if (M > 1 && M <= 8)
    slots = std::max(slots, gemm_tmem_slot_bytes(M, IC, OC_total, rank, n_members, kPlanSms));
  else if (M > 8 && M <= kTmemMaxM && !(tmem_tiles >= kPlanSms && tmem_rest * 4 >= 3 * kPlanSms))
    slots = std::max(slots, static_cast<size_t>(kTmemSlices) * (M <= 32 ? 32 : 64) * 128 * 4);
  if (M > 256) slots = std::max(slots, static_cast<size_t>(kMaxTailSlots) * 4 * kSlotBytes);
  if (rank > 0 && M > 1 && M <= kTmemMaxM) slots += gemm_tmem_r_bytes(M, IC, rank);
  if (slots == 0) return kWsHeaderBytes;
  return kWsSlotsOffset + slots + 256;
}

namespace {
// What the routes of a group call hang on.
struct GemmRoute {
  bool any_corr, any_separate;   // some member is corrected; with a factor other than 1 (an accumulator of its own)
  bool exact;                    // up to 8 tokens, chosen by the library: integer weights and fp32 scales (gemm_tmem.cu)
  bool tmem, r_in_launch;        // up to 64 tokens (gemm_tmem.cu); r computed by the members' launch
};
GemmRoute gemm_route(const glowq_w4a16_group_t& g) {
  GemmRoute rt{};
  for (int i = 0; i < g.n_members && g.r_mode != GLOWQ_R_NONE; ++i) {
    const bool corr = g.members[i].L && g.members[i].alpha != 0.f;
    rt.any_corr = rt.any_corr || corr;
    rt.any_separate = rt.any_separate || (corr && g.members[i].alpha != 1.f);
  }
  rt.exact = g.M <= 8 && g.kernel == GLOWQ_KERNEL_AUTO;
  rt.tmem = g.M <= kTmemMaxM;
  rt.r_in_launch = g.r_mode == GLOWQ_R_COMPUTE &&
                   g.workspace_bytes >= (rt.tmem ? kWsSlotsOffset + gemm_tmem_r_bytes(g.M, g.IC, g.rank) : kWsRllOffset);
  return rt;
}
}  // namespace

double gemm_tmem_exact_us(const glowq_w4a16_group_t& g, bool compute_r, bool any_corr, int sms);

// Microseconds of a call of up to 8 tokens in the exact form, as far as its workspace goes (-1: r would need a launch of its own).
double gemm_exact_us(const glowq_w4a16_group_t& g, int sms) {
  const GemmRoute rt = gemm_route(g);
  if (g.r_mode == GLOWQ_R_COMPUTE && !rt.r_in_launch) return -1.0;
  return gemm_tmem_exact_us(g, rt.r_in_launch, rt.any_corr, sms);
}

// (host arithmetic: see glowq_internal_workspace_map)
void gemm_workspace_map(const glowq_w4a16_group_t& g, int sms, WorkspaceMap* map) {
  const GemmRoute rt = gemm_route(g);
  if (rt.tmem) return gemm_tmem_workspace_map(g, rt.exact, rt.r_in_launch, rt.any_corr, rt.any_separate, sms, map);
  gemm_pair_workspace_map(g, rt.r_in_launch, rt.any_corr, rt.any_separate, sms, map);
}

int gemm_group_forward(const glowq_w4a16_group_t& g, cudaStream_t stream, cudaError_t* cuda_err) {
  if (g.workspace_bytes < kWsHeaderBytes) return GLOWQ_ERR_WORKSPACE_TOO_SMALL;
  const GemmRoute rt = gemm_route(g);
  int sms = kPlanSms, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (g.r_mode == GLOWQ_R_COMPUTE && !rt.r_in_launch) {
    // r in a launch of its own: the small one where there is room for its slots, else the pair form's r items alone
    const size_t need = r_product_slot_bytes(g.M, g.IC, g.rank);
    const size_t off = g.workspace_bytes >= need ? ((g.workspace_bytes - need) & ~static_cast<size_t>(255)) : 0;
    if (rt.tmem && off >= kWsSlotsOffset && cdiv(g.rank, 16) * cdiv(g.M, 64) <= kRpCtrWords) {
      unsigned char* ws = static_cast<unsigned char*>(g.workspace);
      const cudaError_t e = launch_r_product(static_cast<const __half*>(g.x), static_cast<const __half*>(g.R),
                                             static_cast<__half*>(g.r_buf), reinterpret_cast<float*>(ws + off),
                                             reinterpret_cast<uint32_t*>(ws + kWsHeaderBytes), g.M, g.IC, g.rank, g.x_stride,
                                             g.R_stride, stream);
      if (e != cudaSuccess) {
        *cuda_err = e;
        return GLOWQ_ERR_CUDA;
      }
    } else if (const int rc = gemm_pair_forward(g, true, true, rt.any_corr, rt.any_separate, sms, stream, cuda_err)) {
      return rc;
    }
  }
  if (rt.tmem) return gemm_tmem_forward(g, rt.exact, rt.r_in_launch, rt.any_corr, rt.any_separate, sms, stream, cuda_err);
  return gemm_pair_forward(g, rt.r_in_launch, false, rt.any_corr, rt.any_separate, sms, stream, cuda_err);
}

}  // namespace glowq
