// Instantiates the CUDA-core kernels for ONE mask functor: compile with -DCHILL_INST_MASK=<functor struct>
#include "simt.cuh"
#include "split.cuh"
#include "tc_launch.h"

#ifndef CHILL_INST_MASK
#error "define CHILL_INST_MASK"
#endif

namespace chill {

using InstMask = CHILL_INST_MASK;

namespace simt {

// Rows of a CTA's tile = 8 * RT.  The large tile is the one whose accumulators still leave two CTAs per SM; the small one
// (RT = 2) trades shared-memory traffic per FMA for more CTAs and is taken when the large tiles would leave more than half
// of the SMs without work: (1, 2, 128, 64) 10.6 us forward and 14.5 us backward against 20.6 and 30.5 with the large
// tile; (2, 8, 512, 64), 128 large tiles: 61.6 and 176 us against 57.5 and 119.
constexpr int fwd_rows(int DP) { return DP <= 128 ? 8 : 4; }
constexpr int bwd_rows(int DP) { return DP <= 64 ? 8 : (DP == 128 ? 4 : 2); }

template <int DP, int RT, bool kRepair = false>
static int fwd_one(const FwdParams& p, cudaStream_t st) {
  auto kern = simt_fwd_kernel<DP, RT, InstMask, kRepair>;
  constexpr int smem = FwdSmem<DP, RT>::kBytes;
  static_assert(smem <= 232448, "exceeds the 227 KB of shared memory a CTA can opt in to");
  struct Tag {};
  cudaError_t e = ensure_dynamic_smem<Tag>(kern, smem, /*prefer_max_carveout=*/true);
  if (e != cudaSuccess) return (int)e;
  const Geo& g = p.f.g;
  dim3 grid((unsigned)((g.Lq + 8 * RT - 1) / (8 * RT)), (unsigned)g.H, (unsigned)g.B);
  kern<<<grid, kThreads, smem, st>>>(p);
  return (int)cudaGetLastError();
}

template <int DP>
static int fwd_dim(const FwdParams& p, cudaStream_t st) {
  constexpr int RT = fwd_rows(DP);
  const Geo& g = p.f.g;
  if constexpr (DP <= 64) {  // the head dims of split.cuh
    if (p.repair) return fwd_one<DP, RT, true>(p, st);
  }
  const long long ctas = (long long)((g.Lq + 8 * RT - 1) / (8 * RT)) * g.H * g.B;
  if (2 * ctas < sm_count()) return fwd_one<DP, 2>(p, st);
  return fwd_one<DP, RT>(p, st);
}

template <int DP, int RT, bool kRepair = false>
static int bwd_one(BwdParams p, int which, cudaStream_t st) {
  auto kern = simt_bwd_kernel<DP, RT, InstMask, kRepair>;
  constexpr int smem = BwdSmem<DP, RT>::kBytes;
  static_assert(smem <= 232448, "exceeds the 227 KB of shared memory a CTA can opt in to");
  struct Tag {};
  cudaError_t e = ensure_dynamic_smem<Tag>(kern, smem, /*prefer_max_carveout=*/true);
  if (e != cudaSuccess) return (int)e;
  const Geo& g = p.b.g;
  const long long nk = (which & 1) ? (long long)((g.Lk + 8 * RT - 1) / (8 * RT)) * g.Hkv * g.B : 0;
  const long long nq = (which & 2) ? (long long)((g.Lq + 8 * RT - 1) / (8 * RT)) * g.H * g.B : 0;
  if (nk + nq > 0x7fffffffll) return (int)cudaErrorInvalidConfiguration;
  p.n_key_ctas = (int)nk;
  kern<<<(unsigned)(nk + nq), kThreads, smem, st>>>(p);
  return (int)cudaGetLastError();
}

template <int DP>
static int bwd_dim(const BwdParams& p, int which, cudaStream_t st) {
  constexpr int RT = bwd_rows(DP);
  if constexpr (DP <= 64) {
    if (p.repair) return bwd_one<DP, RT, true>(p, which, st);
  }
  if constexpr (RT > 2) {
    const Geo& g = p.b.g;
    const long long ctas = (long long)((g.Lk + 8 * RT - 1) / (8 * RT)) * g.Hkv * g.B + (long long)((g.Lq + 8 * RT - 1) / (8 * RT)) * g.H * g.B;
    if (2 * ctas < sm_count()) return bwd_one<DP, 2>(p, which, st);
  }
  return bwd_one<DP, RT>(p, which, st);
}

}  // namespace simt

template <>
int split_launch_fwd<InstMask>(const split::FwdParams& p, cudaStream_t st) {
  auto kern = split::split_fwd_kernel<InstMask>;
  constexpr int smem = split::FwdSmem::kDynamic;
  static_assert(smem <= 232448, "exceeds the 227 KB of shared memory a CTA can opt in to");
  struct Tag {};
  cudaError_t e = ensure_dynamic_smem<Tag>(kern, smem, /*prefer_max_carveout=*/true);
  if (e != cudaSuccess) return (int)e;
  const Geo& g = p.f.g;
  kern<<<dim3((unsigned)((g.Lq + split::kRows - 1) / split::kRows), (unsigned)g.H, (unsigned)g.B), split::kFwdThreads, smem, st>>>(p);
  return (int)cudaGetLastError();
}

template <>
int split_launch_bwd<InstMask>(split::BwdParams p, int which, cudaStream_t st) {
  auto kern = split::split_bwd_kernel<InstMask>;
  constexpr int smem = split::BwdSmem::kDynamic;
  static_assert(smem <= 232448, "exceeds the 227 KB of shared memory a CTA can opt in to");
  struct Tag {};
  cudaError_t e = ensure_dynamic_smem<Tag>(kern, smem, /*prefer_max_carveout=*/true);
  if (e != cudaSuccess) return (int)e;
  const Geo& g = p.b.g;
  const long long nk = (which & 1) ? (long long)((g.Lk + split::kRows - 1) / split::kRows) * g.Hkv * g.B : 0;
  const long long nq = (which & 2) ? (long long)((g.Lq + split::kRows - 1) / split::kRows) * g.H * g.B : 0;
  if (nk + nq > 0x7fffffffll) return (int)cudaErrorInvalidConfiguration;
  p.n_key_ctas = (int)nk;
  kern<<<(unsigned)(nk + nq), split::kBwdThreads, smem, st>>>(p);
  return (int)cudaGetLastError();
}

template <>
int simt_launch_fwd<InstMask>(const simt::FwdParams& p, cudaStream_t st) {
  const int D = p.f.g.D;
  if (D <= 32) return simt::fwd_dim<32>(p, st);
  if (D <= 64) return simt::fwd_dim<64>(p, st);
  if (D <= 128) return simt::fwd_dim<128>(p, st);
  if (D <= 256) return simt::fwd_dim<256>(p, st);
  return (int)cudaErrorInvalidValue;
}

template <>
int simt_launch_bwd<InstMask>(const simt::BwdParams& p, int which, cudaStream_t st) {
  const int D = p.b.g.D;
  if (D <= 32) return simt::bwd_dim<32>(p, which, st);
  if (D <= 64) return simt::bwd_dim<64>(p, which, st);
  if (D <= 128) return simt::bwd_dim<128>(p, which, st);
  if (D <= 256) return simt::bwd_dim<256>(p, which, st);
  return (int)cudaErrorInvalidValue;
}

}  // namespace chill
