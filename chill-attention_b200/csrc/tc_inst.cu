// Instantiates the tensor-core kernels for ONE mask functor: compile with
//   -DCHILL_INST_MASK=<functor struct>   (e.g. CausalMask)
#include "bwd_fused64.cuh"
#include "bwd_tc.cuh"
#include "bwd_tf32.cuh"
#include "bwd_wide.cuh"
#include "fwd_tc.cuh"
#include "fwd_tf32.cuh"
#include "tc_launch.h"

#ifndef CHILL_INST_MASK
#error "define CHILL_INST_MASK"
#endif

namespace chill {

using InstMask = CHILL_INST_MASK;

template <typename T, int D, int NS>
static int launch_fwd_one(const CUtensorMap* maps, const tc::FwdTcParams& p, dim3 grid, cudaStream_t st) {
  auto kern = tc::fwd_tc_kernel<T, D, InstMask, NS>;
  using SH = tc::FwdShape<D, NS>;
  constexpr int smem = tc::FwdSmem<D, SH::kStages, SH::kKeys, NS>::kDynamic;
  static_assert(SH::kCtasPerSm * smem <= 232448, "the CTAs that are to share an SM must fit its shared memory");
  struct Tag {};
  cudaError_t e = ensure_dynamic_smem<Tag>(kern, smem, /*prefer_max_carveout=*/true);
  if (e != cudaSuccess) return (int)e;
  kern<<<grid, SH::kThreads, smem, st>>>(maps[0], maps[1], maps[2], maps[3], p);
  return (int)cudaGetLastError();
}

template <>
bool tc_fwd_two_streams<InstMask>(const Geo& g, int D) {
  const long long ctas = (long long)((g.Lq + tc::kTile - 1) / tc::kTile) * g.H * g.B;
  return D <= 128 && ctas <= 0x7fffffffll && tc::fwd_two_streams<InstMask>(g, D, (int)ctas);
}

template <typename T>
static int launch_fwd_dim(int D, const CUtensorMap* maps, const tc::FwdTcParams& p, dim3 grid, cudaStream_t st) {
  const bool two = tc_fwd_two_streams<InstMask>(p.g, D);
  if (D == 128) return two ? launch_fwd_one<T, 128, 2>(maps, p, grid, st) : launch_fwd_one<T, 128, 1>(maps, p, grid, st);
  if (D == 64) return two ? launch_fwd_one<T, 64, 2>(maps, p, grid, st) : launch_fwd_one<T, 64, 1>(maps, p, grid, st);
  if (D == 256) return launch_fwd_one<T, 256, 1>(maps, p, grid, st);
  return (int)cudaErrorInvalidValue;
}

template <>
int tc_launch_fwd<InstMask>(int dtype, int D, const CUtensorMap* maps, const tc::FwdTcParams& p, dim3 grid,
                            cudaStream_t st) {
  if (dtype == 2) return launch_fwd_dim<__nv_bfloat16>(D, maps, p, grid, st);
  if (dtype == 1) return launch_fwd_dim<__half>(D, maps, p, grid, st);
  return (int)cudaErrorInvalidValue;
}

template <int D>
static int launch_fwd_tf32_one(const CUtensorMap* maps, const tc::FwdTcParams& p, dim3 grid, cudaStream_t st) {
  auto kern = tc::fwd_tf32_kernel<D, InstMask>;
  constexpr int smem = tc::FwdTf32Smem<D>::kDynamic;
  static_assert(smem <= 232448, "exceeds the 227 KB of shared memory a CTA can opt in to");
  struct Tag {};
  cudaError_t e = ensure_dynamic_smem<Tag>(kern, smem, /*prefer_max_carveout=*/true);
  if (e != cudaSuccess) return (int)e;
  kern<<<grid, tc::kFwdThreads, smem, st>>>(maps[0], maps[1], maps[2], maps[3], p);
  return (int)cudaGetLastError();
}

template <>
int tc_launch_fwd_tf32<InstMask>(int D, const CUtensorMap* maps, const tc::FwdTcParams& p, dim3 grid, cudaStream_t st) {
  if (D == 64) return launch_fwd_tf32_one<64>(maps, p, grid, st);
  if (D == 128) return launch_fwd_tf32_one<128>(maps, p, grid, st);
  return (int)cudaErrorInvalidValue;
}

template <>
int tc_launch_bwd_tf32<InstMask>(int D, const CUtensorMap* maps, const tc::BwdTcParams& p, cudaStream_t st) {
  return tc::launch_bwd_tf32<InstMask>(D, maps, p, st);
}

template <>
int tc_launch_bwd<InstMask>(int dtype, int D, const CUtensorMap* maps, const tc::BwdTcParams& p, cudaStream_t st) {
  if (p.dq_accum != nullptr) return tc::launch_bwd_fused_all<InstMask>(dtype, D, maps, p, st);
  return tc::launch_bwd_all<InstMask>(dtype, D, maps, p, st);
}

template <>
bool tc_bwd_short_loops<InstMask>(const Geo& g, int D) {
  return tc::bwd_short_loops<InstMask>(g, D);
}

template <>
int tc_launch_bwd_wide<InstMask>(int dtype, const CUtensorMap* maps, const tc::BwdTcParams& p, cudaStream_t st) {
  return tc::launch_bwd_wide_all<InstMask>(dtype, maps, p, st);
}

}  // namespace chill
