// What every kernel shares: tensor references, call geometry, scalar conversions; and the kernels that are not attention
// itself: delta (chill_attention/utils.py:93-217) and the tabulation of a mask functor.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math_constants.h>

#include "masks.cuh"

namespace chill {

struct TRef {
  void* p;
  long long sb, sh, sl, sd;  // element strides of [batch][head][position][channel]
};

struct Geo {
  int B, H, Hkv, Lq, Lk, D;
  int q_off, k_off, seq_len;
  float scale;
  const int* lens;
  MaskArgs margs;
};

struct FwdP {
  Geo g;
  TRef q, k, v, o;
  float* lse;
  long long lse_sb, lse_sh, lse_sl;
};

// Optional fp32 copies of the un-rounded dK (times sm_scale) and dV for the first `head` and the last `tail` key
// rows of a call: key row j < head is part row j, key row j >= Lk - tail is part row head + j - (Lk - tail).
struct PartOut {
  float *dk = nullptr, *dv = nullptr;
  long long sb = 0, sh = 0, sl = 0;  // element strides of [batch][kv head][part row]; channels are contiguous
  int head = 0, tail = 0;
  // address of the part row of key row j in tensor `t` (dk or dv), or nullptr if the row is outside both windows
  __device__ __forceinline__ float* row(float* t, int b, int hk, int j, int Lk) const {
    if (t == nullptr || j >= Lk) return nullptr;
    int pr;
    if (j < head) pr = j;
    else if (j >= Lk - tail) pr = head + j - (Lk - tail);
    else return nullptr;
    return t + b * sb + hk * sh + pr * sl;
  }
};

struct BwdP {
  Geo g;
  TRef q, k, v, o, d_o, dq, dk, dv;
  const float* lse;
  long long lse_sb, lse_sh, lse_sl;
  float* delta;  // contiguous [B][H][Lq]
  PartOut part;
};

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kGenericWarps = 4;
constexpr int kMaxD = 256;

__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(__half x) { return __half2float(x); }
__device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
template <typename T>
__device__ __forceinline__ T from_f(float x);
template <>
__device__ __forceinline__ float from_f<float>(float x) { return x; }
template <>
__device__ __forceinline__ __half from_f<__half>(float x) { return __float2half_rn(x); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

template <typename T>
__device__ __forceinline__ const T* row_ptr(const TRef& t, int b, int h, int l) {
  return reinterpret_cast<const T*>(t.p) + b * t.sb + h * t.sh + l * t.sl;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

__device__ __forceinline__ int valid_len(const Geo& g, int b) {
  int n = g.seq_len;
  if (g.lens != nullptr) n = imin(n, g.lens[b]);
  return n;
}

// Steps of ROWS queries x 64 keys of a call, over all heads: `total`, and the most a tile of queries has (for the rules that choose
// between kernels).  At most 32 tiles are looked at (four where a tile's range takes a loop over its rows); lens is not known here.
template <class M, int ROWS = 128>
void count_steps(const Geo& g, long long& total, int& most) {
  constexpr int kRows = ROWS, kCols = 64, kLooks = M::kKLimsContinuous ? 32 : 4;
  const int n_rt = (g.Lq + kRows - 1) / kRows, every = (n_rt + kLooks - 1) / kLooks;
  long long sum = 0, looks = 0;
  most = 0;
  for (int t = n_rt - 1; t >= 0; t -= every, ++looks) {
    int lo, hi;
    tile_range<M, true>(t * kRows + g.q_off, imin(kRows, g.Lq - t * kRows), g.seq_len, g.margs, lo, hi);
    lo = imax(lo - g.k_off, 0);
    hi = imin(imin(hi, g.seq_len - 1) - g.k_off, g.Lk - 1);
    const int n = hi >= lo ? (hi - lo) / kCols + 1 : 0;
    sum += n;
    most = imax(most, n);
  }
  total = sum * n_rt / looks * g.B * g.H;
}

// --------------------------------------------------------------------------------- delta
// delta[b,h,t] = sum_d O*dO in fp32; one warp per row, every row (no `lens`), like the reference.
template <typename T>
__global__ void __launch_bounds__(kGenericWarps * 32) delta_kernel(TRef o, TRef d_o, float* delta, int H, int Lq, int D,
                                                                   const float* dlse, long long dl_sb, long long dl_sh, long long dl_sl) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * kGenericWarps + warp;
  const int h = blockIdx.y, b = blockIdx.z;
  if (row >= Lq) return;
  const T* orow = row_ptr<T>(o, b, h, row);
  const T* drow = row_ptr<T>(d_o, b, h, row);
  float acc = 0.f;
  for (int d = lane; d < D; d += 32) acc = fmaf(to_f(orow[d * o.sd]), to_f(drow[d * d_o.sd]), acc);
  acc = warp_sum(acc);
  if (dlse != nullptr) acc -= kLog2e * dlse[b * dl_sb + h * dl_sh + row * dl_sl];  // gradient through the returned LSE
  if (lane == 0) delta[((long long)b * H + h) * Lq + row] = acc;
}

// Contiguous 16-bit rows of 16, 32, 64 or 128 channels: 2, 4, 8 or 16 lanes x 16 B cover one
// row, so a warp streams 16 to 2 rows per step.  Bandwidth-bound: 2 reads of B*H*L*D elements.
template <typename T, int D>
__global__ void __launch_bounds__(256) delta_rows16_kernel(const T* __restrict__ o, const T* __restrict__ d_o,
                                                           float* __restrict__ delta, long long o_sb, long long o_sh,
                                                           long long o_sl, long long do_sb, long long do_sh,
                                                           long long do_sl, int H, int Lq, const float* __restrict__ dlse,
                                                           long long dl_sb, long long dl_sh, long long dl_sl) {
  constexpr int LPR = D / 8;  // lanes per row
  constexpr int RPW = 32 / LPR;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / LPR, li = lane % LPR;
  const int h = blockIdx.y, b = blockIdx.z;
  const int row = (blockIdx.x * 8 + warp) * RPW + sub;
  float acc = 0.f;
  if (row < Lq) {
    const uint4 a = *reinterpret_cast<const uint4*>(o + b * o_sb + h * o_sh + row * o_sl + li * 8);
    const uint4 c = *reinterpret_cast<const uint4*>(d_o + b * do_sb + h * do_sh + row * do_sl + li * 8);
    const T* pa = reinterpret_cast<const T*>(&a);
    const T* pc = reinterpret_cast<const T*>(&c);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc = fmaf(to_f(pa[i]), to_f(pc[i]), acc);
  }
#pragma unroll
  for (int ofs = LPR / 2; ofs > 0; ofs >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, ofs);
  if (row < Lq && li == 0) {
    if (dlse != nullptr) acc -= kLog2e * dlse[b * dl_sb + h * dl_sh + row * dl_sl];  // gradient through the returned LSE
    delta[((long long)b * H + h) * Lq + row] = acc;
  }
}

// ----------------------------------------------------------------------- mask tabulation
template <class M>
__global__ void mask_tabulate_kernel(MaskArgs a, int n, int tile, uint8_t* dense, int* k_lims, int* q_lims,
                                     int* k_full, int* q_full) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (dense != nullptr && idx < (long long)n * n) {
    const int q = (int)(idx / n), k = (int)(idx % n);
    dense[idx] = M::mask(q, k, n, a) ? 1 : 0;
  }
  if (idx < n) {
    int lo, hi;
    if (k_lims != nullptr) {
      M::k_range_for_q((int)idx, n, a, lo, hi);
      k_lims[2 * idx] = lo;
      k_lims[2 * idx + 1] = hi;
    }
    if (q_lims != nullptr) {
      M::q_range_for_k((int)idx, n, a, lo, hi);
      q_lims[2 * idx] = lo;
      q_lims[2 * idx + 1] = hi;
    }
  }
  const int ntiles = (n + tile - 1) / tile;
  if (idx < ntiles) {
    int lo, hi;
    if (k_full != nullptr) {
      M::k_full_range_for_q((int)idx * tile, tile, n, a, lo, hi);
      k_full[2 * idx] = lo;
      k_full[2 * idx + 1] = hi;
    }
    if (q_full != nullptr) {
      M::q_full_range_for_k((int)idx * tile, tile, n, a, lo, hi);
      q_full[2 * idx] = lo;
      q_full[2 * idx + 1] = hi;
    }
  }
}

template <class M>
__global__ void mask_tabulate_blocks_kernel(MaskArgs a, int n, int q_tile, int k_tile, uint8_t* full) {
  const int nq = (n + q_tile - 1) / q_tile, nk = (n + k_tile - 1) / k_tile;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < (long long)nq * nk) {
    const int qi = (int)(idx / nk), ki = (int)(idx % nk);
    full[idx] = M::is_full_block(qi * q_tile, ki * k_tile, q_tile, k_tile, n, a) ? 1 : 0;
  }
}

}  // namespace chill
