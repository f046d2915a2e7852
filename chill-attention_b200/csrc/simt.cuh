// CUDA-core kernels (fp32 arithmetic): any dtype, any head dim <= 256, any strides.
//
// They serve every call the tensor-core kernels cannot take: fp32 tensors with IEEE precision (the default for fp32) where
// split.cuh does not pay (head dims above 64, little work) or cannot load them, 16-bit tensors whose layout TMA cannot
// describe, sm_scale <= 0.  Behind split.cuh they repeat the rows it has marked (`repair`).
//
//   simt_fwd_kernel   O, LSE            (reference math: chill_attention/chill_fwd.py:188-359)
//   simt_bwd_kernel   dK, dV and dQ     (chill_attention/chill_bwd_dkdv.py:15-277, chill_bwd_dq.py:15-229)
//
// Both are tiled matrix products.  A CTA of four warps owns a tile of 8 * RT rows (queries, or keys in the dK / dV part)
// and streams the other axis through shared memory in tiles of 64 positions.  A half-warp owns RT rows, a lane four
// of the 64 columns of the score tile and DP / 16 channels of the accumulators:
//
//   scores       s[RT][4] = A B^T: packed fp32 FMAs (two channels per instruction) on 16-byte shared-memory reads; the
//                RT rows of A are broadcast to the half-warp
//   accumulate   acc[RT][DP / 16] += W X: W (P or dS) goes through shared memory, but only between the lanes of one warp
//
// What bounds them is the FMA pipe (128 fp32 FMAs per clock and SM) as long as the shared-memory reads keep up: per
// 16 bytes x 4 channels a lane reads RT + 4 vectors for 8 * RT packed FMAs, i.e. RT = 8 needs half of the shared-memory
// bandwidth and RT = 4 three quarters of it.  Rows of 16-byte chunks are stored with the chunk index XORed by
// (row / 4) % 8, which makes the lanes' reads of four consecutive rows conflict-free (measured: 3 wavefronts per read).
//
// Measured, fp32 full mask (2, 8, 1000, 64): forward 143 us, dK / dV and dQ together 444 us, i.e. 29 / 32 TFLOP/s of the
// 74 that 148 SMs issue (one warp per output row and 32 positions per step, the form before: 4831 and 17126 us, every
// dot product re-reading its row of K or V from L1).  What is left is latency: 240 registers a thread leave eight
// warps on an SM, which keep the FMA pipe 50 % busy; RT = 4 doubles the warps and their shared-memory reads per FMA
// (forward 164-182 against 155 us when it was tried).
//
// What a row may not see does not reach it, whatever the value: padding enters the tiles as zeros, and see accumulate for
// what the mask hides.  The check of the accumulators and the second loop cost the backward 1 to 4 % (444 against 437 us) and
// the forward nothing; a probe of every tile for NaN and Inf as it is loaded cost both 2 to 6 %.
#pragma once
#include "generic.cuh"
#include "split.cuh"
#include "tc_common.cuh"

namespace chill {
namespace simt {

constexpr int kThreads = 128;  // four warps, eight half-warps of RT rows
constexpr int kCols = 64;      // positions of the streamed axis per step

struct BwdParams {
  BwdP b;
  int n_key_ctas;    // the first n_key_ctas CTAs compute dK / dV, the others dQ
  uint32_t vec;      // kVec*: tensors whose rows are read / written in 16-byte vectors (fp32 only)
  int dtype;
  bool repair = false;  // only rows that split.cuh has marked (kRepair)
};
struct FwdParams {
  FwdP f;
  uint32_t vec;
  int dtype;
  bool repair = false;
};
enum : uint32_t { kVecQ = 1, kVecK = 2, kVecV = 4, kVecO = 8, kVecDo = 16, kVecDq = 32, kVecDk = 64, kVecDv = 128 };

// Element access by run-time type (0 fp32, 1 fp16, 2 bf16, as in the C ABI): the arithmetic is fp32 whatever the tensors
// are, so one instantiation serves all three and only loads and stores look at the type.
__device__ __forceinline__ float load_elem(const void* p, long long i, int dtype) {
  if (dtype == 0) return static_cast<const float*>(p)[i];
  if (dtype == 1) return to_f(static_cast<const __half*>(p)[i]);
  return to_f(static_cast<const __nv_bfloat16*>(p)[i]);
}
__device__ __forceinline__ void store_elem(void* p, long long i, int dtype, float v) {
  if (dtype == 0) static_cast<float*>(p)[i] = v;
  else if (dtype == 1) static_cast<__half*>(p)[i] = from_f<__half>(v);
  else static_cast<__nv_bfloat16*>(p)[i] = from_f<__nv_bfloat16>(v);
}

// Rows of a half-warp whose fp32 result carries the mark of a row that split.cuh left to these kernels: bit i = row0 + i.
template <int RT>
__device__ __forceinline__ uint32_t marked(const TRef& t, int b, int h, int row0, int end) {
  uint32_t bits = 0;
#pragma unroll
  for (int i = 0; i < RT; ++i)
    if (row0 + i < end && __float_as_uint(static_cast<const float*>(t.p)[b * t.sb + h * t.sh + (row0 + i) * t.sl]) == kRepairMark) bits |= 1u << i;
  return bits;
}

__device__ __forceinline__ int swz(int row) { return (row >> 2) & 7; }

// One tile of ROWS x DP elements, starting at row `row0` of head h of batch row b, to shared memory as fp32; rows beyond
// rows_in (what does not exist or is padding, which may hold anything) and channels beyond D become zeros.
template <int DP, int ROWS>
__device__ __forceinline__ void load_tile(float* s, const TRef& t, int b, int h, int row0, int rows_in, int D, int dtype, bool vec) {
  constexpr int kChunks = DP / 4, kPerThread = ROWS * kChunks / kThreads;
  static_assert(ROWS * kChunks % kThreads == 0, "every thread moves the same number of chunks");
  constexpr int kBatch = kPerThread < 8 ? kPerThread : 8;  // loads in flight per thread
  const long long origin = b * t.sb + h * t.sh + row0 * t.sl;
#pragma unroll 1
  for (int i0 = 0; i0 < kPerThread; i0 += kBatch) {
    float4 v[kBatch];
    if (vec) {
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int idx = (i0 + i) * kThreads + threadIdx.x;
        const int row = idx / kChunks, c = idx % kChunks;
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < rows_in && c * 4 < D) v[i] = *reinterpret_cast<const float4*>(static_cast<const float*>(t.p) + origin + row * t.sl + c * 4);
      }
    } else {
#pragma unroll 1
      for (int i = 0; i < kBatch; ++i) {
        const int idx = (i0 + i) * kThreads + threadIdx.x;
        const int row = idx / kChunks, c = idx % kChunks;
        float e[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) e[k] = (row < rows_in && c * 4 + k < D) ? load_elem(t.p, origin + row * t.sl + (c * 4 + k) * t.sd, dtype) : 0.f;
        *reinterpret_cast<float4*>(s + row * DP + 4 * (c ^ swz(row))) = make_float4(e[0], e[1], e[2], e[3]);
      }
      continue;
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int idx = (i0 + i) * kThreads + threadIdx.x;
      const int row = idx / kChunks, c = idx % kChunks;
      *reinterpret_cast<float4*>(s + row * DP + 4 * (c ^ swz(row))) = v[i];
    }
  }
}

// s[i][j] = sum over channels of A[row0 + i][.] * B[4 * l16 + j][.]
template <int DP, int RT>
__device__ __forceinline__ void scores(const float* A, const float* B, int row0, int l16, float (&s)[RT][4]) {
  uint64_t acc[RT][4];
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  const float* bp = B + 4 * l16 * DP;
  const int fb = l16 & 7;                    // swz(4 * l16 + j)
  const int fa = swz(row0);                  // RT = 8: rows 4..7 of the half-warp are in the next group of four
#pragma unroll 4
  for (int c = 0; c < DP / 4; ++c) {
    ulonglong2 b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(bp + j * DP + 4 * (c ^ fb));
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(A + (row0 + i) * DP + 4 * (c ^ (fa + (i >> 2))));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = tc::ffma2(a.x, b[j].x, acc[i][j]);
        acc[i][j] = tc::ffma2(a.y, b[j].y, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lo, hi;
      tc::upk2(acc[i][j], lo, hi);
      s[i][j] = lo + hi;
    }
}

// Channels of one lane: DP / 16 of them as pairs.  DP >= 64: chunk c is the four channels at 4 * (l16 + 16 c);
// DP = 32: the two channels at 2 * l16.
template <int DP>
struct Lane {
  static constexpr int kPairs = DP / 32;
};

// The channels of one lane in row `row` of the streamed tile X (fx = swz(row)).
template <int DP>
__device__ __forceinline__ void lane_channels(const float* X, int row, int fx, int l16, uint64_t (&x)[Lane<DP>::kPairs]) {
  const float* xr = X + row * DP;
  if constexpr (DP == 32) {
    x[0] = *reinterpret_cast<const uint64_t*>(xr + 4 * ((l16 >> 1) ^ fx) + 2 * (l16 & 1));
  } else {
#pragma unroll
    for (int c = 0; c < DP / 64; ++c) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(xr + 4 * ((l16 + 16 * c) ^ fx));
      x[2 * c] = v.x;
      x[2 * c + 1] = v.y;
    }
  }
}

// acc[i][.] += sum over the 64 streamed positions of W[row0 + i][.] * X[.][channels of this lane]
//
// A hidden pair must add nothing, but 0 * NaN and 0 * Inf are NaN.  No NaN ever leaves an accumulator again, so a CTA that ends
// without one has met no such product; one that ends with a NaN repeats its work with `careful` set, which takes a loop that
// leaves the pairs out for which skip(row, position, weight) is true.
template <int DP, int RT, class Skip>
__device__ __forceinline__ void accumulate(const float* W, const float* X, int row0, int l16, uint64_t (&acc)[RT][Lane<DP>::kPairs], bool careful,
                                           const Skip& skip) {
  const int fa = swz(row0);
  if (careful) {
#pragma unroll 1
    for (int kx = 0; kx < kCols; ++kx) {
      uint64_t x[Lane<DP>::kPairs];
      lane_channels<DP>(X, kx, swz(kx), l16, x);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const float wk = W[(row0 + i) * kCols + 4 * ((kx >> 2) ^ (fa + (i >> 2))) + (kx & 3)];
        if (skip(i, kx, wk)) continue;
        const uint64_t w2 = tc::pk2(wk, wk);
#pragma unroll
        for (int pidx = 0; pidx < Lane<DP>::kPairs; ++pidx) acc[i][pidx] = tc::ffma2(w2, x[pidx], acc[i][pidx]);
      }
    }
    return;
  }
#pragma unroll 2
  for (int k4 = 0; k4 < kCols / 4; ++k4) {
    float4 w[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) w[i] = *reinterpret_cast<const float4*>(W + (row0 + i) * kCols + 4 * (k4 ^ (fa + (i >> 2))));
    const int fx = k4 & 7;  // swz of positions 4 * k4 .. 4 * k4 + 3
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint64_t x[Lane<DP>::kPairs];
      lane_channels<DP>(X, 4 * k4 + kk, fx, l16, x);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const float wk = kk == 0 ? w[i].x : (kk == 1 ? w[i].y : (kk == 2 ? w[i].z : w[i].w));
        const uint64_t w2 = tc::pk2(wk, wk);
#pragma unroll
        for (int pidx = 0; pidx < Lane<DP>::kPairs; ++pidx) acc[i][pidx] = tc::ffma2(w2, x[pidx], acc[i][pidx]);
      }
    }
  }
}

// Whether one of the accumulators is NaN (or two are opposite infinities).
template <int DP, int N>
__device__ __forceinline__ bool any_nan(const uint64_t (&acc)[N][Lane<DP>::kPairs]) {
  uint64_t sum[2] = {};
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int pidx = 0; pidx < Lane<DP>::kPairs; ++pidx) sum[(i + pidx) & 1] = tc::fadd2(sum[(i + pidx) & 1], acc[i][pidx]);
  float lo, hi;
  tc::upk2(tc::fadd2(sum[0], sum[1]), lo, hi);
  return lo + hi != lo + hi;
}

template <int DP>
__device__ __forceinline__ int pair_channel(int l16, int pidx) {
  return DP == 32 ? 2 * l16 : 4 * (l16 + 16 * (pidx >> 1)) + 2 * (pidx & 1);
}

// One row of accumulators, times `mul`, to element offset `off` of tensor p; a row of padding (`valid` false) is zero.
template <int DP>
__device__ __forceinline__ void store_row(void* p, long long off, long long sd, int D, int dtype, bool vec, int l16, const uint64_t* acc, float mul, bool valid) {
#pragma unroll
  for (int pidx = 0; pidx < Lane<DP>::kPairs; ++pidx) {
    float a, b;
    tc::upk2(acc[pidx], a, b);
    a = valid ? a * mul : 0.f;
    b = valid ? b * mul : 0.f;
    const int ch = pair_channel<DP>(l16, pidx);
    if (vec) {
      if (ch < D) *reinterpret_cast<float2*>(static_cast<float*>(p) + off + ch) = make_float2(a, b);
    } else {
      if (ch < D) store_elem(p, off + ch * sd, dtype, a);
      if (ch + 1 < D) store_elem(p, off + (ch + 1) * sd, dtype, b);
    }
  }
}

// Columns of one row of a boundary tile that the row may see: bit j = column 4 * l16 + j.
template <class M, bool KForQ>
__device__ __forceinline__ uint32_t visible4(int pos, int col0, int ncols, int l16, int n, const MaskArgs& margs) {
  uint32_t bits = 0;
  if constexpr (interval_rows<M>::value) {
    int lo, hi;
    row_window<M, KForQ>(pos, col0, ncols, n, margs, lo, hi);
#pragma unroll
    for (int j = 0; j < 4; ++j) bits |= (4 * l16 + j >= lo && 4 * l16 + j <= hi) ? (1u << j) : 0u;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cc = 4 * l16 + j;
      const bool v = pos < n && cc < ncols && (KForQ ? M::mask(pos, col0 + cc, n, margs) : M::mask(col0 + cc, pos, n, margs));
      bits |= v ? (1u << j) : 0u;
    }
  }
  return bits;
}

// ------------------------------------------------------------------------------- forward
template <int DP, int RT>
struct FwdSmem {
  static constexpr int kRows = 8 * RT;
  static constexpr int kQ = 0, kK = kQ + kRows * DP, kV = kK + kCols * DP, kW = kV + kCols * DP;  // in floats
  static constexpr int kBytes = (kW + kRows * kCols) * 4;
};

// kRepair: only the rows that split.cuh has marked.  A form of its own: at head dim 128 the test at the stores alone costs 4 %.
template <int DP, int RT, class M, bool kRepair>
__global__ void __launch_bounds__(kThreads, (DP == 256 ? 1 : (RT == 2 ? 4 : 2))) simt_fwd_kernel(const __grid_constant__ FwdParams pp) {
  using L = FwdSmem<DP, RT>;
  constexpr int kRows = L::kRows;
  extern __shared__ float4 smem4[];
  float* sm = reinterpret_cast<float*>(smem4);
  float *sQ = sm + L::kQ, *sK = sm + L::kK, *sV = sm + L::kV, *sW = sm + L::kW;
  const FwdP& p = pp.f;
  const Geo& g = p.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l16 = lane & 15, row0 = (warp * 2 + (lane >> 4)) * RT;
  const int qb = (int)(gridDim.x - 1 - blockIdx.x) * kRows;  // late (long) causal tiles first
  const int h = blockIdx.y, b = blockIdx.z;
  const int hk = h / (g.H / g.Hkv);
  const int n = valid_len(g, b), D = g.D;
  const int qg0 = qb + g.q_off;
  const int rows_in = imin(kRows, g.Lq - qb);
  uint32_t keep = ~0u;  // rows to store
  if (kRepair) {
    keep = marked<RT>(p.o, b, h, qb + row0, g.Lq);
    if (!__syncthreads_or(keep != 0)) return;
  }
  int kt_lo = 0, kt_hi = 0, full_lo = 0, full_hi = 0;
  if (qg0 < n) {
    int lo, hi;
    tile_range<M, true>(qg0, rows_in, n, g.margs, lo, hi);
    const int lo_l = imax(lo - g.k_off, 0), hi_l = imin(imin(hi, n - 1) - g.k_off, g.Lk - 1);
    if (hi_l >= lo_l) {
      kt_lo = lo_l / kCols;
      kt_hi = hi_l / kCols + 1;
    }
    if (M::kHasKFullRange) M::k_full_range_for_q(qg0, kRows, n, g.margs, full_lo, full_hi);
  }
  load_tile<DP, kRows>(sQ, p.q, b, h, qb, imin(rows_in, n - qg0), D, pp.dtype, pp.vec & kVecQ);
  const float c = g.scale * kLog2e;
  float m[RT], l[RT];
  uint64_t acc[RT][Lane<DP>::kPairs];
  for (bool careful = kRepair;; careful = true) {  // marked rows have met a non-finite number as a rule
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      m[i] = -CUDART_INF_F;
      l[i] = 0.f;
#pragma unroll
      for (int pidx = 0; pidx < Lane<DP>::kPairs; ++pidx) acc[i][pidx] = 0ull;
    }
    for (int kt = kt_lo; kt < kt_hi; ++kt) {
      const int kb = kt * kCols, kg0 = kb + g.k_off;
      const int ncols = imin(n - kg0, g.Lk - kb);
      __syncthreads();  // the previous step has read K and V
      load_tile<DP, kCols>(sK, p.k, b, hk, kb, ncols, D, pp.dtype, pp.vec & kVecK);
      load_tile<DP, kCols>(sV, p.v, b, hk, kb, ncols, D, pp.dtype, pp.vec & kVecV);
      __syncthreads();
      float s[RT][4];
      scores<DP, RT>(sQ, sK, row0, l16, s);
      const bool full = M::kHasKFullRange && kg0 >= full_lo && kg0 + kCols <= full_hi && ncols >= kCols;
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const uint32_t vis = full ? 15u : visible4<M, true>(qg0 + row0 + i, kg0, ncols, l16, n, g.margs);
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = ((vis >> j) & 1u) ? s[i][j] * c : -CUDART_INF_F;
        float mx = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_new = fmaxf(m[i], mx);
        const float m_safe = (m_new == -CUDART_INF_F) ? 0.f : m_new;
        const float alpha = exp2f(m[i] - m_safe);
        m[i] = m_new;
        float4 w;
        w.x = exp2f(s[i][0] - m_safe);
        w.y = exp2f(s[i][1] - m_safe);
        w.z = exp2f(s[i][2] - m_safe);
        w.w = exp2f(s[i][3] - m_safe);
        l[i] = l[i] * alpha + ((w.x + w.y) + (w.z + w.w));  // this lane's columns; summed over the row at the end
        const uint64_t a2 = tc::pk2(alpha, alpha);
#pragma unroll
        for (int pidx = 0; pidx < Lane<DP>::kPairs; ++pidx) acc[i][pidx] = tc::fmul2(acc[i][pidx], a2);
        *reinterpret_cast<float4*>(sW + (row0 + i) * kCols + 4 * (l16 ^ swz(row0 + i))) = w;
      }
      __syncwarp();  // a row of W is written and read by one half-warp
      accumulate<DP, RT>(sW, sV, row0, l16, acc, careful, [](int, int, float wk) { return wk == 0.f; });
      __syncwarp();
    }
    if (careful || !__syncthreads_or(any_nan<DP>(acc))) break;
  }
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    float sum = l[i];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const int row = qb + row0 + i;
    if (row >= g.Lq || (kRepair && !((keep >> i) & 1u))) continue;
    const bool valid = row + g.q_off < n;  // padded query rows: O = 0, LSE = 0
    const float inv = sum != 0.f ? 1.f / sum : 0.f;
    store_row<DP>(p.o.p, b * p.o.sb + h * p.o.sh + row * p.o.sl, p.o.sd, D, pp.dtype, pp.vec & kVecO, l16, acc[i], inv, valid);
    if (p.lse != nullptr && l16 == 0)
      p.lse[b * p.lse_sb + h * p.lse_sh + row * p.lse_sl] = valid ? (sum == 0.f ? -CUDART_INF_F : m[i] + log2f(sum)) : 0.f;
  }
}

// ------------------------------------------------------------------------------ backward
template <int DP, int RT>
struct BwdSmem {
  static constexpr int kRows = 8 * RT;
  static constexpr int kR1 = 0, kR2 = kR1 + kRows * DP, kC1 = kR2 + kRows * DP, kC2 = kC1 + kCols * DP, kW = kC2 + kCols * DP;
  static constexpr int kBytes = (kW + kRows * kCols) * 4;
};

// dK / dV part: rows are keys, R1 = K, R2 = V, the streamed tiles C1 = Q and C2 = dO of every query head of the group:
//     S = K Q^T, dP = V dO^T, P = 2^(S c - LSE), dV += P dO, dS = P (dP - delta), dK += dS Q
// dQ part: rows are queries, R1 = Q, R2 = dO, C1 = K, C2 = V:   S = Q K^T, dP = dO V^T, dQ += dS K
template <int DP, int RT, class M, bool kKeyRows, bool kRepair>
__device__ __forceinline__ void bwd_body(const BwdParams& pp, float* sm, int tile_id) {
  using L = BwdSmem<DP, RT>;
  constexpr int kRows = L::kRows;
  float *sR1 = sm + L::kR1, *sR2 = sm + L::kR2, *sC1 = sm + L::kC1, *sC2 = sm + L::kC2, *sW = sm + L::kW;
  const BwdP& p = pp.b;
  const Geo& g = p.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l16 = lane & 15, row0 = (warp * 2 + (lane >> 4)) * RT;
  const int G = g.H / g.Hkv;
  const int n_units = g.B * (kKeyRows ? g.Hkv : g.H);
  const int n_tiles = ((kKeyRows ? g.Lk : g.Lq) + kRows - 1) / kRows;
  const int rank = tile_id / n_units, unit = tile_id - rank * n_units;
  const int rt = kKeyRows ? rank : n_tiles - 1 - rank;  // longest tiles of a causal mask first
  const int hr = kKeyRows ? unit % g.Hkv : unit % g.H, b = kKeyRows ? unit / g.Hkv : unit / g.H;
  const int rb = rt * kRows, rg0 = rb + (kKeyRows ? g.k_off : g.q_off);
  const int rows_in = imin(kRows, (kKeyRows ? g.Lk : g.Lq) - rb);
  uint32_t keep = ~0u;  // rows to store
  if (kRepair) {
    keep = marked<RT>(kKeyRows ? p.dk : p.dq, b, hr, rb + row0, rb + rows_in);
    if (!__syncthreads_or(keep != 0)) return;
  }
  const int c_off = kKeyRows ? g.q_off : g.k_off, c_len = kKeyRows ? g.Lq : g.Lk;
  const int n = valid_len(g, b), D = g.D;
  int ct_lo = 0, ct_hi = 0, full_lo = 0, full_hi = 0;
  if (rg0 < n) {
    int lo, hi;
    tile_range<M, !kKeyRows>(rg0, rows_in, n, g.margs, lo, hi);
    const int lo_l = imax(lo - c_off, 0), hi_l = imin(imin(hi, n - 1) - c_off, c_len - 1);
    if (hi_l >= lo_l) {
      ct_lo = lo_l / kCols;
      ct_hi = hi_l / kCols + 1;
    }
    if (kKeyRows && M::kHasQFullRange) M::q_full_range_for_k(rg0, kRows, n, g.margs, full_lo, full_hi);
    if (!kKeyRows && M::kHasKFullRange) M::k_full_range_for_q(rg0, kRows, n, g.margs, full_lo, full_hi);
  }
  const TRef& r1 = kKeyRows ? p.k : p.q;
  const TRef& r2 = kKeyRows ? p.v : p.d_o;
  const TRef& c1 = kKeyRows ? p.q : p.k;
  const TRef& c2 = kKeyRows ? p.d_o : p.v;
  const int rows_valid = imin(rows_in, n - rg0);
  load_tile<DP, kRows>(sR1, r1, b, hr, rb, rows_valid, D, pp.dtype, pp.vec & (kKeyRows ? kVecK : kVecQ));
  load_tile<DP, kRows>(sR2, r2, b, hr, rb, rows_valid, D, pp.dtype, pp.vec & (kKeyRows ? kVecV : kVecDo));
  const float c = g.scale * kLog2e;
  float lse_r[RT], delta_r[RT];  // dQ part: of this half-warp's rows
  uint64_t acc1[RT][Lane<DP>::kPairs];                    // dK or dQ
  uint64_t acc2[kKeyRows ? RT : 1][Lane<DP>::kPairs];     // dV
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    lse_r[i] = delta_r[i] = 0.f;
    if (!kKeyRows && rb + row0 + i < g.Lq) {
      const float v = p.lse[b * p.lse_sb + hr * p.lse_sh + (rb + row0 + i) * p.lse_sl];
      lse_r[i] = v == -CUDART_INF_F ? 0.f : v;
      delta_r[i] = p.delta[((long long)b * g.H + hr) * g.Lq + rb + row0 + i];
    }
  }
  for (bool careful = kRepair;; careful = true) {  // marked rows have met a non-finite number as a rule
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int pidx = 0; pidx < Lane<DP>::kPairs; ++pidx) {
        acc1[i][pidx] = 0ull;
        if (kKeyRows) acc2[kKeyRows ? i : 0][pidx] = 0ull;
      }
    for (int gi = 0; gi < (kKeyRows ? G : 1); ++gi) {
      const int hc = kKeyRows ? hr * G + gi : hr / G;
      for (int ct = ct_lo; ct < ct_hi; ++ct) {
        const int cb = ct * kCols, cg0 = cb + c_off;
        const int ncols = imin(n - cg0, c_len - cb);
        __syncthreads();  // the previous step has read the streamed tiles
        load_tile<DP, kCols>(sC1, c1, b, hc, cb, ncols, D, pp.dtype, pp.vec & (kKeyRows ? kVecQ : kVecK));
        load_tile<DP, kCols>(sC2, c2, b, hc, cb, ncols, D, pp.dtype, pp.vec & (kKeyRows ? kVecDo : kVecV));
        float lse_c[4], delta_c[4];  // dK / dV part: of this lane's columns
        if (kKeyRows) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int q = imin(cb + 4 * l16 + j, g.Lq - 1);  // columns beyond Lq are masked out
            const float v = p.lse[b * p.lse_sb + hc * p.lse_sh + q * p.lse_sl];
            lse_c[j] = v == -CUDART_INF_F ? 0.f : v;
            delta_c[j] = p.delta[((long long)b * g.H + hc) * g.Lq + q];
          }
        }
        __syncthreads();
        const bool has_full = kKeyRows ? M::kHasQFullRange : M::kHasKFullRange;
        const bool full = has_full && cg0 >= full_lo && cg0 + kCols <= full_hi && ncols >= kCols && rows_valid == kRows;
        float w[RT][4];
        scores<DP, RT>(sR1, sC1, row0, l16, w);
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          uint32_t vis = 15u;
          if (!full) vis = row0 + i < rows_in ? visible4<M, !kKeyRows>(rg0 + row0 + i, cg0, ncols, l16, n, g.margs) : 0u;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float pe = exp2f(fmaf(w[i][j], c, -(kKeyRows ? lse_c[j] : lse_r[i])));
            w[i][j] = ((vis >> j) & 1u) ? pe : 0.f;
          }
          if (kKeyRows)
            *reinterpret_cast<float4*>(sW + (row0 + i) * kCols + 4 * (l16 ^ swz(row0 + i))) = make_float4(w[i][0], w[i][1], w[i][2], w[i][3]);
        }
        auto hidden = [&](int i, int kx) {
          const int r = rg0 + row0 + i, cc = cg0 + kx;
          return row0 + i >= rows_valid || kx >= ncols || !(kKeyRows ? M::mask(cc, r, n, g.margs) : M::mask(r, cc, n, g.margs));
        };
        if constexpr (kKeyRows) {
          __syncwarp();
          accumulate<DP, RT>(sW, sC2, row0, l16, acc2, careful, [&](int i, int kx, float) { return hidden(i, kx); });
          __syncwarp();
        }
        {
          float dp[RT][4];
          scores<DP, RT>(sR2, sC2, row0, l16, dp);
#pragma unroll
          for (int i = 0; i < RT; ++i) {
#pragma unroll
            for (int j = 0; j < 4; ++j) w[i][j] *= dp[i][j] - (kKeyRows ? delta_c[j] : delta_r[i]);  // hidden pairs: 0 * anything
            *reinterpret_cast<float4*>(sW + (row0 + i) * kCols + 4 * (l16 ^ swz(row0 + i))) = make_float4(w[i][0], w[i][1], w[i][2], w[i][3]);
          }
        }
        __syncwarp();
        accumulate<DP, RT>(sW, sC1, row0, l16, acc1, careful, [&](int i, int kx, float wk) { return wk == 0.f || hidden(i, kx); });
        __syncwarp();
      }
    }
    const bool nan = any_nan<DP>(acc1) || (kKeyRows && any_nan<DP>(acc2));
    if (careful || !__syncthreads_or(nan)) break;
  }
  if constexpr (kKeyRows) {
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int j = rb + row0 + i;
      if (j >= g.Lk || (kRepair && !((keep >> i) & 1u))) continue;
      const bool valid = row0 + i < rows_valid;
      store_row<DP>(p.dk.p, b * p.dk.sb + hr * p.dk.sh + j * p.dk.sl, p.dk.sd, D, pp.dtype, pp.vec & kVecDk, l16, acc1[i], g.scale, valid);
      store_row<DP>(p.dv.p, b * p.dv.sb + hr * p.dv.sh + j * p.dv.sl, p.dv.sd, D, pp.dtype, pp.vec & kVecDv, l16, acc2[i], 1.f, valid);
      float* dkpart = p.part.row(p.part.dk, b, hr, j, g.Lk);
      if (dkpart != nullptr) {
        store_row<DP>(dkpart, 0, 1, D, 0, true, l16, acc1[i], g.scale, valid);
        store_row<DP>(p.part.row(p.part.dv, b, hr, j, g.Lk), 0, 1, D, 0, true, l16, acc2[i], 1.f, valid);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int row = rb + row0 + i;
      if (row < g.Lq && (!kRepair || ((keep >> i) & 1u)))
        store_row<DP>(p.dq.p, b * p.dq.sb + hr * p.dq.sh + row * p.dq.sl, p.dq.sd, D, pp.dtype, pp.vec & kVecDq, l16, acc1[i], g.scale,
                      row0 + i < rows_valid);
    }
  }
}

// One launch for both halves of the backward: dQ does not depend on dK / dV, so its CTAs fill the SMs as the last dK / dV
// CTAs drain.
template <int DP, int RT, class M, bool kRepair>
__global__ void __launch_bounds__(kThreads, (DP == 256 ? 1 : (RT == 2 ? 4 : 2))) simt_bwd_kernel(const __grid_constant__ BwdParams pp) {
  extern __shared__ float4 smem4[];
  float* sm = reinterpret_cast<float*>(smem4);
  if ((int)blockIdx.x < pp.n_key_ctas) bwd_body<DP, RT, M, true, kRepair>(pp, sm, (int)blockIdx.x);
  else bwd_body<DP, RT, M, false, kRepair>(pp, sm, (int)blockIdx.x - pp.n_key_ctas);
}

}  // namespace simt
}  // namespace chill
