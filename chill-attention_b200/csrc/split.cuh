// fp32 attention in IEEE-like accuracy on the tensor cores (sm_100a): head dims 16, 32, 48 and 64, every operand as THREE bf16 parts.
//
// An fp32 number of at least 2^-110 is exactly the sum of three bf16 numbers x = h + m + l (8 + 8 + 8 significand bits), and a
// product of two bf16 numbers is exact in fp32.  Of the nine products of two such sums the kernels form six, hh, hm, mh, hl, mm and
// lh; ml and lm are each at most 2^-25 of |x y| and ll 2^-34, together one rounding of fp32 at most.  So a GEMM costs six bf16 MMAs,
// which is still a multiple of the CUDA cores' fp32 rate.
//
// What would cost accuracy is not the split but the tensor core's accumulator, which truncates: its error is one-sided and
// grows with the number of additions.  It is kept below that of a chain of rounded fp32 FMAs (simt.cuh) by
//   * adding the large products (hh) into columns of their own, or last, after the small ones, so that only the contraction
//     of one tile (64 channels or 64 positions: four MMA steps) is ever truncated at full magnitude, and
//   * starting every tile's product from zero and adding the tiles up in registers, rounded.
// What is left is one-sided all the same: O of V with a common component is low by up to 2.5e-7, and delta with it, which shows where
// dP - delta cancels (V and dO from N(3, 1): dK off by 1.3e-5 at 129 keys, simt.cuh 1.1e-6; at 2048 keys 9e-6 and 3.5e-5).  Large and
// small products of the scores in groups of their own change nothing there.
//
// What the parts cannot hold: NaN, Inf and |x| > 3.39e38 would make 0 * NaN of what the mask hides, and numbers below 2^-110 are no
// sum of three bf16 numbers any more.  The first enter the parts of a streamed tile as zeros; the tile says which of its positions
// have one, or eight channels that are all smaller than 2^-94, and a row that sees such a position is not stored but marked
// (kRepairMark in its first channel); so is a row that has such channels itself or ends with a NaN.  The CUDA-core kernel is launched
// behind these and replaces the marked rows, all others keep their bits.  A non-finite V only concerns its own channel of O: the
// forward adds up to four of them per row and stream to their channels and marks nothing; rows that see more are marked.  Time
// with NaN in every element, (2,8,1000), split and repair / CUDA cores alone, us: q 284 / 377, k and v 331 / 377, backward 1110 / 1200.
//
// Measured against simt.cuh (full mask, head dim 64, us): (2,8,1000) forward 143 -> 44, backward 442 -> 130; (4,8,2048) forward
// 938 -> 274, backward 2975 -> 825.  Distance from the 64-bit result (N(0, 1) inputs, 2-norm): O 5.9e-7 -> 2.0e-7, dQ, dK and dV
// 0.3 to 0.95 of what it was at lengths from 129 to 2048, all masks.  What bounds them is the chain of a step, not a resource: the
// tensor pipe is busy for 35 to 38 % of the time (16 MMAs per score product, 6 up to 32 channels, and 24 with N = 64 per accumulating
// one), shared memory for 30 %, the L2 for 10 % (profiles/split_fp32_kernels_ncu.md).  In the forward the loaders' part of it, loads,
// split and stores of one tile after the other, is as long as what the streams do.  MMA loops are rolled where their operands only
// differ by an addition.
#pragma once
#include <type_traits>

#include "generic.cuh"
#include "tc_common.cuh"

namespace chill {

constexpr uint32_t kRepairMark = 0x7fc0deadu;  // a NaN no arithmetic produces

namespace split {

using tc::Guard;
using tc::mbar_wait;
typedef __nv_bfloat16 BF;

constexpr int kRows = 128;                      // rows of a CTA's tile
constexpr int kCols = 64;                       // streamed positions per step
constexpr int kRowPart = kRows * 128;           // one bf16 part of a row operand: 128 rows of one 128-byte line
constexpr int kColPart = kCols * 128;           // one part of a streamed tile
constexpr int kLoaders = 128;                   // threads that load and split
// Eight neighbouring channels of a position go into the parts as they are if the largest is 0 or in [kLeast, kMost): kMost is what
// bf16 can hold; elements below 2^-110 lose the bits of their third part that lie under bf16's smallest subnormal, 2^-133, which is
// less than 2^-39 of a neighbour of kLeast.
constexpr float kLeast = 0x1p-94f, kMost = 3.39e38f;
constexpr float kUp = 65536.f, kDown = 1.f / kUp;  // dS is split times 2^16: it may be tiny although V and dO are not

enum : int { kStSplitLoad = 701, kStSplitMma = 702, kStSplitCompute = 703 };

struct FwdParams {
  FwdP f;
  int* status;
};
struct BwdParams {
  BwdP b;
  int n_key_ctas;  // the first n_key_ctas CTAs compute dK / dV, the others dQ
  int* status;
};

// Parts of two numbers, packed.
__device__ __forceinline__ void split2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  float x, y;
  h = tc::pack2<BF>(a, b);
  tc::unpack2<BF>(h, x, y);
  a -= x;
  b -= y;
  m = tc::pack2<BF>(a, b);
  tc::unpack2<BF>(m, x, y);
  l = tc::pack2<BF>(a - x, b - y);
}

__device__ __forceinline__ float max3_nan(float a, float b, float c) {  // of the magnitudes; NaN if one is
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(fabsf(a)), "f"(fabsf(b)), "f"(fabsf(c)));
  return d;
}
__device__ __forceinline__ bool unfit(float x) { return !(fabsf(x) < kMost); }

// ROWS x 64 fp32 elements of one (batch, head), eight channels of a row per thread and unit: from global memory into
// registers, and from there as three parts into 128B-swizzled shared memory.  Rows beyond rows_in and channels beyond D are
// zero and not read.
template <int ROWS>
struct TileRegs {
  static constexpr int kUnits = ROWS * 8 / kLoaders;
  float4 v[kUnits][2];
  __device__ __forceinline__ void fetch(const TRef& t, int b, int h, int row0, int rows_in, int D, int tid) {
    const float* p = static_cast<const float*>(t.p) + b * t.sb + h * t.sh + row0 * t.sl;
#pragma unroll
    for (int i = 0; i < kUnits; ++i) {
      const int idx = i * kLoaders + tid, row = idx >> 3, u = idx & 7;
      v[i][0] = v[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < rows_in && u * 8 < D) {
        const float4* s = reinterpret_cast<const float4*>(p + row * t.sl + u * 8);
        v[i][0] = s[0];
        v[i][1] = s[1];
      }
    }
  }
  // magnitude of the largest element of unit i, NaN if one is
  __device__ __forceinline__ float largest(int i) const {
    const float4 &a = v[i][0], &b = v[i][1];
    return max3_nan(max3_nan(a.x, a.y, a.z), max3_nan(a.w, b.x, b.y), max3_nan(b.z, b.w, 0.f));
  }
  __device__ __forceinline__ void put(uint8_t* dst, int part_bytes, int tid) const {
#pragma unroll
    for (int i = 0; i < kUnits; ++i) {
      const int idx = i * kLoaders + tid, row = idx >> 3, u = idx & 7;
      uint32_t h[4], m[4], l[4];
      split2(v[i][0].x, v[i][0].y, h[0], m[0], l[0]);
      split2(v[i][0].z, v[i][0].w, h[1], m[1], l[1]);
      split2(v[i][1].x, v[i][1].y, h[2], m[2], l[2]);
      split2(v[i][1].z, v[i][1].w, h[3], m[3], l[3]);
      uint8_t* d = dst + row * 128 + ((u ^ (row & 7)) << 4);
      *reinterpret_cast<uint4*>(d) = make_uint4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint4*>(d + part_bytes) = make_uint4(m[0], m[1], m[2], m[3]);
      *reinterpret_cast<uint4*>(d + 2 * part_bytes) = make_uint4(l[0], l[1], l[2], l[3]);
    }
  }
};
// A streamed tile: elements that bf16 cannot hold are replaced by zeros.  Returns, to every lane, which of this warp's rows have
// channels that are no part of a sum of parts (NaN, Inf, too large, too small): bit 4 i + e stands for row 16 i + 4 (warp) + e.
__device__ __forceinline__ uint32_t clean(TileRegs<kCols>& t) {
  constexpr int N = TileRegs<kCols>::kUnits;
  bool bad[N], any = false;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float mx = t.largest(i);
    bad[i] = unfit(mx) || (mx < kLeast && mx > 0.f);
    any = any || bad[i];
  }
  uint32_t rows = 0;
  if (__any_sync(0xffffffffu, any)) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      float4 &a = t.v[i][0], &b = t.v[i][1];
      const uint32_t who = __ballot_sync(0xffffffffu, bad[i]);
      float* f[8] = {&a.x, &a.y, &a.z, &a.w, &b.x, &b.y, &b.z, &b.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) *f[e] = unfit(*f[e]) ? 0.f : *f[e];
#pragma unroll
      for (int e = 0; e < 4; ++e) rows |= ((who >> (8 * e)) & 0xffu) != 0 ? 1u << (4 * i + e) : 0u;
    }
  }
  return rows;
}
// Rows of half a resident tile with channels that are too small, like clean(); NaN, Inf and too large ones make the row's results
// NaN by themselves.
__device__ __forceinline__ uint32_t small_rows(const TileRegs<64>& t) {
  uint32_t rows = 0;
#pragma unroll
  for (int i = 0; i < TileRegs<64>::kUnits; ++i) {
    const float mx = t.largest(i);
    const uint32_t who = __ballot_sync(0xffffffffu, mx < kLeast && mx > 0.f);
#pragma unroll
    for (int e = 0; e < 4; ++e) rows |= ((who >> (8 * e)) & 0xffu) != 0 ? 1u << (4 * i + e) : 0u;
  }
  return rows;
}
// Whether row r of the resident tile is one of them; words: [half][loader warp].
__device__ __forceinline__ bool is_small(const uint32_t* words, int r) {
  return ((words[(r >> 6) * 4 + ((r >> 2) & 3)] >> (4 * ((r >> 4) & 3) + (r & 3))) & 1u) != 0;
}
// Positions that clean() has found in the two streamed tiles of a step; words: of the four loader warps, for the first tile and for
// the second.  f(position, in the first, in the second) for each.
template <class F>
__device__ __forceinline__ void for_unfit(const uint4* words, const F& f) {
  const uint4 a = words[0], b = words[1];
  if ((a.x | a.y | a.z | a.w | b.x | b.y | b.z | b.w) == 0) return;
#pragma unroll 1
  for (int pos = 0; pos < kCols; ++pos) {
    const int w = (pos >> 2) & 3, bit = 4 * (pos >> 4) + (pos & 3);
    const bool in_a = (reinterpret_cast<const uint32_t*>(words)[w] >> bit) & 1u, in_b = (reinterpret_cast<const uint32_t*>(words)[4 + w] >> bit) & 1u;
    if (in_a || in_b) f(pos, in_a, in_b);
  }
}
// The tile is visible to the tensor cores; one arrival per loader warp.
__device__ __forceinline__ void publish(uint32_t bar, int lane) {
  tc::fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) tc::mbar_arrive(bar);
}
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, const Guard& g, int code) {
  const bool ok = mbar_wait(bar, parity, g, code);
  return __all_sync(0xffffffffu, ok);  // the warp stays converged
}

// Scores [128 rows][64 positions], contraction over 64 channels, in three groups of 64 columns whose sum they are: the large
// products of channels 0-31 | those of channels 32-63 after hm + mh of 0-31 | all the others.  Splitting the large products
// halves what truncation takes from them, which counts where dP - delta cancels (inputs of one sign: dK 5.1e-7 from the exact
// values in one group, 2.5e-7 in two, 2.9e-7 in simt.cuh).
// The parts of the streamed tile lie one after the other, so one MMA with N = 192 / 128 takes several of them at once.
__device__ __forceinline__ void mma_scores(uint32_t t, uint32_t rows_smem, uint32_t cols_smem, int D) {
  constexpr uint32_t hi = tc::desc_hi_sw128(1024);
  constexpr uint32_t id3 = tc::make_idesc<BF>(kRows, 3 * kCols, false, false), id2 = tc::make_idesc<BF>(kRows, 2 * kCols, false, false),
                     id1 = tc::make_idesc<BF>(kRows, kCols, false, false);
  constexpr uint32_t rp = kRowPart / 16, cp = kColPart / 16;
  const uint32_t a = tc::desc_lo_sw128(rows_smem, 16), b = tc::desc_lo_sw128(cols_smem, 16);
#pragma unroll 1
  for (uint32_t k = 0; k < 4; k += 2) {  // 16 channels = 2 units per MMA
    tc::mma_ss_lh(t, a + k, b + k, hi, id3, k > 0 ? 1u : 0u);
    tc::mma_ss_lh(t + kCols, a + rp + k, b + k, hi, id2, 1u);
    tc::mma_ss_lh(t + 2 * kCols, a + 2 * rp + k, b + k, hi, id1, 1u);
  }
  if (D <= 32) return;
#pragma unroll 1
  for (uint32_t k = 4; k < 8; k += 2) {
    tc::mma_ss_lh(t + 2 * kCols, a + k, b + 2 * cp + k, hi, id1, 1u);
    tc::mma_ss_lh(t + 2 * kCols, a + rp + k, b + cp + k, hi, id1, 1u);
    tc::mma_ss_lh(t + 2 * kCols, a + 2 * rp + k, b + k, hi, id1, 1u);
    tc::mma_ss_lh(t + 2 * kCols, a + rp + k, b + k, hi, id1, 1u);
    tc::mma_ss_lh(t + kCols, a + k, b + k, hi, id2, 1u);
  }
}
// dst[128][64 channels] = W X over the 64 streamed positions: W's parts from TMEM, X's parts from shared memory, MN-major; small
// products first.  Columns of W: part q starts at kW(q), its 16 positions kk at kPos(kk).
struct WFwd {  // one thread holds all 64 positions of a row
  static __device__ __forceinline__ uint32_t part(uint32_t q) { return 32 * q; }
  static __device__ __forceinline__ constexpr uint32_t pos(int kk) { return 8 * kk; }
};
struct WBwd {  // two warpgroups hold 32 positions each and write over columns that only they read
  static __device__ __forceinline__ uint32_t part(uint32_t q) { return q == 2 ? 64 : 16 * q; }
  static __device__ __forceinline__ constexpr uint32_t pos(int kk) { return 32 * (kk / 2) + 8 * (kk % 2); }
};
template <class W>
__device__ __forceinline__ void mma_accumulate(uint32_t dst, uint32_t w, uint32_t x_smem) {
  constexpr uint32_t hi = tc::desc_hi_sw128(1024), id = tc::make_idesc<BF>(kRows, 64, false, true);
  const uint32_t x = tc::desc_lo_sw128(x_smem, kColPart);
#pragma unroll 1
  for (int o = 0; o < 6; ++o) {
    const uint32_t wp = (0x001012u >> (4 * o)) & 15u, xp = (0x010210u >> (4 * o)) & 15u;  // part of W, part of X
    const uint32_t wa = w + W::part(wp), xa = x + xp * (kColPart / 16);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) tc::mma_ts_lh(dst, wa + W::pos(kk), xa + kk * 128, hi, id, (kk > 0 || o > 0) ? 1u : 0u);
  }
}
// Sums of the three column groups for 16 positions.
__device__ __forceinline__ void load_scores16(uint32_t t, float* s) {
  uint32_t a[16], b[16], c[16];
  tc::tmem_ld16(t, a);
  tc::tmem_ld16(t + kCols, b);
  tc::tmem_ld16(t + 2 * kCols, c);
  tc::tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < 16; ++i) s[i] = __uint_as_float(a[i]) + (__uint_as_float(b[i]) + __uint_as_float(c[i]));
}

// 32 lanes x 8 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

__device__ __forceinline__ void store_row_f32(float* dst, const float* v, int n) {
#pragma unroll
  for (int i = 0; i < n; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}

// ------------------------------------------------------------------------------- forward
// One CTA per SM owns 128 query rows.  Two softmax warpgroups take the key tiles in turn (even / odd), each with scores, product,
// maximum and sums of its own, and the two results are merged at the end: the chain of a tile (scores, softmax, product) is
// serial, so the issuing thread works for one of them while the other is in its softmax.
constexpr int kFwdThreads = 512;  // warps 0-3 / 4-7 softmax of stream 0 / 1 (thread = query row), 8-11 loaders, 12 / 13 MMA issuers of
// stream 0 / 1 (12 owns TMEM)
constexpr int kFwdSoftmaxRegs = 160, kFwdLoadRegs = 112, kFwdOtherRegs = 80;  // 256 * 160 + 128 * 112 + 128 * 80 = 512 * 128

struct FwdSmem {
  static constexpr int kQ = 0;
  static constexpr int kKv = kQ + 3 * kRowPart;  // per stream: parts of K, parts of V; at the end stream 1's O, maximum and sum
  static constexpr int kStream = 6 * kColPart;
  static constexpr int kUnfit = kKv + 2 * kStream;  // per stream, for every other of its tiles: words of K, words of V (four each)
  static constexpr int kBars = kUnfit + 4 * 32;
  static constexpr int kMisc = kBars + 8 * 12;
  static constexpr int kSeenV = 4;               // positions a row remembers (softmax threads: 256)
  static constexpr int kRowSmall = kMisc + 16;   // see is_small
  static constexpr int kSeen = kRowSmall + 32;
  static constexpr int kDynamic = kSeen + kSeenV * 256 * 4 + 1024;
  static_assert(kRows * (64 + 4) * 4 <= kStream, "the merge uses the stream's tiles");
};

template <class M>
__global__ void __launch_bounds__(kFwdThreads, 1) split_fwd_kernel(const __grid_constant__ FwdParams pp) {
  using L = FwdSmem;
  const FwdP& p = pp.f;
  const Geo& g = p.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qb = (int)(gridDim.x - 1 - blockIdx.x) * kRows;  // late (long) causal tiles first
  const int h = blockIdx.y, b = blockIdx.z;
  const int hk = h / (g.H / g.Hkv);
  const int n = valid_len(g, b), D = g.D;
  const int qg0 = qb + g.q_off;
  const int rows_in = imin(kRows, g.Lq - qb);
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
  const int n_tiles = kt_hi - kt_lo;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (tc::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - tc::smem_u32(smem_raw));
  const uint32_t bars = base + L::kBars;
  // per stream w: + 8 w
  const uint32_t bar_k = bars, bar_v = bars + 16, bar_s = bars + 32, bar_p = bars + 48, bar_o = bars + 64, bar_q = bars + 80, bar_merge = bars + 88;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + L::kMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + L::kMisc + 4);
  uint32_t* row_small = reinterpret_cast<uint32_t*>(gen + L::kRowSmall);
  const Guard guard{pp.status, abort_flag};
  if (warp == 12) {
    if (lane == 0) {
      *abort_flag = 0;
      for (int w = 0; w < 2; ++w) {
        tc::mbar_init(bar_k + 8 * w, 4);
        tc::mbar_init(bar_v + 8 * w, 4);
        tc::mbar_init(bar_s + 8 * w, 1);
        tc::mbar_init(bar_p + 8 * w, 4);
        tc::mbar_init(bar_o + 8 * w, 1);
      }
      tc::mbar_init(bar_q, 4);
      tc::mbar_init(bar_merge, 4);
      tc::fence_barrier_init();
    }
    __syncwarp();
    tc::tmem_alloc(tc::smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;  // per stream: scores 192 columns (the parts of P over the first 96), product of the tile 64

  if (warp >= 12) {
    tc::reg_dealloc<kFwdOtherRegs>();
    if (warp < 14 && lane == 0 && n_tiles > warp - 12) {
      // ------------------------------------------------- MMA issuer of stream 0 (warp 12) or 1 (warp 13)
      const uint32_t w = (uint32_t)(warp - 12), t = tmem + 256 * w, kv = base + L::kKv + L::kStream * w;
      bool ok = mbar_wait(bar_q, 0, guard, kStSplitMma);
      for (int j = (int)w; j < n_tiles && ok; j += 2) {
        const uint32_t par = (uint32_t)(j >> 1) & 1u;
        if (!(ok = mbar_wait(bar_k + 8 * w, par, guard, kStSplitMma))) break;
        tc::tc_fence_after();
        mma_scores(t, base + L::kQ, kv, D);  // over the previous P, which the MMAs before these have read
        tc::mma_commit(bar_s + 8 * w);
        if (!(ok = mbar_wait(bar_v + 8 * w, par, guard, kStSplitMma))) break;
        if (!(ok = mbar_wait(bar_p + 8 * w, par, guard, kStSplitMma))) break;
        tc::tc_fence_after();
        mma_accumulate<WFwd>(t + 3 * kCols, t, kv + 3 * kColPart);
        tc::mma_commit(bar_o + 8 * w);
      }
    }
  } else if (warp >= 8) {
    tc::reg_dealloc<kFwdLoadRegs>();
    // ------------------------------------------------------------------------ loaders
    const int tid = threadIdx.x - 256;
    if (n_tiles > 0) {
      const int q_rows = imin(rows_in, n - qg0);
      TileRegs<64> r;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        r.fetch(p.q, b, h, qb + 64 * half, q_rows - 64 * half, D, tid);
        const uint32_t small = small_rows(r);
        if (lane == 0) row_small[4 * half + warp - 8] = small;
        r.put(gen + L::kQ + 64 * half * 128, kRowPart, tid);
      }
      publish(bar_q, lane);
    }
    for (int j = 0; j < n_tiles; ++j) {
      const uint32_t w = (uint32_t)j & 1u, prev = ((uint32_t)(j >> 1) & 1u) ^ 1u;
      const int kb = (kt_lo + j) * kCols, rows = imin(n - (kb + g.k_off), g.Lk - kb);
      uint8_t* kv = gen + L::kKv + L::kStream * w;
      TileRegs<kCols> rk, rv;
      rk.fetch(p.k, b, hk, kb, rows, D, tid);
      rv.fetch(p.v, b, hk, kb, rows, D, tid);
      // The words of tile j - 4 have been read when P of tile j - 2 has been sent.
      uint32_t* words = reinterpret_cast<uint32_t*>(gen + L::kUnfit + 64 * w + 32 * ((j >> 1) & 1)) + (warp - 8);
      const uint32_t bad_k = clean(rk);
      if (j >= 2 && !warp_wait(bar_s + 8 * w, prev, guard, kStSplitLoad)) break;  // the scores of tile j - 2 have read K
      rk.put(kv, kColPart, tid);
      publish(bar_k + 8 * w, lane);
      const uint32_t bad_v = clean(rv);
      if (j >= 2 && !warp_wait(bar_o + 8 * w, prev, guard, kStSplitLoad)) break;  // P V of tile j - 2 has read V
      if (lane == 0) {
        words[0] = bad_k;
        words[4] = bad_v;
      }
      rv.put(kv + 3 * kColPart, kColPart, tid);
      publish(bar_v + 8 * w, lane);
    }
  } else {
    tc::reg_alloc<kFwdSoftmaxRegs>();
    // --------------------------------------------------------- softmax + output rows
    const int w = warp >> 2;                  // stream
    const int r = (warp & 3) * 32 + lane;     // row inside the tile == TMEM lane
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + 256 * w + lane_sel, tO = tS + 3 * kCols;
    const int qg = qg0 + r;
    const float c = g.scale * kLog2e;
    float m = -CUDART_INF_F, l = 0.f;
    float o[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) o[i] = 0.f;
    bool ok = true, repair = false;
    int n_v = 0;                               // unfit positions of V that this row sees; the first few of them:
    int* seen_v = reinterpret_cast<int*>(gen + L::kSeen) + threadIdx.x;
    for (int j = w; j < n_tiles; j += 2) {
      const uint32_t par = (uint32_t)(j >> 1) & 1u;
      const int kb = (kt_lo + j) * kCols, kg0 = kb + g.k_off;
      const int ncols = imin(n - kg0, g.Lk - kb);
      if (!(ok = warp_wait(bar_s + 8 * w, par, guard, kStSplitCompute))) break;
      tc::tc_fence_after();
      float s[kCols];
#pragma unroll
      for (int q = 0; q < 4; ++q) load_scores16(tS + q * 16, s + q * 16);
      const bool full = M::kHasKFullRange && kg0 >= full_lo && kg0 + kCols <= full_hi && ncols >= kCols;
      if (!full) {
        if (interval_rows<M>::value) {
          int lo, hi;
          row_window<M, true>(qg, kg0, ncols, n, g.margs, lo, hi);
#pragma unroll
          for (int i = 0; i < kCols; ++i) s[i] = (i >= lo && i <= hi) ? s[i] * c : -CUDART_INF_F;
        } else {
#pragma unroll
          for (int i = 0; i < kCols; ++i) s[i] = (qg < n && i < ncols && M::mask(qg, kg0 + i, n, g.margs)) ? s[i] * c : -CUDART_INF_F;
        }
      } else {
#pragma unroll
        for (int i = 0; i < kCols; ++i) s[i] *= c;
      }
      float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int i = 4; i < kCols; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
      const float m_new = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
      const float m_safe = (m_new == -CUDART_INF_F) ? 0.f : m_new;
      const float alpha = tc::ex2(m - m_safe);
      m = m_new;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // 16 positions: 8 columns of each part
        uint32_t ph[8], pm[8], pl[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float a = tc::ex2(s[q * 16 + 2 * i] - m_safe), bb = tc::ex2(s[q * 16 + 2 * i + 1] - m_safe);
          sum[i & 3] += a + bb;
          split2(a, bb, ph[i], pm[i], pl[i]);
        }
        tmem_st8(tS + q * 8, ph);
        tmem_st8(tS + 32 + q * 8, pm);
        tmem_st8(tS + 64 + q * 8, pl);
      }
      l = l * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar_p + 8 * w);
      if (!(ok = warp_wait(bar_o + 8 * w, par, guard, kStSplitCompute))) break;
      tc::tc_fence_after();
      for_unfit(reinterpret_cast<const uint4*>(gen + L::kUnfit + 64 * w + 32 * par), [&](int pos, bool in_k, bool in_v) {
        if (qg >= n || pos >= ncols || !M::mask(qg, kg0 + pos, n, g.margs)) return;
        repair = repair || in_k;
        if (in_v && n_v < L::kSeenV) seen_v[n_v * 256] = kb + pos;
        n_v += in_v ? 1 : 0;
      });
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t t[32];
        tc::tmem_ld32(tO + q * 32, t);
        tc::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) o[q * 32 + i] = fmaf(o[q * 32 + i], alpha, __uint_as_float(t[i]));
      }
      tc::tc_fence_before();
    }
    // ---- merge: stream 1 hands its rows over in its own K / V tiles, which nothing reads any more
    float4* mo = reinterpret_cast<float4*>(gen + L::kKv + L::kStream) + r;
    float4* ml = reinterpret_cast<float4*>(gen + L::kKv + L::kStream + kRows * 64 * 4) + r;
    if (n_tiles > 1 && w == 1 && ok) {
#pragma unroll
      for (int i = 0; i < 16; ++i) mo[i * kRows] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
      *ml = make_float4(m, l, repair ? 1.f : 0.f, (float)n_v);
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar_merge);
    }
    int n_v1 = 0;  // like n_v, of stream 1
    if (n_tiles > 1 && w == 0 && ok) {
      ok = warp_wait(bar_merge, 0, guard, kStSplitCompute);
      if (ok) {
        const float4 v = *ml;
        repair = repair || v.z != 0.f;
        n_v1 = (int)v.w;
        const float m_all = fmaxf(m, v.x), m_safe = (m_all == -CUDART_INF_F) ? 0.f : m_all;
        const float a0 = tc::ex2(m - m_safe), a1 = tc::ex2(v.x - m_safe);
        m = m_all;
        l = l * a0 + v.y * a1;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float4 x = mo[i * kRows];
          o[4 * i] = o[4 * i] * a0 + x.x * a1;
          o[4 * i + 1] = o[4 * i + 1] * a0 + x.y * a1;
          o[4 * i + 2] = o[4 * i + 2] * a0 + x.z * a1;
          o[4 * i + 3] = o[4 * i + 3] * a0 + x.w * a1;
        }
      }
    }
    const int row = qb + r;
    if (w == 0 && ok && row < g.Lq) {
      const bool valid = qg < n;  // padded query rows: O = 0, LSE = 0
      // Elements of V that went into the product as zeros: NaN and Inf are added to their channels, the others keep their bits.  A row
      // that sees many such positions is left to the CUDA cores.
      if (n_v > L::kSeenV || n_v1 > L::kSeenV || (n_tiles > 0 && is_small(row_small, r))) repair = true;
#pragma unroll 1
      for (int e = 0; e < n_v + n_v1 && !repair; ++e) {
        const int pos = e < n_v ? seen_v[e * 256] : seen_v[(e - n_v) * 256 + 128];
        const float* q = static_cast<const float*>(p.q.p) + b * p.q.sb + h * p.q.sh + (long long)row * p.q.sl;
        const float* k = static_cast<const float*>(p.k.p) + b * p.k.sb + hk * p.k.sh + (long long)pos * p.k.sl;
        const float* v = static_cast<const float*>(p.v.p) + b * p.v.sb + hk * p.v.sh + (long long)pos * p.v.sl;
        float sc = 0.f;
#pragma unroll 1
        for (int i = 0; i < D; ++i) sc = fmaf(q[i], k[i], sc);
        const float weight = tc::ex2(sc * (g.scale * kLog2e) - m);
        if (weight == 0.f) continue;  // as if hidden, like simt.cuh
#pragma unroll
        for (int i = 0; i < 64; i += 8) {
          float mx = 0.f;  // of the finite ones
#pragma unroll
          for (int ii = i; ii < i + 8; ++ii) {
            const float x = ii < D ? v[ii] : 0.f;
            if (x - x != 0.f) o[ii] += weight * x;
            else mx = fmaxf(mx, fabsf(x));
          }
          if (mx >= kMost || (mx < kLeast && mx > 0.f)) repair = true;
        }
      }
      const float inv = (valid && l != 0.f) ? 1.f / l : 0.f;
#pragma unroll
      for (int i = 0; i < 64; ++i) o[i] = valid ? o[i] * inv : 0.f;
      if (valid && (repair || l != l)) o[0] = __uint_as_float(kRepairMark);
      float* orow = static_cast<float*>(p.o.p) + b * p.o.sb + h * p.o.sh + row * p.o.sl;
      store_row_f32(orow, o, 16);
      if (D > 16) store_row_f32(orow + 16, o + 16, 16);
      if (D > 32) store_row_f32(orow + 32, o + 32, 16);
      if (D > 48) store_row_f32(orow + 48, o + 48, 16);
      if (p.lse != nullptr)
        p.lse[b * p.lse_sb + h * p.lse_sh + row * p.lse_sl] = valid ? (l == 0.f ? -CUDART_INF_F : m + log2f(l)) : 0.f;
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 12) tc::tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------------------ backward
// dK / dV part: rows are keys, R1 = K, R2 = V, the streamed tiles C1 = Q and C2 = dO of every query head of the group:
//     S = K Q^T, dP = V dO^T, P = 2^(S c - LSE), dV += P dO, dS = P (dP - delta), dK += dS Q
// dQ part: rows are queries, R1 = Q, R2 = dO, C1 = K, C2 = V:   S = Q K^T, dP = dO V^T, dQ += dS K
//
// TMEM (512 columns): S 192 (P's parts over it) | dP 192 (dS's parts over it) | product with C1 64 | product with C2 64.
// Two issuing threads, one for S(u), dV(u), S(u+1) ..., the other for dP(u), dK(u), dP(u+1) ...: the scores of the next step run
// during the elementwise work of this one.
constexpr int kBwdThreads = 512;  // warps 0-7 compute (thread = row; warps 0-3 / 4-7 split the 64 positions and the 64 channels), 8-11 loaders, 12 / 13 MMA issuers
constexpr int kBwdComputeRegs = 160, kBwdLoadRegs = 112, kBwdOtherRegs = 80;  // 256 * 160 + 128 * 112 + 128 * 80 = 512 * 128

struct BwdSmem {
  static constexpr int kR1 = 0, kR2 = kR1 + 3 * kRowPart;
  static constexpr int kC = kR2 + 3 * kRowPart;      // two stages of the parts of C1, parts of C2
  static constexpr int kStage = 6 * kColPart;
  static constexpr int kVec = kC + 2 * kStage;       // per compute warp: -LSE and -delta of its 32 streamed positions
  static constexpr int kBad = kVec + 8 * 2 * 32 * 4;  // per row: the second warpgroup's half holds a NaN
  static constexpr int kUnfit = kBad + kRows * 4;  // per stage: words of C1, words of C2 (four each)
  static constexpr int kBars = kUnfit + 2 * 32;
  static constexpr int kMisc = kBars + 8 * 14;
  static constexpr int kRowSmall = kMisc + 16;       // see is_small
  static constexpr int kDynamic = kRowSmall + 32 + 1024;
};

template <class M, bool kKeyRows>
__device__ __forceinline__ void bwd_body(const BwdParams& pp, uint8_t* smem_raw, int tile_id) {
  using L = BwdSmem;
  const BwdP& p = pp.b;
  const Geo& g = p.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = g.H / g.Hkv;
  const int n_units = g.B * (kKeyRows ? g.Hkv : g.H);
  const int n_rt = ((kKeyRows ? g.Lk : g.Lq) + kRows - 1) / kRows;
  const int rank = tile_id / n_units, unit = tile_id - rank * n_units;
  const int rt = kKeyRows ? rank : n_rt - 1 - rank;  // longest tiles of a causal mask first
  const int hr = kKeyRows ? unit % g.Hkv : unit % g.H, b = kKeyRows ? unit / g.Hkv : unit / g.H;
  const int rb = rt * kRows, rg0 = rb + (kKeyRows ? g.k_off : g.q_off);
  const int rows_in = imin(kRows, (kKeyRows ? g.Lk : g.Lq) - rb);
  const int c_off = kKeyRows ? g.q_off : g.k_off, c_len = kKeyRows ? g.Lq : g.Lk;
  const int n = valid_len(g, b), D = g.D;
  const int rows_valid = imin(rows_in, n - rg0);
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
  const int n_ct = ct_hi - ct_lo;
  const int n_it = n_ct * (kKeyRows ? G : 1);

  const uint32_t base = (tc::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - tc::smem_u32(smem_raw));
  const uint32_t bars = base + L::kBars;
  // per stage: + 8 s
  const uint32_t bar_r = bars, bar_s = bars + 8, bar_dp = bars + 16, bar_p = bars + 24, bar_ds = bars + 32, bar_bad = bars + 40, bar_c1 = bars + 48,
                 bar_c2 = bars + 64, bar_acc = bars + 80;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + L::kMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + L::kMisc + 4);
  uint32_t* row_small = reinterpret_cast<uint32_t*>(gen + L::kRowSmall);
  const Guard guard{pp.status, abort_flag};
  if (warp == 12) {
    if (lane == 0) {
      *abort_flag = 0;
      tc::mbar_init(bar_r, 4);
      tc::mbar_init(bar_s, 1);
      tc::mbar_init(bar_dp, 1);
      tc::mbar_init(bar_p, 8);
      tc::mbar_init(bar_ds, 8);
      tc::mbar_init(bar_bad, 4);
      for (int s = 0; s < 2; ++s) {
        tc::mbar_init(bar_c1 + 8 * s, 4);
        tc::mbar_init(bar_c2 + 8 * s, 4);
        tc::mbar_init(bar_acc + 8 * s, kKeyRows ? 2 : 1);
      }
      tc::fence_barrier_init();
    }
    __syncwarp();
    tc::tmem_alloc(tc::smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot, tS = tmem, tdP = tmem + 3 * kCols, tAcc1 = tmem + 6 * kCols, tAcc2 = tAcc1 + 64;

  if (warp >= 12) {
    tc::reg_dealloc<kBwdOtherRegs>();
    if (warp < 14 && lane == 0 && n_it > 0) {
      // ------------- MMA issuers: warp 12 for S and the product with P, warp 13 for dP and the product with dS
      const bool first = warp == 12;
      const uint32_t t = first ? tS : tdP, r = base + (first ? L::kR1 : L::kR2), c_bar = first ? bar_c1 : bar_c2, s_bar = first ? bar_s : bar_dp,
                     w_bar = first ? bar_p : bar_ds;
      bool ok = mbar_wait(bar_r, 0, guard, kStSplitMma);
      for (int it = 0; it < n_it && ok; ++it) {
        const uint32_t st = (uint32_t)(it & 1), stage = base + L::kC + st * L::kStage;
        if (!(ok = mbar_wait(c_bar + 8 * st, (uint32_t)(it >> 1) & 1u, guard, kStSplitMma))) break;
        tc::tc_fence_after();
        mma_scores(t, r, stage + (first ? 0 : 3 * kColPart), D);  // over the parts that this thread's previous MMAs have read
        tc::mma_commit(s_bar);
        if (!(ok = mbar_wait(w_bar, (uint32_t)it & 1u, guard, kStSplitMma))) break;  // the parts are in place (S of the dQ part: read)
        if (first && !kKeyRows) continue;
        tc::tc_fence_after();
        mma_accumulate<WBwd>(first ? tAcc2 : tAcc1, t, stage + (first ? 3 * kColPart : 0));
        tc::mma_commit(bar_acc + 8 * st);  // with the other thread's: the products are there, the stage may be refilled
      }
    }
  } else if (warp >= 8) {
    tc::reg_dealloc<kBwdLoadRegs>();
    // ------------------------------------------------------------------------ loaders
    const int tid = threadIdx.x - 256;
    const TRef& r1 = kKeyRows ? p.k : p.q;
    const TRef& r2 = kKeyRows ? p.v : p.d_o;
    const TRef& c1 = kKeyRows ? p.q : p.k;
    const TRef& c2 = kKeyRows ? p.d_o : p.v;
    if (n_it > 0) {
      TileRegs<64> r;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        r.fetch(r1, b, hr, rb + 64 * half, rows_valid - 64 * half, D, tid);
        uint32_t small = small_rows(r);
        r.put(gen + L::kR1 + 64 * half * 128, kRowPart, tid);
        r.fetch(r2, b, hr, rb + 64 * half, rows_valid - 64 * half, D, tid);
        small |= small_rows(r);
        if (lane == 0) row_small[4 * half + warp - 8] = small;
        r.put(gen + L::kR2 + 64 * half * 128, kRowPart, tid);
      }
      publish(bar_r, lane);
    }
    int hc = kKeyRows ? hr * G : hr / G, ct = ct_lo;
    for (int it = 0; it < n_it; ++it) {
      const uint32_t s = (uint32_t)it & 1u, prev = ((uint32_t)(it >> 1) & 1u) ^ 1u;
      const int cb = ct * kCols, rows = imin(n - (cb + c_off), c_len - cb);
      uint8_t* st = gen + L::kC + s * L::kStage;
      TileRegs<kCols> a, d;
      a.fetch(c1, b, hc, cb, rows, D, tid);
      d.fetch(c2, b, hc, cb, rows, D, tid);
      uint32_t* words = reinterpret_cast<uint32_t*>(gen + L::kUnfit + 32 * s) + (warp - 8);
      const uint32_t bad1 = clean(a);
      if (it >= 2 && !warp_wait(bar_acc + 8 * s, prev, guard, kStSplitLoad)) break;  // step it - 2 has read its tiles
      a.put(st, kColPart, tid);
      publish(bar_c1 + 8 * s, lane);
      const uint32_t bad2 = clean(d);
      if (lane == 0) {
        words[0] = bad1;
        words[4] = bad2;
      }
      d.put(st + 3 * kColPart, kColPart, tid);
      publish(bar_c2 + 8 * s, lane);
      if (++ct == ct_hi) {
        ct = ct_lo;
        ++hc;
      }
    }
  } else {
    tc::reg_alloc<kBwdComputeRegs>();
    // ------------------------------------------------------------------ compute + output rows
    const int wg = warp >> 2;
    const int r = (warp & 3) * 32 + lane;  // row inside the tile == TMEM lane
    const int c0 = 32 * wg;                // first streamed position, and first channel, of this thread
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const int rg = rg0 + r;
    const float c = g.scale * kLog2e;
    float* vec = reinterpret_cast<float*>(gen + L::kVec) + warp * 64;  // warp-private
    float row_nl = 0.f, row_nd = 0.f;      // dQ part: -LSE and -delta (times 2^16) of this row
    if (!kKeyRows && rb + r < g.Lq) {
      const float v = p.lse[b * p.lse_sb + hr * p.lse_sh + (rb + r) * p.lse_sl];
      row_nl = v == -CUDART_INF_F ? 0.f : -v;
      row_nd = -p.delta[((long long)b * g.H + hr) * g.Lq + rb + r] * kUp;
    }
    float acc1[32], acc2[kKeyRows ? 32 : 1];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      acc1[i] = 0.f;
      if (kKeyRows) acc2[kKeyRows ? i : 0] = 0.f;
    }
    bool ok = true, repair = false;
    auto add_products = [&](int it) -> bool {  // of step `it`
      if (!warp_wait(bar_acc + 8 * (it & 1), (uint32_t)(it >> 1) & 1u, guard, kStSplitCompute)) return false;
      tc::tc_fence_after();
      uint32_t t[32];
      tc::tmem_ld32(tAcc1 + lane_sel + c0, t);
      tc::tmem_wait_ld();
#pragma unroll
      for (int i = 0; i < 32; ++i) acc1[i] += __uint_as_float(t[i]);
      if (kKeyRows) {
        tc::tmem_ld32(tAcc2 + lane_sel + c0, t);
        tc::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) acc2[kKeyRows ? i : 0] += __uint_as_float(t[i]);
      }
      return true;
    };
    auto send = [&](uint32_t t, uint32_t bar, const float* v) {  // parts of 32 values of a row over the scores they come from
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t xh[8], xm[8], xl[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) split2(v[q * 16 + 2 * i], v[q * 16 + 2 * i + 1], xh[i], xm[i], xl[i]);
        tmem_st8(t + q * 8, xh);
        tmem_st8(t + 16 + q * 8, xm);
        tmem_st8(t + 64 + q * 8, xl);
      }
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar);
    };
    int hc = kKeyRows ? hr * G : hr / G, ct = ct_lo;
    float nl_next = 0.f, nd_next = 0.f;  // key rows: LSE and delta of this lane's streamed position, a step ahead
    auto fetch_vec = [&]() {
      const int q = imin(ct * kCols + c0 + lane, g.Lq - 1);  // positions beyond Lq are masked out
      nl_next = p.lse[b * p.lse_sb + hc * p.lse_sh + q * p.lse_sl];
      nd_next = p.delta[((long long)b * g.H + hc) * g.Lq + q];
    };
    if (kKeyRows && n_it > 0) fetch_vec();
    for (int it = 0; it < n_it; ++it) {
      const uint32_t par = (uint32_t)it & 1u;
      const int cb = ct * kCols, cg0 = cb + c_off;
      const int ncols = imin(n - cg0, c_len - cb);
      if (++ct == ct_hi) {
        ct = ct_lo;
        ++hc;
      }
      if (kKeyRows) {
        __syncwarp();
        vec[lane] = nl_next == -CUDART_INF_F ? 0.f : -nl_next;
        vec[32 + lane] = -nd_next * kUp;
        __syncwarp();
        if (it + 1 < n_it) fetch_vec();
      }
      const bool has_full = kKeyRows ? M::kHasQFullRange : M::kHasKFullRange;
      const bool full = has_full && cg0 >= full_lo && cg0 + kCols <= full_hi && ncols >= kCols && rows_valid == kRows;
      if (!(ok = warp_wait(bar_s, par, guard, kStSplitCompute))) break;
      tc::tc_fence_after();
      auto sees = [&](int cc) {
        return rg < n && cc < ncols && (kKeyRows ? M::mask(cg0 + cc, rg, n, g.margs) : M::mask(rg, cg0 + cc, n, g.margs));
      };
      float pe[32];
      load_scores16(tS + lane_sel + c0, pe);
      load_scores16(tS + lane_sel + c0 + 16, pe + 16);
      if (!kKeyRows) {  // S has been read
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar_p);
      }
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        float4 nl = make_float4(row_nl, row_nl, row_nl, row_nl);
        if (kKeyRows) nl = *reinterpret_cast<const float4*>(vec + i);
        pe[i] = tc::ex2(fmaf(pe[i], c, nl.x));
        pe[i + 1] = tc::ex2(fmaf(pe[i + 1], c, nl.y));
        pe[i + 2] = tc::ex2(fmaf(pe[i + 2], c, nl.z));
        pe[i + 3] = tc::ex2(fmaf(pe[i + 3], c, nl.w));
      }
      uint32_t vis = 0xffffffffu;  // bit i: this row and position c0 + i
      if (!full) {
        vis = 0;
        if (interval_rows<M>::value) {
          int lo, hi;
          row_window<M, !kKeyRows>(rg, cg0, ncols, n, g.margs, lo, hi);
#pragma unroll
          for (int i = 0; i < 32; ++i) vis |= (c0 + i >= lo && c0 + i <= hi) ? 1u << i : 0u;
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) vis |= sees(c0 + i) ? 1u << i : 0u;
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) pe[i] = ((vis >> i) & 1u) ? pe[i] : 0.f;
      }
      if (it > 0 && !(ok = add_products(it - 1))) break;  // before this step's products replace them
      if (kKeyRows) send(tS + lane_sel + c0, bar_p, pe);
      if (!(ok = warp_wait(bar_dp, par, guard, kStSplitCompute))) break;
      tc::tc_fence_after();
      for_unfit(reinterpret_cast<const uint4*>(gen + L::kUnfit + 32 * (it & 1)), [&](int pos, bool, bool) { repair = repair || sees(pos); });
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float d[16];
        load_scores16(tdP + lane_sel + c0 + q * 16, d);
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          float4 nd = make_float4(row_nd, row_nd, row_nd, row_nd);
          if (kKeyRows) nd = *reinterpret_cast<const float4*>(vec + 32 + q * 16 + i);
          pe[q * 16 + i] *= fmaf(d[i], kUp, nd.x);
          pe[q * 16 + i + 1] *= fmaf(d[i + 1], kUp, nd.y);
          pe[q * 16 + i + 2] *= fmaf(d[i + 2], kUp, nd.z);
          pe[q * 16 + i + 3] *= fmaf(d[i + 3], kUp, nd.w);
        }
      }
      if (!full) {  // once more: delta of a hidden query may be NaN
#pragma unroll
        for (int i = 0; i < 32; ++i) pe[i] = ((vis >> i) & 1u) ? pe[i] : 0.f;
      }
      send(tdP + lane_sel + c0, bar_ds, pe);
    }
    if (ok && n_it > 0) ok = add_products(n_it - 1);

    // ---- rows: this thread has channels [c0, c0 + 32) of one row; the first warpgroup marks a row with a NaN in either half
    volatile int* bad = reinterpret_cast<volatile int*>(gen + L::kBad);
    float nan = repair || (n_it > 0 && is_small(row_small, r)) ? CUDART_NAN_F : 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      nan += acc1[i] - acc1[i];
      if (kKeyRows) nan += acc2[kKeyRows ? i : 0] - acc2[kKeyRows ? i : 0];
    }
    if (wg == 1) {
      bad[r] = nan != nan ? 1 : 0;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar_bad);
    } else if (ok) {
      ok = warp_wait(bar_bad, 0, guard, kStSplitCompute);
    }
    if (ok && r < rows_in && c0 < D) {
      const bool valid = r < rows_valid;
      const TRef& t1 = kKeyRows ? p.dk : p.dq;
      float* d1 = static_cast<float*>(t1.p) + b * t1.sb + hr * t1.sh + (long long)(rb + r) * t1.sl + c0;
#pragma unroll
      for (int i = 0; i < 32; ++i) acc1[i] = valid ? acc1[i] * (g.scale * kDown) : 0.f;
      if (valid && wg == 0 && (nan != nan || bad[r] != 0)) acc1[0] = __uint_as_float(kRepairMark);
      store_row_f32(d1, acc1, 16);
      if (c0 + 16 < D) store_row_f32(d1 + 16, acc1 + 16, 16);
      if constexpr (kKeyRows) {
        float* d2 = static_cast<float*>(p.dv.p) + b * p.dv.sb + hr * p.dv.sh + (long long)(rb + r) * p.dv.sl + c0;
#pragma unroll
        for (int i = 0; i < 32; ++i) acc2[i] = valid ? acc2[i] : 0.f;
        store_row_f32(d2, acc2, 16);
        if (c0 + 16 < D) store_row_f32(d2 + 16, acc2 + 16, 16);
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 12) tc::tmem_dealloc(tmem, 512);
}

// One launch for both halves, as in simt.cuh.
template <class M>
__global__ void __launch_bounds__(kBwdThreads, 1) split_bwd_kernel(const __grid_constant__ BwdParams pp) {
  extern __shared__ uint8_t smem_raw[];
  if ((int)blockIdx.x < pp.n_key_ctas) bwd_body<M, true>(pp, smem_raw, (int)blockIdx.x);
  else bwd_body<M, false>(pp, smem_raw, (int)blockIdx.x - pp.n_key_ctas);
}

}  // namespace split
}  // namespace chill
