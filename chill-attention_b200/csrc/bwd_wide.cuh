// Backward attention for head dim 256 on tcgen05 tensor cores (sm_100a, 16-bit inputs).
//
// At D = 256 the accumulators of dK and dV alone would fill TMEM (2 x 256 of 512 columns), so the gradients are
// computed by THREE launches of one kernel template, each with a single 128 x 256 accumulator and the scores
// recomputed (eight GEMMs per tile pair instead of the five of the single-kernel backward for D <= 128):
//
//   kWideDV  one CTA per (batch, kv head, 128 keys):   S^T = K Q^T,                  W = P^T,                dV += W dO
//   kWideDK  same rows:                                S^T = K Q^T, dP^T = V dO^T,   W = P^T (dP^T - delta), dK += W Q
//   kWideDQ  one CTA per (batch, head, 128 queries):   S = Q K^T,   dP = dO V^T,     W = P (dP - delta),     dQ += W K
//
// with P = 2^(S c - LSE) from the stored LSE (no running maximum).  The "row" operands (K / V, resp. Q / dO: 64 KB
// each) stay in shared memory, the other axis streams through in tiles of 64 positions, clipped by the mask functor's
// range function.  Two buffers of scores in TMEM and two stages of the "late" tile, which the accumulating GEMM reads (the
// "early" one, read by a score GEMM only, has what shared memory leaves: one stage, for dV two), let the issuing thread run
//     scores(j + 1)   accumulate(j)   scores(j + 2) ...
// so the elementwise work of a step hides behind the scores of the next one and the loads behind both.  Roles: warps 0-7 own one
// tile row per thread and one half of the 64 positions and turn the fp32 scores in TMEM into the 16-bit W (written over the
// scores that the same thread has read, A operand of the accumulating GEMM), warp 8 is the TMA producer, warp 9 owns TMEM and
// issues the MMAs.
// TMEM columns: [0,128) two buffers of S (W over them), [128,256) of dP, [256,512) accumulator.
//
// Measured (causal bf16 (2,16,4096,256), dV / dK / dQ in us): 338 / 522 / 558 with one stage, one buffer of scores and four
// elementwise warps (each step a chain of load, scores, elementwise, accumulate), 250 / 403 / 436 with two, 253 / 378 / 432 with
// eight warps as well, which masked tiles need (chunkwise(100, 3) (2,8/4,2048): all three 580 -> 521 -> 323).  What bounds them now is
// the chain again: tensor pipe 46 to 52 %, shared-memory data pipe 52 to 61 % (a score MMA with N = 64 reads 6 KB in its 48 clocks),
// L2 17 to 34 %, DRAM 9 to 11 % (counters: profiles/c2d256s_causal_bf16_bwd_wide_ncu.md).
// Reference math: chill_attention/chill_bwd_dkdv.py:347-508, chill_bwd_dq.py:300-394.
#pragma once
#include "bwd_tc.cuh"

namespace chill {
namespace tc {

enum : int { kWideDV = 0, kWideDK = 1, kWideDQ = 2 };
constexpr int kWideThreads = 384;  // warps 0-7 elementwise + epilogue, 8 TMA producer, 9 MMA issuer, 10-11 idle

constexpr int kWideAlign = 128;  // of the dynamic shared memory, as declared

template <int D, int MODE>
struct WideSmem {
  static constexpr int kRowBytes = kTile * D * 2;      // a 128-row operand
  static constexpr int kColBytes = kWideCols * D * 2;  // a 64-row streamed tile
  static constexpr int kEarly = MODE == kWideDV ? 2 : 1;  // stages of the tile that only a score GEMM reads
  static constexpr int kR1 = 0;
  static constexpr int kR2 = kR1 + kRowBytes;
  static constexpr int kE = MODE == kWideDV ? kR2 : kR2 + kRowBytes;
  static constexpr int kL = kE + kEarly * kColBytes;   // two stages of the tile the accumulating GEMM reads
  static constexpr int kVec = kL + 2 * kColBytes;      // per warp: -LSE and -delta of 32 streamed columns
  static constexpr int kBars = kVec + 8 * 2 * 32 * 4;
  static constexpr int kNumBars = 14;
  static constexpr int kMisc = kBars + 8 * kNumBars;
  static constexpr int kTotal = kMisc + 16;
  // What aligning the declared base to 1 KB by hand can take.  (Declared with 1 KB the kernels need none of it, but all three together
  // take 10 % longer on causal (2,16,4096,256): 1087 -> 1200 us with delta.)
  static constexpr int kDynamic = kTotal + 1024 - kWideAlign;
};

enum : int { kStWideProducer = 501, kStWideMma = 502, kStWideCompute = 503, kStWideEpilogue = 504 };

// maps: R1, R2 = 128-row boxes of the row operands; C1, C2 = 64-row boxes of the streamed operands; OUT = 128-row
// box of the gradient written.  kWideDV: R1 = K, (R2 unused), C1 = Q, C2 = dO, OUT = dV.  kWideDK: R1 = K, R2 = V,
// C1 = Q, C2 = dO, OUT = dK.  kWideDQ: R1 = Q, R2 = dO, C1 = K, C2 = V, OUT = dQ.
template <typename T, int D, class M, int MODE>
__global__ void __launch_bounds__(kWideThreads, 1)
bwd_wide_kernel(const __grid_constant__ CUtensorMap tmR1, const __grid_constant__ CUtensorMap tmR2,
                const __grid_constant__ CUtensorMap tmC1, const __grid_constant__ CUtensorMap tmC2,
                const __grid_constant__ CUtensorMap tmOut, BwdTcParams p) {
  using L = WideSmem<D, MODE>;
  constexpr bool kKeyRows = MODE != kWideDQ;   // tile rows are keys (dV, dK) or queries (dQ)
  constexpr bool kTwoScores = MODE != kWideDV;  // dP is needed as well
  constexpr int CT = kWideCols;
  constexpr int kChunks = D / 64;
  constexpr int kChunkBytes = kTile * 128;  // one 64-channel column block of a 128-row tile
  constexpr int kColChunkBytes = CT * 128;  // the same of a streamed tile
  const Geo& g = p.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = g.H / g.Hkv;
  const int n_rt = ((kKeyRows ? g.Lk : g.Lq) + kTile - 1) / kTile;
  const int n_units = kKeyRows ? g.B * g.Hkv : g.B * g.H;
  int unit, rank;
  cta_order((int)blockIdx.x, n_units, n_rt, unit, rank);
  const int rt = kKeyRows ? rank : n_rt - 1 - rank;  // longest tiles first under a causal mask
  const int hr = kKeyRows ? unit % g.Hkv : unit % g.H;  // head index of the row operands
  const int b = kKeyRows ? unit / g.Hkv : unit / g.H;
  const int hk = kKeyRows ? hr : hr / G;
  const int rb = rt * kTile;                                   // first local row
  const int rg0 = rb + (kKeyRows ? g.k_off : g.q_off);         // its global position
  const int rows_here = imin(kTile, (kKeyRows ? g.Lk : g.Lq) - rb);
  int n = g.seq_len;
  if (g.lens != nullptr) n = imin(n, g.lens[b]);

  // ---- range of the streamed axis, in tiles of CT local positions
  int ct_lo = 0, ct_hi = 0;
  if (rg0 < n) {
    int lo, hi;
    tile_range<M, !kKeyRows>(rg0, rows_here, n, g.margs, lo, hi);
    const int off = kKeyRows ? g.q_off : g.k_off, len = kKeyRows ? g.Lq : g.Lk;
    const int lo_l = imax(lo - off, 0);
    const int hi_l = imin(imin(hi, n - 1) - off, len - 1);
    if (hi_l >= lo_l) {
      ct_lo = lo_l / CT;
      ct_hi = hi_l / CT + 1;
    }
  }
  const int n_ct = ct_hi - ct_lo;
  const int n_it = n_ct * (kKeyRows ? G : 1);  // key rows: every head of the GQA group contributes
  T* out_base = reinterpret_cast<T*>(MODE == kWideDV ? p.dv : (MODE == kWideDK ? p.dk : p.dq));
  const long long o_sb = MODE == kWideDV ? p.dv_sb : (MODE == kWideDK ? p.dk_sb : p.dq_sb);
  const long long o_sh = MODE == kWideDV ? p.dv_sh : (MODE == kWideDK ? p.dk_sh : p.dq_sh);
  const long long o_sl = MODE == kWideDV ? p.dv_sl : (MODE == kWideDK ? p.dk_sl : p.dq_sl);
  if (n_it == 0) {  // padding rows, or rows nothing on this shard can see: zero gradient
    zero_rows<T>(out_base + b * o_sb + hr * o_sh + rb * o_sl, o_sl, rows_here, D, kWideThreads);
    if (MODE == kWideDV) zero_part_rows<D>(p.part, b, hr, rb, rows_here, g.Lk, kWideThreads);  // dK and dV partials
    return;
  }

  extern __shared__ __align__(kWideAlign) uint8_t smem_wide[];
  const uint32_t base = (smem_u32(smem_wide) + 1023u) & ~1023u;
  uint8_t* gen_base = smem_wide + (base - smem_u32(smem_wide));
  const uint32_t sR1 = base + L::kR1, sR2 = base + L::kR2, sE = base + L::kE, sL = base + L::kL;
  const uint32_t bars = base + L::kBars;
  // "Early" tile: Q for dV, dO / V for dK / dQ, read by one score GEMM (e_done: that GEMM has finished).  "Late" tile: also, or
  // only, the B operand of the accumulating GEMM.  Per stage + 8 s.  t_full: the scores of a step are there.
  const uint32_t bar_r_full = bars, bar_acc_full = bars + 8, bar_e_full = bars + 16, bar_e_done = bars + 32, bar_l_full = bars + 48,
                 bar_l_empty = bars + 64, bar_t_full = bars + 80, bar_w_full = bars + 96;
  constexpr int NE = L::kEarly;
  const CUtensorMap* tmEarly = MODE == kWideDV ? &tmC1 : &tmC2;
  const CUtensorMap* tmLate = MODE == kWideDV ? &tmC2 : &tmC1;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen_base + L::kMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen_base + L::kMisc + 4);
  const Guard guard{p.status, abort_flag};
  const int col_head0 = kKeyRows ? hk * G : hk;  // head of the first streamed tile

  if (warp == 8) {
    if (lane == 0) {
      *abort_flag = 0;
      mbar_init(bar_r_full, 1);
      mbar_init(bar_acc_full, 1);
      for (int s = 0; s < 2; ++s) {
        mbar_init(bar_e_full + 8 * s, 1);
        mbar_init(bar_e_done + 8 * s, 1);
        mbar_init(bar_l_full + 8 * s, 1);
        mbar_init(bar_l_empty + 8 * s, 1);
        mbar_init(bar_t_full + 8 * s, 1);
        mbar_init(bar_w_full + 8 * s, 8);
      }
      fence_barrier_init();
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(bar_r_full, (kTwoScores ? 2 : 1) * L::kRowBytes);
      for (int c = 0; c < kChunks; ++c) {
        tma_load_4d(sR1 + c * kChunkBytes, &tmR1, bar_r_full, c * 64, rb, hr, b);
        if (kTwoScores) tma_load_4d(sR2 + c * kChunkBytes, &tmR2, bar_r_full, c * 64, rb, hr, b);
      }
    }
  } else if (warp == 9) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // two buffers of scores: + CT per buffer
  const uint32_t tS = tmem, tdP = tmem + 2 * CT, tAcc = tmem + 4 * CT;

  if (warp == 8) {
    // ------------------------------------------------------------------- TMA producer
    if (lane == 0) {
      bool ok = true;
      int ct = ct_lo, hc = col_head0;
      for (int it = 0; it < n_it && ok; ++it) {
        const uint32_t es = (uint32_t)(it % NE), ls = (uint32_t)it & 1u;
        ok = it < NE || mbar_wait(bar_e_done + 8 * es, (uint32_t)(it / NE - 1) & 1u, guard, kStWideProducer);
        if (!ok) break;
        mbar_arrive_expect_tx(bar_e_full + 8 * es, L::kColBytes);
        for (int c = 0; c < kChunks; ++c)
          tma_load_4d(sE + es * L::kColBytes + c * kColChunkBytes, tmEarly, bar_e_full + 8 * es, c * 64, ct * CT, hc, b);
        ok = it < 2 || mbar_wait(bar_l_empty + 8 * ls, (uint32_t)((it >> 1) - 1) & 1u, guard, kStWideProducer);
        if (!ok) break;
        mbar_arrive_expect_tx(bar_l_full + 8 * ls, L::kColBytes);
        for (int c = 0; c < kChunks; ++c)
          tma_load_4d(sL + ls * L::kColBytes + c * kColChunkBytes, tmLate, bar_l_full + 8 * ls, c * 64, ct * CT, hc, b);
        if (++ct == ct_hi) {
          ct = ct_lo;
          ++hc;
        }
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 9) {
    // --------------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc<T>(kTile, CT, false, false);
      constexpr uint32_t idesc_acc = make_idesc<T>(kTile, D, false, true);  // A from TMEM, B MN-major
      constexpr uint32_t hi_k = desc_hi_sw128(1024);
      const uint32_t r1_lo = desc_lo_sw128(sR1, 16), r2_lo = desc_lo_sw128(sR2, 16);
      const uint32_t e_lo = desc_lo_sw128(sE, 16), l_lo = desc_lo_sw128(sL, 16);
      const uint32_t x_lo = desc_lo_sw128(sL, kColChunkBytes);  // MN-major, channel blocks one chunk apart
      constexpr uint32_t kStage = L::kColBytes / 16;
      bool ok = mbar_wait(bar_r_full, 0, guard, kStWideMma);
      auto score = [&](uint32_t t_dst, uint32_t r_lo, uint32_t c_lo) {  // rows x 64 positions, contraction over D
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          mma_ss_lh(t_dst, r_lo + kmajor_step(kk), c_lo + (uint32_t)((kk / 4) * (kColChunkBytes / 16) + (kk % 4) * 2), hi_k,
                    idesc_s, kk > 0 ? 1u : 0u);
      };
      // Scores of step `it` into buffer it % 2: over W and dP of step it - 2, whose accumulating GEMM was issued before.
      auto scores = [&](int it) -> bool {
        const uint32_t es = (uint32_t)(it % NE), buf = (uint32_t)it & 1u;
        if (!mbar_wait(bar_e_full + 8 * es, (uint32_t)(it / NE) & 1u, guard, kStWideMma)) return false;
        tc_fence_after();
        if (MODE == kWideDV) score(tS + buf * CT, r1_lo, e_lo + es * kStage);
        else score(tdP + buf * CT, r2_lo, e_lo + es * kStage);
        mma_commit(bar_e_done + 8 * es);
        if (kTwoScores) {
          if (!mbar_wait(bar_l_full + 8 * buf, (uint32_t)(it >> 1) & 1u, guard, kStWideMma)) return false;
          tc_fence_after();
          score(tS + buf * CT, r1_lo, l_lo + buf * kStage);
        }
        mma_commit(bar_t_full + 8 * buf);
        return true;
      };
      if (ok) ok = scores(0);
      for (int it = 0; it < n_it && ok; ++it) {
        const uint32_t buf = (uint32_t)it & 1u, par = (uint32_t)(it >> 1) & 1u;
        if (it + 1 < n_it && !(ok = scores(it + 1))) break;  // runs during the elementwise work of step `it`
        if (!kTwoScores && !(ok = mbar_wait(bar_l_full + 8 * buf, par, guard, kStWideMma))) break;
        if (!(ok = mbar_wait(bar_w_full + 8 * buf, par, guard, kStWideMma))) break;
        tc_fence_after();
        // accumulator += W X: W (16-bit) from TMEM, 16 streamed positions = 8 columns of W and 2 KB of X per MMA
#pragma unroll
        for (int kk = 0; kk < CT / 16; ++kk)
          mma_ts_lh(tAcc, tS + buf * CT + (kk / 2) * 32 + (kk % 2) * 8, x_lo + buf * kStage + kk * 128, hi_k, idesc_acc, (it > 0 || kk > 0) ? 1u : 0u);
        mma_commit(bar_l_empty + 8 * buf);
      }
      if (ok) mma_commit(bar_acc_full);
    }
  } else if (warp < 8) {
    // --------------------------------------------------------- elementwise + epilogue warps
    const int wg = warp >> 2;               // half of the streamed positions: [32 wg, 32 wg + 32)
    const int r = (warp & 3) * 32 + lane;   // row inside the tile == TMEM lane
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const int c0 = 32 * wg;
    const int rg = rg0 + r;  // global position of this thread's row (a key, or a query for kWideDQ)
    const bool row_ok = rg < n && r < rows_here;
    const float c = g.scale * kLog2e;
    float row_nl = 0.f, row_nd = 0.f;  // kWideDQ: -LSE and -delta of this thread's query row
    if (!kKeyRows && r < rows_here) {
      const float lv = p.lse[b * p.lse_sb + hr * p.lse_sh + (rb + r) * p.lse_sl];
      row_nl = (lv == -CUDART_INF_F) ? 0.f : -lv;
      row_nd = -p.delta[((long long)b * g.H + hr) * g.Lq + rb + r];
    }
    // streamed positions that EVERY row of this tile sees (half-open, global): tiles inside skip the mask arithmetic
    int full_lo = 0, full_hi = 0;
    constexpr bool kHasFull = kKeyRows ? M::kHasQFullRange : M::kHasKFullRange;
    if (kHasFull && rg0 + kTile <= n && rows_here == kTile) {
      if (kKeyRows) M::q_full_range_for_k(rg0, kTile, n, g.margs, full_lo, full_hi);
      else M::k_full_range_for_q(rg0, kTile, n, g.margs, full_lo, full_hi);
    }
    bool ok = true;
    float* vb = reinterpret_cast<float*>(gen_base + L::kVec) + warp * 64;  // warp-private copy: no barrier across warps inside the loop
    int ct = ct_lo, hc = col_head0;
    // LSE and delta of this lane's query column, fetched a step ahead
    float nl_next = 0.f, nd_next = 0.f;
    auto fetch_cols = [&]() {
      const int q = imin(ct * CT + c0 + lane, g.Lq - 1);
      nl_next = __ldg(p.lse + b * p.lse_sb + hc * p.lse_sh + q * p.lse_sl);
      if (kTwoScores) nd_next = __ldg(p.delta + ((long long)b * g.H + hc) * g.Lq + q);
    };
    if (kKeyRows) fetch_cols();
    for (int it = 0; it < n_it; ++it) {
      const uint32_t par = (uint32_t)(it >> 1) & 1u, buf = (uint32_t)it & 1u;
      const int cpos = ct * CT;  // first local position of the streamed tile
      const int cg0 = cpos + (kKeyRows ? g.q_off : g.k_off);
      const int clim = imin(n - cg0, (kKeyRows ? g.Lq : g.Lk) - cpos);  // streamed positions >= clim do not exist
      if (++ct == ct_hi) {
        ct = ct_lo;
        ++hc;
      }
      if (kKeyRows) {
        __syncwarp();  // the previous step's reads of vb are done
        vb[lane] = nl_next == -CUDART_INF_F ? 0.f : -nl_next;
        if (kTwoScores) vb[32 + lane] = -nd_next;
        __syncwarp();
        if (it + 1 < n_it) fetch_cols();
      }
      ok = mbar_wait(bar_t_full + 8 * buf, par, guard, kStWideCompute);
      ok = __all_sync(0xffffffffu, ok);  // keep the warp converged for the .sync.aligned TMEM accesses
      if (!ok) break;
      tc_fence_after();
      const bool full = kHasFull && cg0 >= full_lo && cg0 + CT <= full_hi && clim >= CT;
      uint32_t w[CT / 4];
      auto body = [&](auto masked_tag) {  // two copies: full tiles run without any mask arithmetic
        constexpr bool kMasked = decltype(masked_tag)::value;
        uint32_t sreg[32], dreg[32];
        tmem_ld32(tS + buf * CT + lane_sel + c0, sreg);
        if (kTwoScores) tmem_ld32(tdP + buf * CT + lane_sel + c0, dreg);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          float4 nl4 = make_float4(row_nl, row_nl, row_nl, row_nl), nd4 = make_float4(row_nd, row_nd, row_nd, row_nd);
          if (kKeyRows) {
            nl4 = *reinterpret_cast<const float4*>(vb + i);
            if (kTwoScores) nd4 = *reinterpret_cast<const float4*>(vb + 32 + i);
          }
          const float nl[4] = {nl4.x, nl4.y, nl4.z, nl4.w}, nd[4] = {nd4.x, nd4.y, nd4.z, nd4.w};
          float wv[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int cc = c0 + i + e;
            float pv = ex2(fmaf(__uint_as_float(sreg[i + e]), c, nl[e]));
            if (kMasked) {
              const int qg = kKeyRows ? cg0 + cc : rg, kg = kKeyRows ? rg : cg0 + cc;
              pv = (row_ok && cc < clim && M::mask(qg, kg, n, g.margs)) ? pv : 0.f;
            }
            if (kTwoScores) pv *= __uint_as_float(dreg[i + e]) + nd[e];
            wv[e] = pv;
          }
          w[i / 2] = pack2<T>(wv[0], wv[1]);
          w[i / 2 + 1] = pack2<T>(wv[2], wv[3]);
        }
      };
      if (full) body(std::false_type{});
      else body(std::true_type{});
      tmem_st16(tS + buf * CT + lane_sel + c0, w);  // 16 columns of 16-bit pairs over scores that only this thread reads
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_w_full + 8 * buf);
    }

    // ---- epilogue: accumulator (x sm_scale for dK, dQ) -> 16-bit -> swizzled shared memory (R1's buffer) -> TMA store
    if (ok) ok = mbar_wait(bar_acc_full, 0, guard, kStWideEpilogue);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    const float mul = MODE == kWideDV ? 1.f : g.scale;
    // optional un-rounded fp32 copy of this key row's dV / dK (first / last key rows of the call, see PartOut)
    float* part_row = kKeyRows ? p.part.row(MODE == kWideDV ? p.part.dv : p.part.dk, b, hr, rb + r, g.Lk) : nullptr;
#pragma unroll 1
    for (int q4 = wg * (D / 64); q4 < (wg + 1) * (D / 64); ++q4) {
      uint32_t acc[32];
      if (ok) {
        tmem_ld32(tAcc + lane_sel + q4 * 32, acc);
        tmem_wait_ld();
      }
      stage_row32<T>(gen_base + L::kR1, r, q4, acc, mul, ok && row_ok);
      if (part_row != nullptr) store_part32(part_row + q4 * 32, acc, mul, ok && row_ok);
    }
    fence_proxy_async_smem();
    named_bar_sync(1, 256);
    if (threadIdx.x == 0) {
      for (int cc = 0; cc < kChunks; ++cc) tma_store_4d(&tmOut, sR1 + cc * kChunkBytes, cc * 64, rb, hr, b);
      tma_store_commit();
      tma_store_wait_read();  // shared memory may be released; the global writes complete by kernel end
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, 512);
}

// maps: 0 Q128, 1 K128, 2 V128, 3 dO128 (128-row boxes), 4 Q64, 5 K64, 6 V64, 7 dO64 (64-row boxes), 8 dQ, 9 dK, 10 dV
template <typename T, class M>
int launch_bwd_wide(const CUtensorMap* maps, const BwdTcParams& p, cudaStream_t st) {
  constexpr int D = 256;
  static_assert(WideSmem<D, kWideDK>::kDynamic <= 232448, "exceeds the 227 KB of shared memory a CTA can opt in to");
  const Geo& g = p.g;
  const unsigned key_ctas = (unsigned)(((g.Lk + kTile - 1) / kTile) * g.Hkv * g.B);
  const unsigned query_ctas = (unsigned)(((g.Lq + kTile - 1) / kTile) * g.H * g.B);
  cudaError_t e;
  {
    auto kern = bwd_wide_kernel<T, D, M, kWideDV>;
    constexpr int smem = WideSmem<D, kWideDV>::kDynamic;
    struct Tag {};
    if ((e = ensure_dynamic_smem<Tag>(kern, smem)) != cudaSuccess) return (int)e;
    kern<<<key_ctas, kWideThreads, smem, st>>>(maps[1], maps[2], maps[4], maps[7], maps[10], p);
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  }
  {
    auto kern = bwd_wide_kernel<T, D, M, kWideDK>;
    constexpr int smem = WideSmem<D, kWideDK>::kDynamic;
    struct Tag {};
    if ((e = ensure_dynamic_smem<Tag>(kern, smem)) != cudaSuccess) return (int)e;
    kern<<<key_ctas, kWideThreads, smem, st>>>(maps[1], maps[2], maps[4], maps[7], maps[9], p);
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  }
  {
    auto kern = bwd_wide_kernel<T, D, M, kWideDQ>;
    constexpr int smem = WideSmem<D, kWideDQ>::kDynamic;
    struct Tag {};
    if ((e = ensure_dynamic_smem<Tag>(kern, smem)) != cudaSuccess) return (int)e;
    kern<<<query_ctas, kWideThreads, smem, st>>>(maps[0], maps[3], maps[5], maps[6], maps[8], p);
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  }
  return 0;
}

template <class M>
int launch_bwd_wide_all(int dtype, const CUtensorMap* maps, const BwdTcParams& p, cudaStream_t st) {
  if (dtype == 2) return launch_bwd_wide<__nv_bfloat16, M>(maps, p, st);
  if (dtype == 1) return launch_bwd_wide<__half, M>(maps, p, st);
  return (int)cudaErrorInvalidValue;
}

}  // namespace tc
}  // namespace chill
