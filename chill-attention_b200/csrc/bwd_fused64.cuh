// Single-kernel backward for 16-bit inputs of head dim 64 (and 16 / 32, whose tensor maps have the true width).  The same
// five GEMMs, dQ accumulator and roles as bwd_fused.cuh, cut so that TWO CTAs share an SM.
//
// With one CTA per SM and 128-query steps the tensor cores idle while a CTA sets up, fills its ring, waits for its first
// scores and stores its results: about 13 000 of the 22 000 clocks a CTA took on a chunkwise mask (three query tiles per key
// tile).  At head dim 64 half of that kernel's resources suffice if the queries come in steps of 64: TMEM holds
// S^T 64 | dP^T 64 | dV 64 | dK 64 = 256 columns, shared memory K, V, two 64-query stages of [Q | dO] and the dS^T tile
// (113 KB), so one CTA's fixed part and the latencies of its chain overlap the other's MMAs.
// Chunkwise (128, 2) fp16 (4,32,16384,64): 1131 -> 968 us, window(16, 16) (8,12,2085,64): 124 -> 89 us against that kernel.
// What bounds it now is the chain of each CTA (about 3400 clocks per step, of which 1000 exponentials): of the kernel's time on
// (4,8,16384,64) the tensor pipe is active 24 %, the shared-memory pipe 36 %, instructions issue 51 %, DRAM delivers 2.3 TB/s.
// Leaving out the dQ reductions alone gains 8 %, the exponentials 5 %.  Variants, both against 993 us of an earlier state of
// this kernel: persistent CTAs that overlap one tile's stores with the next one's loads 1026 us; four compute warps instead of
// eight 981 us, but 95 against 89 us on the narrow window.
//
// A step is 64 queries; two steps form a query tile, the unit of the dQ GEMM (M = 128 queries) and of the accumulator:
//     S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q          every step
//     dQ = dS K  into the columns of dP^T                              last step of a query tile that the mask leaves
// The steps of a key tile start at the 32-row group of the first query that sees it (the accumulator is made of such groups), and
// query tiles are pairs of them; if the last one has one step only, the dQ rows of the other half are not drained (the dS^T
// columns they come from are stale).  With steps at multiples of 64 and tiles at multiples of 128, a window(16, 16) took four
// steps and three dQ tiles per key tile instead of three and two: fp16 (8,12,2085,64) 91 -> 79 us.
//
// Order of the issuing thread for step u:   dV(u)  S(u+1)  [dQ]  dK(u)  dP(u+1)
//     dV(u)    needs P^T(u)             | compute warps: wait for dP^T(u)
//     S(u+1)   overwrites P^T(u) (in order after dV(u))
//     dK(u)    needs dS^T(u)            | compute warps: exponentials of S^T(u+1)
//     dP(u+1)  needs dP^T(u) read (implied by dS^T(u)), or dQ drained
// dS^T of a step may be written as soon as dP^T of that step is complete: every GEMM that read the previous contents of
// the buffer was issued before it.
//
// Roles (512 threads): warps 0-7 compute (thread (w % 4) * 32 + lane = key row = TMEM lane; warps 0-3 / 4-7 split the 64 query
// columns), warps 8-11 drain dQ, warp 12 TMA producer and TMEM owner, warp 13 MMA issuer; 14 and 15 only complete the
// warpgroup for setmaxnreg.
#pragma once
#include <type_traits>

#include "bwd_fused.cuh"

namespace chill {
namespace tc {

constexpr int kF64Threads = 512;
constexpr int kF64LaunchRegs = 65536 / (2 * kF64Threads);
constexpr int kF64ComputeRegs = 80, kF64DrainRegs = 48, kF64OtherRegs = 48;
static_assert(2 * kF64ComputeRegs + kF64DrainRegs + kF64OtherRegs <= 4 * kF64LaunchRegs, "setmaxnreg.inc would never be granted");
constexpr int kF64TmemCols = 256;

enum : int { kStF64Producer = 601, kStF64Mma = 602, kStF64Compute = 603, kStF64Drain = 604, kStF64Epilogue = 605 };

struct Fused64Smem {
  static constexpr int kTileBytes = kTile * 128;         // K, V, dK, dV: 128 rows of one 128-byte line
  static constexpr int kStepBytes = kF64Step * 128;      // Q or dO of one step
  static constexpr int kStages = 2;
  static constexpr int kK = 0;
  static constexpr int kV = kK + kTileBytes;
  static constexpr int kRing = kV + kTileBytes;          // per stage: [Q | dO]; in the epilogue the dV and dK staging tiles
  static constexpr int kDs = kRing + kStages * 2 * kStepBytes;  // two 64-query chunks of [128 keys][64 queries]
  static constexpr int kDrainChunkBytes = 8 * 32 * 4;    // 8 channels of a drain warp's 32 rows, fp32
  static constexpr int kDrainBufs = 3;
  static constexpr int kDrain = kDs + 2 * kTileBytes;
  static constexpr int kRows = kDrain + 4 * kDrainBufs * kDrainChunkBytes;  // per compute warp: -lse[32], -delta[32]
  static constexpr int kBars = kRows + 8 * 2 * 32 * 4;
  static constexpr int kNumBars = 8 + 2 * kStages;
  static constexpr int kMisc = kBars + 8 * kNumBars;
  static constexpr int kTotal = kMisc + 16;
  static constexpr int kDynamic = kTotal + 1024;
  static_assert(kStages * 2 * kStepBytes == 2 * kTileBytes, "the ring doubles as staging for dV and dK");
  static_assert(2 * (kDynamic + 1024) <= 228 * 1024, "two CTAs per SM (the system keeps 1 KB per CTA)");
};

template <typename T, class M>
__global__ void __launch_bounds__(kF64Threads, 2)
bwd_fused64_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                      const __grid_constant__ CUtensorMap tmdK, const __grid_constant__ CUtensorMap tmdV, BwdTcParams p) {
  using L = Fused64Smem;
  constexpr int D = 64;
  const Geo& g = p.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int hb, kt;
  cta_order((int)blockIdx.x, g.B * g.Hkv, (g.Lk + kTile - 1) / kTile, hb, kt);  // first key tile = most query tiles (causal)
  const int hk = hb % g.Hkv, b = hb / g.Hkv;
  const int G = g.H / g.Hkv;
  const int kb = kt * kTile;
  const int kg0 = kb + g.k_off;
  const int n_qt_total = (g.Lq + kTile - 1) / kTile;
  int n = g.seq_len;
  if (g.lens != nullptr) n = imin(n, g.lens[b]);

  // steps of 64 queries that can see this key tile, from the 32-row group of the first such query on
  int q_row0 = 0, n_qs = 0, full_lo = 0, full_hi = 0;
  if (kg0 < n) {
    int lo, hi;
    tile_range<M, false>(kg0, imin(kTile, g.Lk - kb), n, g.margs, lo, hi);
    const int lo_l = imax(lo - g.q_off, 0);
    const int hi_l = imin(imin(hi, n - 1) - g.q_off, g.Lq - 1);
    if (hi_l >= lo_l) {
      n_qs = (hi_l - (lo_l & ~31)) / kF64Step + 1;
      // The last step does not end beyond the multiple of 64 behind the last such query (see bwd_fused.cuh).
      q_row0 = imin(lo_l & ~31, (hi_l / kF64Step + 1 - n_qs) * kF64Step);
    }
    if (M::kHasQFullRange) M::q_full_range_for_k(kg0, kTile, n, g.margs, full_lo, full_hi);
  }
  const int n_it = n_qs * G;
  if (n_it == 0) {
    // nobody attends these keys (padding, or outside every query's range on this shard)
    const int rows = imin(kTile, g.Lk - kb);
    zero_rows<T>(reinterpret_cast<T*>(p.dk) + b * p.dk_sb + hk * p.dk_sh + kb * p.dk_sl, p.dk_sl, rows, g.D, kF64Threads);
    zero_rows<T>(reinterpret_cast<T*>(p.dv) + b * p.dv_sb + hk * p.dv_sh + kb * p.dv_sl, p.dv_sl, rows, g.D, kF64Threads);
    zero_part_rows<D>(p.part, b, hk, kb, rows, g.Lk, kF64Threads);
    return;
  }

  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t sK = base + L::kK, sV = base + L::kV, sRing = base + L::kRing, sDs = base + L::kDs;
  const uint32_t bars = base + L::kBars;
  const uint32_t bar_kv_full = bars, bar_acc_full = bars + 8, bar_s_full = bars + 16, bar_dp_full = bars + 24,
                 bar_p_full = bars + 32, bar_ds_full = bars + 40, bar_dq_full = bars + 48, bar_dq_drained = bars + 56;
  const uint32_t bar_ring_full = bars + 64, bar_ring_empty = bar_ring_full + 8 * L::kStages;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen_base + L::kMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen_base + L::kMisc + 4);
  const Guard guard{p.status, abort_flag};

  // step `it` of this CTA: head and step of that head; the last one of its query tile issues / drains dQ
  auto step_head = [&](int it) { return hk * G + it / n_qs; };
  auto step_q = [&](int it) { return it % n_qs; };
  auto ends_tile = [&](int qs) { return (qs & 1) != 0 || qs == n_qs - 1; };
  auto load_step = [&](int it) {
    const int s = it % L::kStages, qrow = q_row0 + step_q(it) * kF64Step, h = step_head(it);
    const uint32_t dst = sRing + s * 2 * L::kStepBytes;
    mbar_arrive_expect_tx(bar_ring_full + 8 * s, 2 * L::kStepBytes);
    tma_load_4d(dst, &tmQ, bar_ring_full + 8 * s, 0, qrow, h, b);
    tma_load_4d(dst + L::kStepBytes, &tmdO, bar_ring_full + 8 * s, 0, qrow, h, b);
  };

  if (warp == 12) {
    // The producer thread initialises the barriers itself and puts K, V and the first two steps in flight before the
    // CTA-wide set-up (TMEM allocation, __syncthreads) completes.
    if (lane == 0) {
      *abort_flag = 0;
      mbar_init(bar_kv_full, 1);
      mbar_init(bar_acc_full, 1);
      mbar_init(bar_s_full, 1);
      mbar_init(bar_dp_full, 1);
      mbar_init(bar_p_full, 8);
      mbar_init(bar_ds_full, 8);
      mbar_init(bar_dq_full, 1);
      mbar_init(bar_dq_drained, 4);
      for (int s = 0; s < L::kStages; ++s) {
        mbar_init(bar_ring_full + 8 * s, 1);
        mbar_init(bar_ring_empty + 8 * s, 1);
      }
      fence_barrier_init();
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(bar_kv_full, 2 * L::kTileBytes);
      tma_load_4d(sK, &tmK, bar_kv_full, 0, kb, hk, b);
      tma_load_4d(sV, &tmV, bar_kv_full, 0, kb, hk, b);
      load_step(0);
      if (n_it > 1) load_step(1);
    }
    __syncwarp();
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), kF64TmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tSt = tmem, tdPt = tmem + 64, tdQ = tmem + 64, tdV = tmem + 128, tdK = tmem + 192;

  if (warp >= 12) {
    reg_dealloc<kF64OtherRegs>();
    if (warp == 12) {
      // ------------------------------------------------------------------- TMA producer
      if (lane == 0) {
        bool ok = true;
        for (int it = L::kStages; it < n_it; ++it) {  // the first round was issued during set-up
          ok = mbar_wait(bar_ring_empty + 8 * (it % L::kStages), ((uint32_t)(it / L::kStages) & 1u) ^ 1u, guard, kStF64Producer);
          if (!ok) break;
          load_step(it);
        }
        if (!ok) {
          const uint64_t t0 = globaltimer_ns();
          while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
        }
      }
    } else if (warp == 13) {
      // --------------------------------------------------------------------- MMA issuer
      if (lane == 0) {
        constexpr uint32_t idesc_s = make_idesc<T>(kTile, kF64Step, false, false);
        constexpr uint32_t idesc_acc = make_idesc<T>(kTile, D, false, true);  // A K-major (or TMEM), B MN-major
        constexpr uint32_t idesc_dq = make_idesc<T>(kTile, D, true, true);    // A and B MN-major
        constexpr uint32_t hi_k = desc_hi_sw128(1024);
        const uint32_t k_lo = desc_lo_sw128(sK, 16), v_lo = desc_lo_sw128(sV, 16);
        const uint32_t kmn_lo = desc_lo_sw128(sK, L::kTileBytes);
        const uint32_t dsmn_lo = desc_lo_sw128(sDs, L::kTileBytes);
        auto stage_q = [&](int it) { return sRing + (it % L::kStages) * 2 * L::kStepBytes; };
        auto issue_s = [&](int it) -> bool {  // S^T(it) = K Q^T; first user of ring stage `it`
          const int s = it % L::kStages;
          if (!mbar_wait(bar_ring_full + 8 * s, (uint32_t)(it / L::kStages) & 1u, guard, kStF64Mma)) return false;
          tc_fence_after();
          const uint32_t q_lo = desc_lo_sw128(stage_q(it), 16);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_ss_lh(tSt, k_lo + kk * 2, q_lo + kk * 2, hi_k, idesc_s, kk > 0);
          mma_commit(bar_s_full);
          return true;
        };
        auto issue_dp = [&](int it) {  // dP^T(it) = V dO^T
          const uint32_t do_lo = desc_lo_sw128(stage_q(it) + L::kStepBytes, 16);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_ss_lh(tdPt, v_lo + kk * 2, do_lo + kk * 2, hi_k, idesc_s, kk > 0);
          mma_commit(bar_dp_full);
        };
        bool ok = mbar_wait(bar_kv_full, 0, guard, kStF64Mma);
        if (ok) ok = issue_s(0);
        if (ok) issue_dp(0);
        int tile_no = 0;
        for (int it = 0; it < n_it && ok; ++it) {
          const uint32_t par = (uint32_t)it & 1u;
          const int qs = step_q(it);
          const uint32_t domn_lo = desc_lo_sw128(stage_q(it) + L::kStepBytes, L::kStepBytes);
          const uint32_t qmn_lo = desc_lo_sw128(stage_q(it), L::kStepBytes);
          const uint32_t dsk_lo = desc_lo_sw128(sDs + (qs & 1) * L::kTileBytes, 16);
          ok = mbar_wait(bar_p_full, par, guard, kStF64Mma);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < kF64Step / 16; ++kk)  // dV += P^T dO   (16 queries per instruction)
            mma_ts_lh(tdV, tSt + (kk / 2) * 32 + (kk % 2) * 8, domn_lo + kk * 128, hi_k, idesc_acc, (it > 0 || kk > 0));
          if (it + 1 < n_it) {
            ok = issue_s(it + 1);
            if (!ok) break;
          }
          ok = mbar_wait(bar_ds_full, par, guard, kStF64Mma);
          if (!ok) break;
          tc_fence_after();
          const bool tile_end = ends_tile(qs);
          if (tile_end) {
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk)  // dQ tile = dS K   (16 keys per instruction; overwrites dP^T(it))
              mma_ss_lh(tdQ, dsmn_lo + kk * 128, kmn_lo + kk * 128, hi_k, idesc_dq, kk > 0);
            mma_commit(bar_dq_full);
          }
#pragma unroll
          for (int kk = 0; kk < kF64Step / 16; ++kk)  // dK += dS^T Q
            mma_ss_lh(tdK, dsk_lo + kk * 2, qmn_lo + kk * 128, hi_k, idesc_acc, (it > 0 || kk > 0));
          mma_commit(bar_ring_empty + 8 * (it % L::kStages));
          if (it + 1 < n_it) {
            if (tile_end) {
              ok = mbar_wait(bar_dq_drained, (uint32_t)tile_no & 1u, guard, kStF64Mma);  // dQ is in registers
              if (!ok) break;
              tc_fence_after();
            }
            issue_dp(it + 1);
          }
          tile_no += tile_end;
        }
        if (ok) mma_commit(bar_acc_full);
      }
    }
  } else if (warp >= 8) {
    // --------------------------------------------------------------------- dQ drain warps
    reg_dealloc<kF64DrainRegs>();
    const int rg = warp & 3;  // query rows [32 rg, 32 rg + 32) of the tile == this warp's TMEM lanes
    const uint32_t lane_sel = (uint32_t)(rg * 32) << 16;
    uint8_t* stage_gen = gen_base + L::kDrain + rg * (L::kDrainBufs * L::kDrainChunkBytes);
    const uint32_t stage_sh = base + L::kDrain + rg * (L::kDrainBufs * L::kDrainChunkBytes);
    int chunk_no = 0, tile_no = 0;
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const int qs = step_q(it);
      if (!ends_tile(qs)) continue;
      // was the step that holds this warp's rows among the steps of this tile?
      const int row = q_row0 + (qs & ~1) * kF64Step + rg * 32;
      const bool have = (qs & ~1) + (rg >> 1) < n_qs;
      float* dst = p.dq_accum + ((size_t)b * g.H + step_head(it)) * n_qt_total * (size_t)(kTile * D) + (size_t)row * D;
      ok = mbar_wait(bar_dq_full, (uint32_t)tile_no & 1u, guard, kStF64Drain);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      ++tile_no;
      tc_fence_after();
      // The channels leave TMEM in two halves; the columns are handed back once the second one is in registers.
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t acc[32];
        if (have) {
          tmem_ld32(tdQ + lane_sel + half * 32, acc);
          tmem_wait_ld();
        }
        if (half == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_dq_drained);
        }
        if (!have) continue;
#pragma unroll
        for (int ch = 0; ch < 4; ++ch, ++chunk_no) {
          const int buf = chunk_no % L::kDrainBufs;
          if (lane == 0) bulk_wait_read<L::kDrainBufs - 1>();  // the reduction that last used this buffer has read it
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 2; ++j)
            *reinterpret_cast<uint4*>(stage_gen + buf * L::kDrainChunkBytes + (j * 32 + lane) * 16) =
                make_uint4(acc[8 * ch + 4 * j], acc[8 * ch + 4 * j + 1], acc[8 * ch + 4 * j + 2], acc[8 * ch + 4 * j + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            bulk_reduce_add_f32(dst + (half * 4 + ch) * (L::kDrainChunkBytes / 4), stage_sh + buf * L::kDrainChunkBytes,
                                L::kDrainChunkBytes);
            tma_store_commit();
          }
        }
      }
    }
    if (lane == 0) bulk_wait_read<0>();  // the staging buffers have been read; the sums land in global memory by kernel end
  } else {
    // ------------------------------------------------------------------- compute warps
    reg_alloc<kF64ComputeRegs>();
    const int wg = warp >> 2, c0 = wg * 32;         // query columns [c0, c0 + 32) of the step
    const int r = (warp & 3) * 32 + lane;           // key row inside the tile == TMEM lane
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const int kg = kg0 + r;
    const bool key_ok = kg < n && kb + r < g.Lk;
    const float c = g.scale * kLog2e;
    const uint64_t c2 = pk2(c, c);
    float* slot = reinterpret_cast<float*>(gen_base + L::kRows) + warp * 64;  // warp-private: -LSE[32], -delta[32]
    bool ok = true;
    // LSE / delta of this lane's query column, fetched one step ahead (step qs_next of head h_next) and not touched until
    // then; the walk over heads and steps is incremental (no divisions)
    int h_next = hk * G, qs_next = 0;
    float lse_next, delta_next;
    auto fetch_rows = [&]() {
      const int qrow = q_row0 + qs_next * kF64Step + c0 + lane;
      const int row = qrow < g.Lq ? qrow : 0;  // row 0 stands in for rows beyond Lq: those columns are masked out anyway
      lse_next = __ldg(p.lse + b * p.lse_sb + h_next * p.lse_sh + row * p.lse_sl);
      delta_next = __ldg(p.delta + ((long long)b * g.H + h_next) * g.Lq + row);
    };
    fetch_rows();
    for (int it = 0; it < n_it; ++it) {
      const uint32_t par = (uint32_t)it & 1u;
      const int qs = qs_next;
      const int q0 = q_row0 + qs * kF64Step, qg0 = q0 + g.q_off;
      if (++qs_next == n_qs) {
        qs_next = 0;
        ++h_next;
      }
      __syncwarp();
      slot[lane] = (lse_next == -CUDART_INF_F) ? 0.f : -lse_next;  // negated: addends of the packed FMA / ADD
      slot[32 + lane] = -delta_next;
      __syncwarp();
      if (it + 1 < n_it) fetch_rows();
      const bool full = M::kHasQFullRange && qg0 >= full_lo && qg0 + kF64Step <= full_hi && qg0 + kF64Step <= n &&
                        q0 + kF64Step <= g.Lq && kg0 + kTile <= n && kb + kTile <= g.Lk;
      const int qlim = imin(n - qg0, g.Lq - q0);
      int w_lo = 0, w_hi = -1;  // visible query columns of this key row inside the step (interval functors)
      if (interval_rows<M>::value && !full && key_ok) row_window<M, false>(kg, qg0, qlim, n, g.margs, w_lo, w_hi);

      // ---- P^T = 2^(S^T c - LSE), masked; 16-bit copy to TMEM for the dV GEMM, kept packed in registers
      ok = mbar_wait(bar_s_full, par, guard, kStF64Compute);
      ok = __all_sync(0xffffffffu, ok);  // keep the warp converged for the .sync.aligned TMEM accesses
      if (!ok) break;
      tc_fence_after();
      uint32_t preg[16];
      {
        uint32_t sreg[32];
        tmem_ld32(tSt + lane_sel + c0, sreg);
        tmem_wait_ld();
        auto body = [&](auto masked_tag) {  // two copies: full tiles run without any mask arithmetic
          constexpr bool kMasked = decltype(masked_tag)::value;
#pragma unroll
          for (int j = 0; j < 8; ++j) {  // four query columns per round
            const float4 nl4 = reinterpret_cast<const float4*>(slot)[j];
            float p0, p1, p2, p3;
            upk2(ex2_pair(ffma2(pk2u(sreg[4 * j], sreg[4 * j + 1]), c2, pk2(nl4.x, nl4.y)), false), p0, p1);
            upk2(ex2_pair(ffma2(pk2u(sreg[4 * j + 2], sreg[4 * j + 3]), c2, pk2(nl4.z, nl4.w)), false), p2, p3);
            if (kMasked) {
              const int cq = c0 + 4 * j;
              if (interval_rows<M>::value) {
                p0 = (cq >= w_lo && cq <= w_hi) ? p0 : 0.f;
                p1 = (cq + 1 >= w_lo && cq + 1 <= w_hi) ? p1 : 0.f;
                p2 = (cq + 2 >= w_lo && cq + 2 <= w_hi) ? p2 : 0.f;
                p3 = (cq + 3 >= w_lo && cq + 3 <= w_hi) ? p3 : 0.f;
              } else {
                p0 = (key_ok && cq < qlim && M::mask(qg0 + cq, kg, n, g.margs)) ? p0 : 0.f;
                p1 = (key_ok && cq + 1 < qlim && M::mask(qg0 + cq + 1, kg, n, g.margs)) ? p1 : 0.f;
                p2 = (key_ok && cq + 2 < qlim && M::mask(qg0 + cq + 2, kg, n, g.margs)) ? p2 : 0.f;
                p3 = (key_ok && cq + 3 < qlim && M::mask(qg0 + cq + 3, kg, n, g.margs)) ? p3 : 0.f;
              }
            }
            preg[2 * j] = pack2<T>(p0, p1);
            preg[2 * j + 1] = pack2<T>(p2, p3);
          }
        };
        if (full) body(std::false_type{});
        else body(std::true_type{});
      }
      tmem_st16(tSt + lane_sel + c0, preg);  // over the first half of the fp32 columns this warp just consumed
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_p_full);

      // ---- dS^T = P^T (dP^T - delta) with the rounded P^T the dV GEMM uses
      ok = mbar_wait(bar_dp_full, par, guard, kStF64Compute);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t dpreg[32];
        tmem_ld32(tdPt + lane_sel + c0, dpreg);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 nd4 = reinterpret_cast<const float4*>(slot + 32)[j];
          float p0, p1, p2, p3, d0, d1, d2, d3;
          unpack2<T>(preg[2 * j], p0, p1);
          unpack2<T>(preg[2 * j + 1], p2, p3);
          upk2(fmul2(pk2(p0, p1), fadd2(pk2u(dpreg[4 * j], dpreg[4 * j + 1]), pk2(nd4.x, nd4.y))), d0, d1);
          upk2(fmul2(pk2(p2, p3), fadd2(pk2u(dpreg[4 * j + 2], dpreg[4 * j + 3]), pk2(nd4.z, nd4.w))), d2, d3);
          preg[2 * j] = pack2<T>(d0, d1);
          preg[2 * j + 1] = pack2<T>(d2, d3);
        }
      }
      tc_fence_before();  // orders this warp's dP^T reads before the GEMMs that re-use the columns
      {
        // row r of the [key][query] chunk of this step is one 128-byte line, this warp's columns half of it
        uint8_t* line = gen_base + L::kDs + (qs & 1) * L::kTileBytes + r * 128;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          *reinterpret_cast<uint4*>(line + (((wg * 4 + u) ^ (r & 7)) * 16)) =
              make_uint4(preg[4 * u], preg[4 * u + 1], preg[4 * u + 2], preg[4 * u + 3]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ds_full);
    }

    // ---- epilogue: warps 0-3 store dV, warps 4-7 store dK * sm_scale (staging = the ring)
    if (ok) ok = mbar_wait(bar_acc_full, 0, guard, kStF64Epilogue);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    const uint32_t tacc = wg == 0 ? tdV : tdK;
    const float mul = wg == 0 ? 1.f : g.scale;
    float* part_row = p.part.row(wg == 0 ? p.part.dv : p.part.dk, b, hk, kb + r, g.Lk);
#pragma unroll
    for (int q4 = 0; q4 < 2; ++q4) {
      uint32_t acc[32];
      if (ok) {
        tmem_ld32(tacc + lane_sel + q4 * 32, acc);
        tmem_wait_ld();
      }
      stage_row32<T>(gen_base + L::kRing + wg * L::kTileBytes, r, q4, acc, mul, ok && key_ok);
      if (part_row != nullptr) store_part32(part_row + q4 * 32, acc, mul, ok && key_ok);
    }
    fence_proxy_async_smem();
    if (wg == 0) named_bar_sync(1, 128);
    else named_bar_sync(2, 128);
    if ((threadIdx.x & 127) == 0) {
      tma_store_4d(wg == 0 ? &tmdV : &tmdK, sRing + wg * L::kTileBytes, 0, kb, hk, b);
      tma_store_commit();
      tma_store_wait_read();  // shared memory may be released; the global writes complete by kernel end
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 12) tmem_dealloc(tmem, kF64TmemCols);
}

// ---------------------------------------------------------------------------- launcher
// The rule of the dispatch: few query tiles for a key tile in the middle of the sequence, counted over all heads of its
// group, and enough key tiles to give every SM its two CTAs.  Main kernel in us, bwd_fused.cuh against this one (fp16, head
// dim 64):
//   (2,32,8192) window(l, 0)  l = 16: 251 / 175   128: 251 / 202   256 (3 tiles): 300 / 264   512 (5): 394 / 370   768: 484 / 475
//   (2,32,8192) chunkwise(128, 2): 292 / 256      chunkwise(128, 3) (4 tiles): 340 / 309    (64,8,512) full: 173 / 159
//   long loops:   (4,16,4096) full: 845 / 964, causal: 476 / 571     (2,32,8192) window(128, 0), 4 heads per key head: 151 / 166
//   few CTAs:     (4,8,300) full, 96 CTAs: 11.7 / 13.5     uneven ones: (8,8,1024) causal (5 tiles): 57 / 66
// so the line lies at four tiles, below what the uniform masks alone would allow.
constexpr int kF64MaxTiles = 4;
template <class M>
bool bwd_short_loops(const Geo& g, int D) {
  const int n_kt = (g.Lk + kTile - 1) / kTile;
  if (D > 64 || (long long)n_kt * g.Hkv * g.B < 2 * sm_count()) return false;
  const int kg0 = (n_kt - 1) / 2 * kTile + g.k_off;
  int lo, hi;
  tile_range<M, false>(kg0, kTile, g.seq_len, g.margs, lo, hi);
  lo = imax(lo - g.q_off, 0);
  hi = imin(imin(hi, g.seq_len - 1) - g.q_off, g.Lq - 1);
  return hi >= lo && (long long)(hi / kTile - lo / kTile + 1) * (g.H / g.Hkv) <= kF64MaxTiles;
}

template <typename T, int D, class M>
int launch_bwd_fused_one(const CUtensorMap* maps, const BwdTcParams& p, cudaStream_t st) {
  const Geo& g = p.g;
  cudaError_t e = cudaMemsetAsync(p.dq_accum, 0, dq_accum_bytes(g.B, g.H, g.Lq, D), st);
  if (e != cudaSuccess) return (int)e;
  // maps: 0 Q, 1 K, 2 V, 3 dO, 4 dQ, 5 dK, 6 dV (boxes of 128 rows; Q and dO with short_loops: kF64Step rows)
  dim3 gk((unsigned)(((g.Lk + kTile - 1) / kTile) * g.Hkv * g.B), 1, 1);
  constexpr bool kHasShort = D == 64;
  if (kHasShort && p.short_loops) {
    auto kern = bwd_fused64_tc_kernel<T, M>;
    struct Tag {};
    e = ensure_dynamic_smem<Tag>(kern, Fused64Smem::kDynamic, /*prefer_max_carveout=*/true);
    if (e != cudaSuccess) return (int)e;
    kern<<<gk, kF64Threads, Fused64Smem::kDynamic, st>>>(maps[0], maps[1], maps[2], maps[3], maps[5], maps[6], p);
  } else {
    auto kern = bwd_fused_tc_kernel<T, D, M>;
    constexpr int smem = FusedSmem<D>::kDynamic;
    static_assert(smem <= 232448, "exceeds the 227 KB of shared memory a CTA can opt in to");
    struct Tag {};
    e = ensure_dynamic_smem<Tag>(kern, smem);
    if (e != cudaSuccess) return (int)e;
    kern<<<gk, kFusedThreads, smem, st>>>(maps[0], maps[1], maps[2], maps[3], maps[5], maps[6], p);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  dim3 gc((unsigned)((g.Lq + kTile - 1) / kTile), (unsigned)g.H, (unsigned)g.B);
  dq_convert_kernel<T, D><<<gc, 256, 0, st>>>(p.dq_accum, reinterpret_cast<T*>(p.dq), p.dq_sb, p.dq_sh, p.dq_sl, g.H,
                                               g.Lq, g.D, g.scale);
  return (int)cudaGetLastError();
}

template <class M>
int launch_bwd_fused_all(int dtype, int D, const CUtensorMap* maps, const BwdTcParams& p, cudaStream_t st) {
  if (dtype == 2) {
    if (D == 128) return launch_bwd_fused_one<__nv_bfloat16, 128, M>(maps, p, st);
    if (D == 64) return launch_bwd_fused_one<__nv_bfloat16, 64, M>(maps, p, st);
  } else if (dtype == 1) {
    if (D == 128) return launch_bwd_fused_one<__half, 128, M>(maps, p, st);
    if (D == 64) return launch_bwd_fused_one<__half, 64, M>(maps, p, st);
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace tc
}  // namespace chill
