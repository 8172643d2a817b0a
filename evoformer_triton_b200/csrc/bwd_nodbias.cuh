// The fused backward kernel for calls that want no d(pair_bias) (inference-like fine tuning, a frozen bias, no
// bias at all), and above a head dimension of 32 for all: the same items, steps and halves as evo_bwd_sm100_kernel.  What
// the missing gradient makes room for in shared memory changes how dQ leaves: a step's partial is one swizzled tile that
// the loader adds to global memory by one bulk reduction (two at DP = 64, a half each), where the other form's warps have
// staging areas and reductions of their own; and the bias has a third half tile where it fits.  Bound, as the other form,
// by the hand-overs and the chain of the compute warps; at DP = 64 also by the gap at an item boundary (a load of K, some
// 4 000 cycles).  Forward and backward of [4,1,2048,32,64] 1 024 us, 928 since K and V have a barrier each, dK and dV leave
// by bulk stores and P and dS are handed over before dS is stored.  With a d(pair_bias) of its own it would be the slower of
// the two at DP = 32: the bulk reductions of both leave one after another.
//
// A d(pair_bias) above a head dimension of 32 comes from bwd_dbias.cuh where there are many rows, else from here (DBIAS,
// see apart_pays): each dS is added to global memory from its register as it is formed, a warp's 32 keys side by side in
// one instruction, since no shared memory is left for staging.  (Staged and reduced in bulk, before this kernel took over
// at DP = 64: [1,4,768,8,64] 79 us, now 76; [4,1,2048,32,64] 1 989 and 1 973; [1,128,128,8,64] 98 and 86.)
#pragma once

#include "bwd_common.cuh"

namespace evo {
namespace {

template <int DP, int BIAS>
struct SmemN : TilesT<DP> {
  using Tiles = TilesT<DP>;
  using Tiles::G, Tiles::kTile, Tiles::kStage, Tiles::kDS;
  // The pair bias: half tiles [64 i][128 j], unswizzled; one more than is read at a time where it fits
  static constexpr int kHalfF32 = HT * BT * 4, kHalf = BIAS == BIAS_16 ? kHalfF32 / 2 : kHalfF32;
  static constexpr int kBufs = BIAS == BIAS_NONE ? 0 : DP == 64 && BIAS == BIAS_F32 ? 2 : 3;
  static constexpr int kOut = BT * DP * 4;                   // a step's dQ partial
  static constexpr int kMaskRows = DP == 64 || (DP == 32 && BIAS == BIAS_F32) ? 0 : G;  // (in registers where a kilobyte is missing, or one row's is waited for anyway)
  static constexpr int offKV = 0;                            // [g][K, V], resident for the whole item
  static constexpr int offStage = offKV + 2 * G * kTile;
  static constexpr int offDS = offStage + kStages * kStage;
  static constexpr int offBias = offDS + kDS;
  static constexpr int offOut = offBias + kBufs * kHalf;
  static constexpr int offMask = offOut + kOut;              // [kMaskRows][128 keys]: what the mask adds to a score
  static constexpr int offBars = offMask + kMaskRows * BT * 4;
  // 64 barrier slots (see the kernel) and the slack for aligning the tiles to 1024 bytes, as much of it as
  // fits: the kernel checks what the base address needs and gives up with a status code if it is more (the
  // dynamic shared memory of a kernel without static shared memory starts on a 1024-byte boundary on this
  // architecture, so it needs none).
  static constexpr int kSlack = offBars + 512 + 1024 <= 232448 ? 1024 : 0;
  static constexpr size_t bytes = offBars + 512 + kSlack;
  static_assert(offDS % 1024 == 0 && kStage % 1024 == 0 && offStage % 1024 == 0 && offOut % 1024 == 0, "swizzled tiles need 1024-byte alignment");
  static_assert(bytes <= 232448, "shared memory budget of one CTA");
};

template <class T, int DP, int BIAS, bool DBIAS>
__global__ void __launch_bounds__(kThreadsT, 1)
evo_bwd_nodbias_sm100_kernel(const Args a, const int n_items, const __grid_constant__ CUtensorMap tmQ,
                const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmDQ,
                const __grid_constant__ CUtensorMap tmNL, const __grid_constant__ CUtensorMap tmDL,
                const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV) {
  using L = SmemN<DP, BIAS>;
  constexpr int G = L::G;
  static_assert(!DBIAS || (G == 1 && BIAS != BIAS_NONE), "d(pair_bias) leaves from here with one row per item only");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (static_cast<int>(smem - smem_raw) > L::kSlack) {  // the same for every thread of every CTA
    if (threadIdx.x == 0 && a.status) atomicCAS(a.status, 0, DEV_TIMEOUT_SYNC);
    return;
  }
  uint8_t* sKV = smem + L::offKV;
  uint8_t* sStage = smem + L::offStage;
  uint8_t* sDS = smem + L::offDS;
  uint8_t* sBias = smem + L::offBias;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::offBars);
  const uint32_t bars_s = smem_u32(bars);
  const Bar kv_full{bars_s + 8 * 0};     // [G] K and V of row g of the current item landed
  const Bar kv_empty{bars_s + 8 * 7};    // [G] ... and every MMA that reads them has completed (G = 1: [0] K, [1] V)
  const Bar drained{bars_s + 8 * 44};    // (G = 1) dK and dV of the item before are in shared memory, over its last dS
  const Bar dkv_sent{bars_s + 8 * 45};   // (G = 1) ... have left it
  const Bar st_full{bars_s + 8 * 32};     // [2] Q, dO and the statistics vectors of a step landed
  const Bar st_empty{bars_s + 8 * 40};    // [2] ... the step's last dV/dK MMAs have completed
  const Bar sd_full{bars_s + 8 * 48};    // [2], two apart: S^T and dP^T of half h of a step are in TMEM, its statistics landed
  const Bar cdone{bars_s + 8 * 52};      // [2], two apart: the warps of that half have its P^T and dS^T in TMEM (for the dV/dK MMAs)
  const Bar sdone{bars_s + 8 * 23};      // [2] ... and dS in shared memory (for the dQ MMAs), with the dQ partial of the step before
  const Bar b_full{bars_s + 8 * 56};     // [kBufs] a half (64 queries) of a pair-bias tile landed
  const Bar b_done{bars_s + 8 * 60};     // [kBufs] ... has been read for the last time
  const Bar dq_full{bars_s + 8 * 36};    // [2] the dQ partial of a step is complete in TMEM, the dS tile read, and the place for it free (DP = 64: [2 halves][2], for what the half takes of it)
  const Bar mk_full{bars_s + 8 * 25};    // [G] the mask of row g of the current item is in shared memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 22);  // (bars 23, 24: sdone; 25..31: mk_full)
  const uint32_t abort_s = smem_u32(const_cast<int*>(abort_flag));

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform, and known to be)
  constexpr bool has_bias = BIAS != BIAS_NONE, kBias16 = BIAS == BIAS_16;
  constexpr int kBufs = has_bias ? L::kBufs : 1, kHalf = L::kHalf;
  constexpr int kBRow = kBias16 ? BT * 2 : BT * 4;  // bytes per row (one query, 128 keys) of the staged bias tile
  const Steps<G> steps(a, n_items);
  const int NT = steps.NT, my_items = steps.items, total_steps = steps.total;

  grid_dependency_wait();
  grid_launch_dependents();
  if (tid == 0) *abort_flag = (a.status && *reinterpret_cast<volatile int*>(a.status) != 0) ? 1 : 0;
  __syncthreads();
  if (*abort_flag) return;

  if (tid == 0) {
    for (int i = 0; i < (G == 1 ? 2 : G); ++i) { mbar_init(bars + 0 + i, 1); mbar_init(bars + 7 + i, G == 1 ? 1 : 3); }  // kv_full; kv_empty: three MMA warps read K/V
    for (int i = 0; i < G; ++i) mbar_init(bars + 25 + i, 1);  // mk_full
    if (G == 1) { mbar_init(bars + 44, kCW); mbar_init(bars + 45, 1); }  // drained, dkv_sent
    for (int i = 0; i < kStages; ++i) { mbar_init(bars + 32 + i, 1); mbar_init(bars + 40 + i, 2); }  // st_full, st_empty
    for (int i = 0; i < 2; ++i) {
      mbar_init(bars + 48 + 2 * i, 3); mbar_init(bars + 52 + 2 * i, kCW / 2);  // sd_full: two commits, one warp; cdone
      mbar_init(bars + 36 + i, 2);                                     // dq_full: the commit, and the loader
      if (DP == 64) mbar_init(bars + 38 + i, 2);
    }
    for (int i = 0; i < kBufs; ++i) { mbar_init(bars + 56 + i, 1); mbar_init(bars + 60 + i, kCW / 2); }  // b_full, b_done
    for (int i = 0; i < 2; ++i) mbar_init(bars + 23 + i, kCW / 2);  // sdone
    fence_mbar_init();
    prefetch_tmap(&tmQ); prefetch_tmap(&tmK); prefetch_tmap(&tmV); prefetch_tmap(&tmDO);
    prefetch_tmap(&tmNL); prefetch_tmap(&tmDL);
    prefetch_tmap(&tmDQ);
    if (has_bias) prefetch_tmap(&tmB);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, L::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp >= kCW) {
    setmaxnreg_dec<kServiceRegs>();
    if (warp <= kCW + 1) {
      // tensor-core issuers of S^T and dV (warp 16), dP^T and dK (warp 17)
      int item = 0;  // whose V is loaded next
      auto load_v = [&] {
        if (item >= my_items) return;
        const StepT d = steps.decode(item * (NT * G));
        mbar_wait(kv_empty + 1, (item & 1) ^ 1, abort_s, DEV_TIMEOUT_MMA);
        if (elect_one()) {
          mbar_expect_tx(kv_full + 1, L::kTile);
          tma_load_5d_s(smem_u32(sKV) + L::kTile, &tmV, (kv_full + 1).a, 0, d.j0, d.s, d.h, d.b);
        }
        __syncwarp();
        ++item;
      };
      if (G == 1 && warp == kCW + 1) load_v();
      issue_scores_and_outputs<T, DP>(warp == kCW, tmem, smem_u32(sKV), smem_u32(sStage), NT, total_steps,
                                      IssueBars{kv_full, kv_empty, st_full, st_empty, sd_full, cdone, drained}, abort_s, load_v);
    } else if (warp == kCW + 2) {
      // =============================== tensor-core issuer of dQ; pair-bias loads ===============================
      const uint32_t sKV_s = smem_u32(sKV), sDS_s = smem_u32(sDS);
      const uint32_t sBias_s = smem_u32(sBias);
      // The bias tile (i, j) is the same for the G rows of a group.  Its halves (64 queries) go round the
      // buffers: half q = 2 * tile + h is loaded into buffer q % kBufs when the warps that read half q - kBufs
      // there have done so for the last time.
      const uint32_t halves = has_bias ? 2u * my_items * NT : 0u;
      uint32_t lq = 0;             // half that is loaded next
      StepT lp = steps.decode(0);  // and its tile
      auto load_bias = [&] {
        const uint32_t buf = lq % kBufs;
        if (elect_one()) {
          mbar_expect_tx(b_full + (int)buf, kHalf);
          tma_load_4d_s(sBias_s + buf * kHalf, &tmB, (b_full + (int)buf).a, lp.j0, lp.it * BT + (int)(lq & 1) * HT, lp.h, lp.b);
        }
        __syncwarp();
        if (++lq % 2 == 0 && ++lp.it == NT && lq < halves) lp = steps.decode((int)(lq >> 1) * G);  // (divisions: here, not before a load)
      };
#pragma unroll 1
      while (lq < (uint32_t)kBufs && lq < halves) load_bias();
      int g = 0, it = 0;  // row of the group, query tile
      int item = 0;       // (G = 1) whose K is loaded next
      StepT kp = steps.decode(0);
      auto load_k = [&] {
        if (item >= my_items) return;
        mbar_wait(kv_empty + 0, (item & 1) ^ 1, abort_s, DEV_TIMEOUT_MMA);
        if (elect_one()) {
          mbar_expect_tx(kv_full + 0, L::kTile);
          tma_load_5d_s(sKV_s, &tmK, kv_full.a, 0, kp.j0, kp.s, kp.h, kp.b);
        }
        __syncwarp();
        if (++item < my_items) kp = steps.decode(item * (NT * G));
      };
      if (G == 1) load_k();
      int item_out = 0;  // (G = 1) whose dK and dV leave next
      StepT op = steps.decode(0);
      uint32_t q = 0;  // half tile that is read next for the last time
#pragma unroll 1
      for (int n = 0; n < total_steps; ++n) {
        if (has_bias && g == G - 1) {  // the group's last step: its halves are free well before its dS is stored
#pragma unroll 1
          for (int h = 0; h < 2; ++h, ++q) {
            if (lq < halves) {
              mbar_wait(b_done + (int)(q % kBufs), (q / kBufs) & 1, abort_s, DEV_TIMEOUT_SYNC);
              load_bias();
            }
          }
        }
        mbar_wait(sdone + 0, n & 1, abort_s, DEV_TIMEOUT_SYNC);
        mbar_wait(sdone + 1, n & 1, abort_s, DEV_TIMEOUT_SYNC);
        tc_fence_after();
        const uint32_t el = issue_dq<T, DP>(tmem + L::colDQ + (n & 1) * DP, sDS_s, sKV_s + 2 * g * L::kTile);
        mma_commit_if_s(el, (dq_full + (n & 1)).a);
        if (DP == 64) mma_commit_if_s(el, (dq_full + 2 + (n & 1)).a);
        if (it == NT - 1) {
          mma_commit_if_s(el, (kv_empty + g).a);  // (G = 1: S^T of these keys is long through)
          if (G == 1) {
            load_k();
            mbar_wait(drained, (item_out & 1), abort_s, DEV_TIMEOUT_SYNC);
            if (elect_one()) {
              tma_store_5d_s(&tmDK, sDS_s, 0, op.j0, op.s, op.h, op.b);
              tma_store_5d_s(&tmDV, sDS_s + L::kTile, 0, op.j0, op.s, op.h, op.b);
              tma_commit_group();
              tma_wait_group_read0();
              mbar_arrive(dkv_sent);
            }
            __syncwarp();
            if (++item_out < my_items) op = steps.decode(item_out * (NT * G));
          }
        }
        if (++g == G) { g = 0; if (++it == NT) it = 0; }
      }
      if (G == 1 && elect_one()) tma_wait_group0();
      __syncwarp();
    } else {
      // =============================== tile loader ===============================
      // K/V of row g stay for the whole item and are replaced when the item's last MMAs that read them
      // have completed; Q, dO and the two statistics vectors of a step ride a two-deep ring.
      const uint32_t sKV_s = smem_u32(sKV), sStage_s = smem_u32(sStage), sMask_s = smem_u32(smem + L::offMask);
      // A step's dQ partial leaves from here too: it is in shared memory when the next step's dS is.  When the
      // reduction has read the place, the next one may be stored there, for which the compute warps wait on
      // dq_full (so sdone of a step cannot come before this warp has seen that of the step before).
      const uint32_t sOut_s = smem_u32(smem + L::offOut);
      // At DP = 64 it is two tiles of 32 columns, one from each half, that leave one after the other.
      constexpr int kBoxes = DP == 64 ? 2 : 1;
      auto send_dq = [&](int box, int row0, int slab) {
        if (elect_one()) {
          if (slab >= 0 && 32 * box < a.D) tma_reduce_add_3d_s(&tmDQ, sOut_s + box * (BT * 128), 32 * box, row0, slab);
          tma_commit_group();
        }
        __syncwarp();
      };
      auto dq_place_free = [&](int m) {  // for the partial of step m
        if (elect_one()) {
          if constexpr (kBoxes == 2) tma_wait_group_read1();
          else tma_wait_group_read0();
          mbar_arrive(dq_full + (m & 1));
          if constexpr (kBoxes == 2) {
            tma_wait_group_read0();
            mbar_arrive(dq_full + 2 + (m & 1));
          }
        }
        __syncwarp();
      };
      StepT d = steps.decode(0);
      auto load_kv = [&](int n) {
        const int k = n / (NT * G);
        float mk[4];
        if constexpr (L::kMaskRows > 0) {  // four keys of the row's mask a lane, loaded before the wait
#pragma unroll
          for (int u = 0; u < 4; ++u) mk[u] = mask_term<T>(a, d.b, d.s, d.j0 + lane + 32 * u);
        }
        mbar_wait(kv_empty + d.g, (k & 1) ^ 1, abort_s, DEV_TIMEOUT_MMA);
        if constexpr (L::kMaskRows > 0) {
          // (the last dQ MMA of the row is behind kv_empty, so its last step has read the mask before)
#pragma unroll
          for (int u = 0; u < 4; ++u) sts_f32(sMask_s + (d.g * BT + lane + 32 * u) * 4, mk[u]);
          __syncwarp();
          if (lane == 0) mbar_arrive(mk_full + d.g);
        }
        if (elect_one()) {
          const uint32_t dst = sKV_s + (2 * d.g) * L::kTile;
          mbar_expect_tx(kv_full + d.g, 2 * L::kTile);
          tma_load_5d_s(dst, &tmK, (kv_full + d.g).a, 0, d.j0, d.s, d.h, d.b);
          tma_load_5d_s(dst + L::kTile, &tmV, (kv_full + d.g).a, 0, d.j0, d.s, d.h, d.b);
        }
        __syncwarp();
      };
      int row1 = 0, slab1 = -1, row2 = 0, slab2 = -1, row3 = 0, slab3 = -1;  // of one, two and three steps ago
#pragma unroll 1
      for (int n = 0; n < total_steps + 2; ++n) {
        const int stg = n % kStages;
        const bool load = n < total_steps;
        if (G > 1 && load && d.it == 0) load_kv(n);
        mbar_wait(st_empty + stg, ((n / kStages) & 1) ^ 1, abort_s, DEV_TIMEOUT_MMA);  // (of step n - 2)
        if (load) {
          if (elect_one()) {
            const uint32_t dst = sStage_s + stg * L::kStage;
            const uint32_t bar = (st_full + stg).a;
            mbar_expect_tx(st_full + stg, L::kStage);
            tma_load_5d_s(dst, &tmQ, bar, 0, d.it * BT, d.s, d.h, d.b);
            tma_load_5d_s(dst + L::kTile, &tmDO, bar, 0, d.it * BT, d.s, d.h, d.b);
            tma_load_3d_s(dst + 2 * L::kTile, &tmNL, bar, d.it * BT, d.s, d.b * a.H + d.h);
            tma_load_3d_s(dst + 2 * L::kTile + L::kVec, &tmDL, bar, d.it * BT, d.s, d.b * a.H + d.h);
          }
          __syncwarp();
        }
        if (n >= 2) {
          mbar_wait(sdone + 0, n & 1, abort_s, DEV_TIMEOUT_SYNC);
          if (kBoxes == 2 && n >= 3) send_dq(0, row3, slab3);
          mbar_wait(sdone + 1, n & 1, abort_s, DEV_TIMEOUT_SYNC);
          if (n >= 3) send_dq(kBoxes - 1, row3, slab3);
          dq_place_free(n - 2);
        }
        row3 = row2; slab3 = slab2;
        row2 = row1; slab2 = slab1;
        row1 = d.it * BT;
        slab1 = d.s < a.S ? (d.b * a.H + d.h) * a.S + d.s : -1;
        if (load) d = steps.advance(d, n + 1);
      }
      if (total_steps > 0) {  // the last step's partial: the compute warps arrive once more
        mbar_wait(sdone + 0, total_steps & 1, abort_s, DEV_TIMEOUT_SYNC);
        mbar_wait(sdone + 1, total_steps & 1, abort_s, DEV_TIMEOUT_SYNC);
        for (int box = 0; box < kBoxes; ++box) send_dq(box, row3, slab3);
        if (elect_one()) tma_wait_group0();
        __syncwarp();
      }
    }
  } else {
    // =============================== compute warps ===============================
    // Warps 0-7 work on half 0 (queries 0..63 of the tile) of every step, warps 8-15 on half 1: two
    // groups that run half a step apart, so that while one waits (for its S^T/dP^T, for tensor
    // memory, for its MMAs) the other has arithmetic to issue.  Warp w: keys 32*(w%4).. (its TMEM
    // lanes), queries 32*((w/4)%2).. of its half, in two chunks of 16.
    setmaxnreg_inc<kComputeRegs>();
    const int q4 = warp & 3, cb2 = (warp >> 2) & 1, H = warp >> 3;
    const int jrow = q4 * 32 + lane;
    const uint32_t t_lane = tmem + (static_cast<uint32_t>(q4 * 32) << 16);
    const uint32_t cS = t_lane + (H ? L::colS1 : L::colS0) + QT * cb2, cP = t_lane + (H ? L::colDP1 : L::colDP0) + QT * cb2;
    const float inv_r = 1.f / (float)a.R;
    const float c1 = a.scale * kLog2e;
    // 32-bit shared-window addresses: every access below stays a shared-memory instruction
    const uint32_t sStage_s = smem_u32(sStage), sDS_s = smem_u32(sDS);
    const uint32_t sBias_s = smem_u32(sBias);
    const uint32_t drow = sDS_s + H * (L::kDS / 2) + jrow * 128;

    // The dQ partial of step m (TMEM lanes = queries): a warp takes DP/4 columns of its 32 query rows.
    constexpr int QC = DP / 4;
    const int colblk = 2 * H + cb2;  // which of the four column blocks this warp takes
    // ... into the swizzled tile (two of 32 columns at DP = 64) that leaves as a whole
    auto store_dq = [&](int m) {
      uint32_t qr[QC];
      tmem_ld<QC>(t_lane + L::colDQ + (m & 1) * DP + colblk * QC, qr);
      tmem_wait_ld();
      const uint32_t out = smem_u32(smem + L::offOut);
#pragma unroll
      for (int c = 0; c < QC / 4; ++c) {
        const int c16 = colblk * (QC / 4) + c;  // 16-byte piece of the row
        const uint32_t at = DP == 16 ? jrow * 64 + ((c16 ^ ((jrow >> 1) & 3)) << 4)
                                     : (c16 >> 3) * (BT * 128) + jrow * 128 + (((c16 & 7) ^ (jrow & 7)) << 4);
        sts_v4(out + at, qr[4 * c], qr[4 * c + 1], qr[4 * c + 2], qr[4 * c + 3]);
      }
    };
    int pb = 0, ph = 0, ps0 = 0, pj0 = 0;  // the item whose dK/dV still sit in TMEM
    const uint32_t mask_s = smem_u32(smem + L::offMask) + jrow * 4;
    float mreg[L::kMaskRows == 0 ? G : 1];
    const F2 c12 = f2_make(c1, c1);
    int n = 0;            // running step
    uint32_t tile = 0;    // running (item, query tile)
    uint32_t bias_s = 0;  // the half bias tile that this warp reads
    Bar bdone{0};
#pragma unroll 1
    for (int k = 0; k < my_items; ++k) {
    const StepT cur = steps.decode(n);
    if constexpr (L::kMaskRows == 0) {
#pragma unroll
      for (int r = 0; r < G; ++r) mreg[r] = mask_term<T>(a, cur.b, cur.s + r, cur.j0 + jrow);
    }
#pragma unroll 1
    for (int it = 0; it < NT; ++it, ++tile)
#pragma unroll 1
    for (int g = 0; g < G; ++g, ++n) {
      const uint32_t vec_s = sStage_s + (n & 1) * L::kStage + 2 * L::kTile;
      const bool last_of_group = (g == G - 1);
      float mj;
      if constexpr (L::kMaskRows == 0) {
        mj = mreg[0];  // (the rows take turns)
#pragma unroll
        for (int r = 0; r + 1 < G; ++r) mreg[r] = mreg[r + 1];
        mreg[G - 1] = mj;
      } else {
        if (it == 0) mbar_wait(mk_full + g, k & 1, abort_s, DEV_TIMEOUT_TMA);
        mj = lds_f32(mask_s + g * (BT * 4));
      }
      if (G == 1 && it == 0 && k > 0) {  // dK and dV of the item before, while this one's K is on its way
        mbar_wait(st_empty + ((n - 1) & 1), ((n - 1) >> 1) & 1, abort_s, DEV_TIMEOUT_MMA);
        mbar_wait(kv_empty + 0, (k - 1) & 1, abort_s, DEV_TIMEOUT_MMA);  // (dQ of the item's last step: its dS has been read)
        tc_fence_after();
        stage_dk_or_dv<T>(t_lane + (H ? L::colDV : L::colDK) + 32 * cb2, sDS_s + H * L::kTile, H ? 1.f : a.scale, jrow, cb2);
        fence_async_shared();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(drained);
      }
      if (has_bias && g == 0) {
        const uint32_t q = 2 * tile + H;
        bias_s = sBias_s + (q % kBufs) * kHalf;
        bdone = b_done + (int)(q % kBufs);
        mbar_wait(b_full + (int)(q % kBufs), (q / kBufs) & 1, abort_s, DEV_TIMEOUT_TMA);
      }
      const uint32_t brow0 = bias_s + QT * cb2 * kBRow + jrow * (kBias16 ? 2 : 4);
      mbar_wait(sd_full + 2 * H, n & 1, abort_s, DEV_TIMEOUT_MMA);  // S^T and dP^T, statistics
      tc_fence_after();
      // a row whose keys are all dropped has this nl for every query (the mask row is shared by all queries of the
      // MSA row): what its scores gave is replaced
      const bool dead = __any_sync(0xffffffffu, lds_f32(vec_s) == kDeadRow);
      const F2 mj2 = f2_make(mj, mj);
      // (DBIAS) d(pair_bias) of this thread's key and its warp's first query; queries left from there, none in a dead row
      float* db = nullptr;
      int db_left = 0;
      if constexpr (DBIAS) {
        const int i = it * BT + H * HT + QT * cb2, j = cur.j0 + jrow;
        db = a.dbias + (((long long)cur.b * a.H + cur.h) * a.R + i) * a.dbias_ld + j;
        db_left = j < a.R && !dead ? a.R - i : 0;
      }
      uint32_t dk[16];
#pragma unroll
      for (int sub = 0; sub < 2; ++sub) {
        // this warp's queries of the half: 32*cb2 + 16*sub .. +16
        uint32_t sr[16], dr[16];
        tmem_ld16(cS + 16 * sub, sr);
        tmem_ld16(cP + 16 * sub, dr);
        const uint32_t vnl = vec_s + (H * HT + QT * cb2 + 16 * sub) * 4, vdl = vnl + BT * 4;
        const uint32_t brow = brow0 + (16 * sub) * kBRow;
        tmem_wait_ld();
        uint32_t pk[8];
        score_chunk<T, has_bias>(sr, dr, vnl, vdl, [&](int e) { return staged_bias<T, kBias16>(brow + e * kBRow); }, c12, mj2, pk,
                                 dk + 8 * sub, [&](int e, F2 ds) {
                                   if constexpr (DBIAS) {  // (32 neighbouring keys an instruction)
                                     const int q = 16 * sub + 2 * e;
                                     float d0, d1;
                                     f2_get(ds, d0, d1);
                                     red_add_if(db + (long long)q * a.dbias_ld, d0, q < db_left);
                                     red_add_if(db + (long long)(q + 1) * a.dbias_ld, d1, q + 1 < db_left);
                                   }
                                 });
        if (dead) {
          const float pu = (cur.j0 + jrow < a.R) ? inv_r : 0.f;
          const uint32_t w = Pack2<T>::pack(pu, pu);
#pragma unroll
          for (int e = 0; e < 8; ++e) { pk[e] = w; dk[8 * sub + e] = 0u; }
        }
        // P^T and dS^T, two 16-bit values per column, over the columns this thread has just read:
        // the A operands of the dV and dK MMAs (16 queries = 8 packed columns each)
        tmem_st8(cS + 16 * sub, pk);
        tmem_st8(cP + 16 * sub, *reinterpret_cast<uint32_t(*)[8]>(&dk[sub * 8]));
      }
      if (has_bias && last_of_group) {  // (every value read has been worked on, so the loads are through)
        __syncwarp();
        if (lane == 0) mbar_arrive(bdone);
      }
      if (G > 1 && H == 0 && it == 0 && k > 0)  // before this step's dV / dK MMAs overwrite them
        // (All of the other half's MMAs into them were issued before the S^T and dP^T of this step.)
        drain_dkdv<T, DP>(a, t_lane, cb2, jrow, pb, ph, ps0 + g, pj0, g);
      // P^T and dS^T are in tensor memory: the dV / dK MMAs and the next S^T and dP^T may go, under what follows
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(cdone + 2 * H);
      // dQ of the previous step is complete, and the place it leaves from is free
      if (n > 0) mbar_wait(dq_full + (DP == 64 ? 2 * H : 0) + ((n - 1) & 1), ((n - 1) >> 1) & 1, abort_s, DEV_TIMEOUT_MMA);
      tc_fence_after();
      if (G == 1 && it == 0 && k > 0) mbar_wait(dkv_sent, (k - 1) & 1, abort_s, DEV_TIMEOUT_SYNC);
      if (n > 0) store_dq(n - 1);
      // dS^T -> shared memory, [key][query] rows of 128 bytes per half, 128-byte swizzle
#pragma unroll
      for (int c = 0; c < 4; ++c)  // dk[4 * c ..]: queries 32 * cb2 + 8 * c .. of this half
        sts_v4(drow + (((4 * cb2 + c) ^ (jrow & 7)) << 4), dk[4 * c], dk[4 * c + 1], dk[4 * c + 2], dk[4 * c + 3]);
      fence_async_shared();
      tc_fence_before();  // (the next MMAs into the dQ columns just read follow from this arrival)
      __syncwarp();
      if (lane == 0) mbar_arrive(sdone + H);
    }
    pb = cur.b; ph = cur.h; ps0 = cur.s; pj0 = cur.j0;
    }

    if (total_steps > 0) {
      mbar_wait(dq_full + (DP == 64 ? 2 * H : 0) + ((total_steps - 1) & 1), ((total_steps - 1) >> 1) & 1, abort_s, DEV_TIMEOUT_MMA);
      tc_fence_after();
      store_dq(total_steps - 1);
      fence_async_shared();
      __syncwarp();
      if (lane == 0) mbar_arrive(sdone + H);
      if (H == 0 || G == 1) {
        // every dV / dK MMA of this CTA has completed once the last step's tile stage has been released
        const int last = total_steps - 1;
        mbar_wait(st_empty + (last & 1), (last >> 1) & 1, abort_s, DEV_TIMEOUT_MMA);
        tc_fence_after();
        if constexpr (G == 1) {
          mbar_wait(kv_empty + 0, (my_items - 1) & 1, abort_s, DEV_TIMEOUT_MMA);
          tc_fence_after();
          stage_dk_or_dv<T>(t_lane + (H ? L::colDV : L::colDK) + 32 * cb2, sDS_s + H * L::kTile, H ? 1.f : a.scale, jrow, cb2);
          fence_async_shared();
          __syncwarp();
          if (lane == 0) mbar_arrive(drained);
        } else {
          for (int g = 0; g < G; ++g) drain_dkdv<T, DP>(a, t_lane, cb2, jrow, pb, ph, ps0 + g, pj0, g);
        }
      }
    }
  }

  end_of_cta(abort_flag, a.status);
  if (warp == 0) tmem_dealloc(tmem, L::kTmemCols);
}

}  // namespace
}  // namespace evo
