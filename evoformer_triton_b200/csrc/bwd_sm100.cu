// Evoformer attention backward for sm_100a: the fused dQ/dK/dV/d(pair_bias) kernel with TRANSPOSED
// score tiles, for head dimensions up to 32 (padded to 16 or 32); above, and without a d(pair_bias), see
// bwd_nodbias.cuh and bwd_dbias.cuh, which are launched from here too.
//
// Replaces dsevoformer-triton/evoformer.py:299-326 (_attn_bwd_preprocess), :479-630
// (_attn_bwd_dk_dv) and :329-476 (_attn_bwd_dq).  The reference recomputes S and dP in two kernels
// and adds every dS element to d_pair_bias with an fp32 atomic (:458); here they are computed once.
// Like the reference's _attn_bwd_dk_dv (evoformer.py:594,607) the scores are computed as
// S^T = K_j Q_i^T and dP^T = V_j dO_i^T, so a thread owns one KEY j (its TMEM lane) and a run of
// queries i.  What that buys on this machine:
//   * P^T and dS^T (rounded to the storage type, evoformer.py:603,611) are written back into
//     tensor memory over the scores they came from and feed dV_j += P^T dO_i and dK_j += dS^T Q_i
//     as the A operand: P never touches shared memory, dS is stored once (for dQ_i = dS K_j).
//   * The residue mask of a key is one register per thread; the row statistics of the queries
//     (-lse*log2e and delta) are two 128-float vectors that arrive with the Q/dO tiles.
//   * The shared memory this frees holds the K/V tiles of a work item for its whole life and the
//     pair-bias tile of a whole row group.
//
// Work item = one 128-key tile j of G consecutive MSA rows of one (b,h): G = 7 at a padded head
// dimension of 16 and 3 at 32 (the dK/dV accumulators of a row take 2*DP of the 512 TMEM columns).
// A persistent CTA walks its items as a flat list of steps (query tile i, row g); a step is two
// halves of 64 queries, each with its own TMEM score buffer and its own eight warps: while one half
// computes, the tensor core finishes the other half's dV/dK MMAs and its next S^T/dP^T.
// dS is summed over the G rows in registers and leaves once per (i, j) tile as bulk tensor
// reductions, half a tile a warp and step; the dQ partial of a step goes to an fp32 accumulator in
// global memory the same way, by the eight warps of half 1, while those of half 0 take dK and dV.
//
// Warps: 0-15 compute (warp w: keys 32*(w%4).., queries 32*((w/4)%2).. of half w/8), 16-18 issue the
// tcgen05.mma (18 also loads the pair-bias tiles), 19 loads the other tiles.
#include "bwd_common.cuh"
#include "bwd_dbias.cuh"
#include "bwd_nodbias.cuh"
#include "common.cuh"
#include "launch.h"
#include "ptx.cuh"
#include "tmap.h"

namespace evo {
namespace {

template <int DP>
struct SmemT : TilesT<DP> {
  static_assert(DP < 64, "above 32 columns bwd_nodbias.cuh serves calls with a d(pair_bias) too");
  using Tiles = TilesT<DP>;
  using Tiles::G, Tiles::kTile, Tiles::kStage, Tiles::kDS;
  static constexpr int kBias = BT * BT * 4;                  // pair-bias tile [128 i][128 j], unswizzled (fp32; half of it for a 16-bit bias)
  // Staging areas, each with a place of its own so that a warp hardly waits for a reduction to have read it:
  // d(pair_bias) of every compute warp (16 queries x 32 keys at a time), and the dQ partial (32 queries, QC columns)
  // of the warps of half 1.
  static constexpr int kOutB = 16 * 32 * 4;
  static constexpr int QC = DP / 2;
  static constexpr int kOutQ = 32 * QC * 4;
  static constexpr int kMaskRows = DP == 32 ? 0 : G;         // (in registers where a kilobyte is missing)
  static constexpr int offKV = 0;                            // [g][K, V], resident for the whole item
  static constexpr int offStage = offKV + 2 * G * kTile;
  static constexpr int offDS = offStage + kStages * kStage;
  static constexpr int offBias = offDS + kDS;
  static constexpr int offOutB = offBias + kBias;
  static constexpr int offOutQ = offOutB + kCW * kOutB;
  static constexpr int offMask = offOutQ + kCW / 2 * kOutQ;      // [kMaskRows][128 keys]: what the mask adds to a score
  static constexpr int offBars = offMask + kMaskRows * BT * 4;
  // 64 barrier slots (see the kernel) and the slack for aligning the tiles to 1024 bytes, where it fits: the
  // kernel checks what the base address needs and gives up with a status code if that is more (the dynamic
  // shared memory of a kernel without static shared memory starts on a 1024-byte boundary on this
  // architecture, so it needs none).
  static constexpr int kSlack = offBars + 512 + 1024 <= 232448 ? 1024 : 0;
  static constexpr size_t bytes = offBars + 512 + kSlack;
  static_assert(offDS % 1024 == 0 && kStage % 1024 == 0 && offStage % 1024 == 0, "swizzled tiles need 1024-byte alignment");
  static_assert(bytes <= 232448, "shared memory budget of one CTA");
};

// The first pass of a backward call: delta[b,h,s,i] = -<dO_i, O_i> (evoformer.py:299-326; negated, so that it is
// added), nl = -lse*log2e,
// and zeros in the buffers that the fused kernel adds to (the fp32 dQ accumulator, d(pair_bias)).
// A row whose keys were all dropped carries lse = -FLT_MAX from the forward; its nl is kDeadRow, which
// the fused kernels recognise.  With a gate (Og = sigmoid(gate) O is the output, G its gradient):
//   dO    = G * sigmoid(gate)                      (what the attention backward needs; into scratch)
//   delta = sum_d dO * O = sum_d G * Og            (so the un-gated O is never needed)
//   dgate = G * O * sigmoid'(gate) = G * Og * (1 - sigmoid(gate))
// Bound by memory.  1 << LG lanes share a row, 16 bytes of each tensor per lane, so every access of a
// warp is a run of whole sectors whatever D is: [1,128,384,8,32] bf16 16 us (106 MB, 6.6 TB/s; 18 us with one
// thread per row and a memset), gated [1,384,384,4,32] 54 us (273 + 26 us in two passes before).
template <class T, int LG, bool GATE>
__global__ void __launch_bounds__(256) prep_kernel(const Args a, float* __restrict__ nl, float* __restrict__ dq_acc,
                                                   const size_t dbias_f4) {
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t gid = blockIdx.x * 256 + threadIdx.x;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  // (64-bit count and position: 2^32 of these pieces are 64 GiB, which fits the device)
  for (size_t e = gid; e < dbias_f4; e += (size_t)gridDim.x * 256) reinterpret_cast<float4*>(a.dbias)[e] = zero;
  const uint32_t row = gid >> LG, c = gid & ((1u << LG) - 1u);
  const uint32_t slab = row / (uint32_t)a.R, i = row - slab * (uint32_t)a.R;
  const uint32_t bh = slab / (uint32_t)a.S, s = slab - bh * (uint32_t)a.S;
  const uint32_t b = bh / (uint32_t)a.H, h = bh - b * (uint32_t)a.H;
  const bool ok = (int)b < a.B;
  float acc = 0.f;
  if (ok && (int)c * 8 < a.D) {
    const int d = (int)c * 8;
    const uint4 ov = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.o) + off4(a.so, b, h, s, i) + d);
    const uint4 gv = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.d_o) + off4(a.sdo, b, h, s, i) + d);
    const T* op = reinterpret_cast<const T*>(&ov);
    const T* gp = reinterpret_cast<const T*>(&gv);
    const size_t at = (size_t)row * a.D + d;
    if constexpr (GATE) {
      const uint4 tv = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.gate) + off4(a.sgate, b, h, s, i) + d);
      const T* tp = reinterpret_cast<const T*>(&tv);
      uint32_t eff[4], dg[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float x[2], y[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const float G = to_float<T>(gp[2 * u + w]), go = G * to_float<T>(op[2 * u + w]);
          const float sg = sigmoid16(to_float<T>(tp[2 * u + w]));
          acc += go;
          x[w] = G * sg;
          y[w] = go * (1.f - sg);
        }
        eff[u] = Pack2<T>::pack(x[0], x[1]);
        dg[u] = Pack2<T>::pack(y[0], y[1]);
      }
      *reinterpret_cast<uint4*>(reinterpret_cast<T*>(a.d_o_eff) + at) = make_uint4(eff[0], eff[1], eff[2], eff[3]);
      *reinterpret_cast<uint4*>(reinterpret_cast<T*>(a.dgate) + off4(a.sdgate, b, h, s, i) + d) = make_uint4(dg[0], dg[1], dg[2], dg[3]);
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u) acc += to_float<T>(op[u]) * to_float<T>(gp[u]);
    }
    reinterpret_cast<float4*>(dq_acc + at)[0] = zero;
    reinterpret_cast<float4*>(dq_acc + at)[1] = zero;
  }
#pragma unroll
  for (int o = (1 << LG) >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (ok && c == 0) {
    const size_t at = (size_t)slab * a.delta_ld + i;
    const float lse = a.lse[row];
    const bool dead = lse == -FLT_MAX;
    a.delta[at] = dead ? 0.f : -acc;  // (its dO and O may hold anything)
    nl[at] = dead ? kDeadRow : -lse * kLog2e;
  }
}

template <class T, bool GATE>
void launch_prep(const Args& a, float* nl, float* dq_acc, cudaStream_t st) {
  const int chunks = a.D / 8;
  const int lg = chunks > 4 ? 3 : chunks > 2 ? 2 : chunks > 1 ? 1 : 0;
  const size_t threads = ((size_t)a.B * a.H * a.S * a.R) << lg;
  const size_t f4 = a.dbias ? (size_t)a.B * a.H * a.R * a.dbias_ld / 4 : 0;
  const unsigned grid = (unsigned)((threads + 255) / 256);
  switch (lg) {
    case 3: launch_dependent(prep_kernel<T, 3, GATE>, grid, 256, 0, st, a, nl, dq_acc, f4); break;
    case 2: launch_dependent(prep_kernel<T, 2, GATE>, grid, 256, 0, st, a, nl, dq_acc, f4); break;
    case 1: launch_dependent(prep_kernel<T, 1, GATE>, grid, 256, 0, st, a, nl, dq_acc, f4); break;
    default: launch_dependent(prep_kernel<T, 0, GATE>, grid, 256, 0, st, a, nl, dq_acc, f4); break;
  }
}

// dq = scale * dq_acc, cast to the storage type (dq_acc: contiguous fp32 [B,H,S,R,D]).  Bound by memory; the position is
// found in 32 bits where that is enough (Index): 64-bit divisions were 400 instructions a warp (forward and backward of
// [1,203,203,4,32] 112.6 us, now 111.0).
template <class T, class Index>
__global__ void __launch_bounds__(256) dq_store_kernel(Args a, const float* __restrict__ acc) {
  grid_dependency_wait();
  grid_launch_dependents();
  const Index d8n = a.D / 8, total = (Index)a.B * a.H * a.S * a.R * d8n;
  const Index idx = (Index)blockIdx.x * 256 + threadIdx.x;
  if (idx >= total) return;
  const float4* src = reinterpret_cast<const float4*>(acc) + 2 * (size_t)idx;
  const float4 x = src[0], y = src[1];
  const Index row = idx / d8n, slab = row / (Index)a.R, bh = slab / (Index)a.S, b = bh / (Index)a.H;
  const int d = (int)(idx - row * d8n) * 8, i = (int)(row - slab * a.R), s = (int)(slab - bh * a.S), h = (int)(bh - b * a.H);
  uint4 pk;
  pk.x = Pack2<T>::pack(x.x * a.scale, x.y * a.scale);
  pk.y = Pack2<T>::pack(x.z * a.scale, x.w * a.scale);
  pk.z = Pack2<T>::pack(y.x * a.scale, y.y * a.scale);
  pk.w = Pack2<T>::pack(y.z * a.scale, y.w * a.scale);
  *reinterpret_cast<uint4*>(reinterpret_cast<T*>(a.dq) + off4(a.sdq, (int)b, h, s, i) + d) = pk;
}

template <class T, int DP, bool kBias16>
__global__ void __launch_bounds__(kThreadsT, 1)
evo_bwd_sm100_kernel(const Args a, const int n_items, const __grid_constant__ CUtensorMap tmQ,
                const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmDB, const __grid_constant__ CUtensorMap tmDQ,
                const __grid_constant__ CUtensorMap tmNL, const __grid_constant__ CUtensorMap tmDL,
                const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV) {
  using L = SmemT<DP>;
  constexpr int G = L::G;

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
  const Bar kv_empty{bars_s + 8 * 7};    // [G] ... and every MMA that reads them has completed
  const Bar st_full{bars_s + 8 * 32};     // [2] Q, dO and the statistics vectors of a step landed
  const Bar st_empty{bars_s + 8 * 40};    // [2] ... the step's last dV/dK MMAs have completed
  const Bar sd_full{bars_s + 8 * 48};    // [2], two apart: S^T and dP^T of half h of a step are in TMEM, its statistics landed
  const Bar cdone{bars_s + 8 * 52};      // [2], two apart: the warps of that half have its P^T and dS^T in TMEM (for the dV/dK MMAs)
  const Bar sdone{bars_s + 8 * 23};      // [2] ... and have stored their half of dS in shared memory (for the dQ MMAs) and read dQ of the step before
  const Bar b_full{bars_s + 8 * 14};     // [2] half h (64 queries) of the pair-bias tile landed
  const Bar b_done{bars_s + 8 * 16};     // [2] ... has been read for the last time
  const Bar dq_full{bars_s + 8 * 19};    // the dQ partial of the step before is complete in TMEM (and the dS tile has been read)
  const Bar mk_full{bars_s + 8 * 25};    // [G] the mask of row g of the current item is in shared memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 22);  // (bars 23, 24: sdone; 25..31: mk_full)
  const uint32_t abort_s = smem_u32(const_cast<int*>(abort_flag));

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform, and known to be)
  constexpr int kBRow = kBias16 ? BT * 2 : BT * 4;  // bytes per row (one query, 128 keys) of the staged bias tile
  const Steps<G> steps(a, n_items);
  const int NT = steps.NT, my_items = steps.items, total_steps = steps.total;

  grid_dependency_wait();
  grid_launch_dependents();
  if (tid == 0) *abort_flag = (a.status && *reinterpret_cast<volatile int*>(a.status) != 0) ? 1 : 0;
  __syncthreads();
  if (*abort_flag) return;

  if (tid == 0) {
    for (int i = 0; i < G; ++i) { mbar_init(bars + 0 + i, 1); mbar_init(bars + 7 + i, 3); mbar_init(bars + 25 + i, 1); }  // kv_full; kv_empty: three MMA warps read K/V
    for (int i = 0; i < kStages; ++i) { mbar_init(bars + 32 + i, 1); mbar_init(bars + 40 + i, 2); }  // st_full, st_empty
    for (int i = 0; i < 2; ++i) {
      mbar_init(bars + 48 + 2 * i, 3); mbar_init(bars + 52 + 2 * i, kCW / 2);  // sd_full: two commits, one warp; cdone
      mbar_init(bars + 14 + i, 1); mbar_init(bars + 16 + i, kCW / 2);  // b_full, b_done
      mbar_init(bars + 23 + i, kCW / 2);                               // sdone
    }
    mbar_init(bars + 19, 1);  // dq_full
    fence_mbar_init();
    prefetch_tmap(&tmQ); prefetch_tmap(&tmK); prefetch_tmap(&tmV); prefetch_tmap(&tmDO);
    prefetch_tmap(&tmNL); prefetch_tmap(&tmDL); prefetch_tmap(&tmDQ);
    prefetch_tmap(&tmB); prefetch_tmap(&tmDB);
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
      issue_scores_and_outputs<T, DP>(warp == kCW, tmem, smem_u32(sKV), smem_u32(sStage), NT, total_steps,
                                      IssueBars{kv_full, kv_empty, st_full, st_empty, sd_full, cdone, Bar{0}}, abort_s, [] {});
    } else if (warp == kCW + 2) {
      // =============================== tensor-core issuer of dQ; pair-bias loads ===============================
      const uint32_t sKV_s = smem_u32(sKV), sDS_s = smem_u32(sDS);
      const uint32_t sBias_s = smem_u32(sBias);
      // The bias tile (i, j) is the same for the G rows of a group; each half (64 queries) is loaded
      // for the group's first step and replaced as soon as the warps of that half have read it for
      // the last time.
      auto load_bias = [&](const StepT& d, int h) {
        if (elect_one()) {
          mbar_expect_tx(b_full + h, HT * kBRow);
          tma_load_4d_s(sBias_s + h * (HT * kBRow), &tmB, (b_full + h).a, d.j0, d.it * BT + h * HT, d.h, d.b);
        }
        __syncwarp();
      };
      const int tiles = my_items * NT;
      if (tiles > 0) { const StepT d0 = steps.decode(0); load_bias(d0, 0); load_bias(d0, 1); }
      if (elect_one()) mbar_arrive(dq_full);  // (for the first step, which has none before it)
      __syncwarp();
      int g = 0, it = 0, t = 0;  // row of the group, query tile, running (item, query tile) index
#pragma unroll 1
      for (int n = 0; n < total_steps; ++n) {
        const bool turn = g == G - 1 && t + 1 < tiles;  // the group's last step: the halves come back
        StepT nb = StepT{0, 0, 0, 0, 0, 0};
        if (turn) nb = steps.decode((t + 1) * G);  // (divisions: before the waits, not between them)
        if (turn) {
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            mbar_wait(b_done + h, t & 1, abort_s, DEV_TIMEOUT_SYNC);
            load_bias(nb, h);
          }
        }
        mbar_wait(sdone + 0, n & 1, abort_s, DEV_TIMEOUT_SYNC);
        mbar_wait(sdone + 1, n & 1, abort_s, DEV_TIMEOUT_SYNC);
        tc_fence_after();
        const uint32_t el = issue_dq<T, DP>(tmem + L::colDQ, sDS_s, sKV_s + 2 * g * L::kTile);
        mma_commit_if_s(el, dq_full.a);
        if (it == NT - 1) mma_commit_if_s(el, (kv_empty + g).a);
        if (++g == G) { g = 0; ++t; if (++it == NT) it = 0; }
      }
    } else {
      // =============================== tile loader ===============================
      // K/V of row g stay for the whole item and are replaced when the item's last MMAs that read them
      // have completed; Q, dO and the two statistics vectors of a step ride a two-deep ring.
      const uint32_t sKV_s = smem_u32(sKV), sStage_s = smem_u32(sStage), sMask_s = smem_u32(smem + L::offMask);
      StepT d = steps.decode(0);
#pragma unroll 1
      for (int n = 0; n < total_steps; ++n) {
        const int stg = n % kStages;
        if (d.it == 0) {
          const int k = n / (NT * G);
          // The mask of the row: four keys a lane, loaded before the wait.  (The last dQ MMA of the row is behind
          // kv_empty, so its last step has read the mask before.)
          float mk[4];
          if constexpr (L::kMaskRows > 0) {
#pragma unroll
            for (int u = 0; u < 4; ++u) mk[u] = mask_term<T>(a, d.b, d.s, d.j0 + lane + 32 * u);
          }
          mbar_wait(kv_empty + d.g, (k & 1) ^ 1, abort_s, DEV_TIMEOUT_MMA);
          if constexpr (L::kMaskRows > 0) {
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
        }
        mbar_wait(st_empty + stg, ((n / kStages) & 1) ^ 1, abort_s, DEV_TIMEOUT_MMA);
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
        d = steps.advance(d, n + 1);
      }
    }
  } else {
    // =============================== compute warps ===============================
    // Warps 0-7 work on half 0 (queries 0..63 of the tile) of every step, warps 8-15 on half 1: two
    // groups that run half a step apart, so that while one waits (for its S^T/dP^T, for tensor
    // memory, for its MMAs) the other has arithmetic to issue.  Warp w: keys 32*(w%4).. (its TMEM
    // lanes), queries 32*((w/4)%2).. of its half, in two chunks of 16.  Their instructions set the pace (five warps
    // a scheduler, no wait of any length): positions are loop counters and the mask of a key comes staged.
    // Backward calls with that, the issue loops walked by converged warps and the waits in one short sequence,
    // before and after, us: [1,128,384,8,32] 211 -> 195, [1,384,384,4,32] 348 -> 306, [1,1024,384,8,8] fp16
    // 1251 -> 1083, [1,128,768,8,64] 1195 -> 1148 (1 096 now), [4,1,2048,32,64] without d(pair_bias) 819 -> 742.
    setmaxnreg_inc<kComputeRegs>();
    const int q4 = warp & 3, cb2 = (warp >> 2) & 1, H = warp >> 3;
    const int jrow = q4 * 32 + lane;
    const uint32_t t_lane = tmem + (static_cast<uint32_t>(q4 * 32) << 16);
    const uint32_t cS = t_lane + (H ? L::colS1 : L::colS0) + QT * cb2, cP = t_lane + (H ? L::colDP1 : L::colDP0) + QT * cb2;
    const float inv_r = 1.f / (float)a.R;
    const float c1 = a.scale * kLog2e;
    // 32-bit shared-window addresses: every access below stays a shared-memory instruction
    const uint32_t sStage_s = smem_u32(sStage), sDS_s = smem_u32(sDS);
    const uint32_t outB_s = smem_u32(smem + L::offOutB) + warp * L::kOutB;  // this warp's own staging areas
    const uint32_t outQ_s = smem_u32(smem + L::offOutQ) + (warp & 7) * L::kOutQ;
    const uint32_t brow0 = smem_u32(sBias) + (H * HT + QT * cb2) * kBRow + jrow * (kBias16 ? 2 : 4);
    const uint32_t drow = sDS_s + H * (L::kDS / 2) + jrow * 128;

    // Every step has one bulk group per warp with its dQ partial (empty in a warp that takes none).  Before that one
    // there may be one with dK or dV, then one with half of a d(pair_bias).
    auto staging_free = [&](bool all) {  // all groups have been read, or all but the last
      if (lane == 0) {
        if (all) tma_wait_group_read0();
        else tma_wait_group_read1();
      }
      __syncwarp();
    };
    // dQ of a step (TMEM lanes = queries): the warps of half 1 take QC columns of 32 query rows each to their staging
    // areas, from where they are added to the fp32 accumulator in global memory by one small bulk tensor reduction per
    // warp.  (Half 0 takes dK and dV.  Rows of 64 bytes instead of 32: 5.1 TB/s of reductions instead of 3.6, the chip
    // over, and half as many instructions.)
    constexpr int QC = L::QC;
    const bool takes_dq = H == 1;
    const int qcol = cb2 * QC;
    auto store_dq = [&](const uint32_t (&qr)[QC]) {  // (rows of 32 or 64 bytes, swizzled as wide: no bank conflicts)
      const int x = QC == 8 ? (lane >> 2) & 1 : (lane >> 1) & 3;
#pragma unroll
      for (int c = 0; c < QC / 4; ++c)
        sts_v4(outQ_s + lane * (QC * 4) + ((c ^ x) << 4), qr[4 * c], qr[4 * c + 1], qr[4 * c + 2], qr[4 * c + 3]);
    };
    // (row0: the first of the 32 query rows; slab: (b,h,s), negative for a padded row)
    auto send_dq = [&](int row0, int slab) {
      if (takes_dq && slab >= 0 && qcol < a.D) tma_reduce_add_3d_s(&tmDQ, outQ_s, qcol, row0, slab);
      tma_commit_group();
    };

    int p_row0 = 0, p_slab = -1;           // the step whose dQ partial has not left yet
    int pb = 0, ph = 0, ps0 = 0, pj0 = 0;  // the item whose dK/dV still sit in TMEM
    const uint32_t mask_s = smem_u32(smem + L::offMask) + jrow * 4;
    float mreg[L::kMaskRows == 0 ? G : 1];
    const F2 c12 = f2_make(c1, c1);
    F2 bacc[16];  // d(pair_bias) of this thread's key and its 32 queries, summed over the rows of a group
#pragma unroll
    for (int e = 0; e < 16; ++e) bacc[e] = f2_make(0.f, 0.f);
    // Half a sum (16 queries x 32 keys of a warp) to the staging area and from there, by a bulk tensor reduction that
    // the warp issues itself, to d(pair_bias).  The first half leaves as soon as the group's last row has been added
    // to it, the second a step later, by when the staging area has been read (at the end of the same step it was
    // waited for, 900 cycles in three steps).
    auto flush_half = [&](int sub, int i0, int j0, int h, int b, bool all) {
      staging_free(all);
#pragma unroll
      for (int c = 0; c < 16; c += 2) {
        F2& acc = bacc[(sub * 16 + c) / 2];
        float b0, b1;
        f2_get(acc, b0, b1);
        sts_f32(outB_s + c * 128 + lane * 4, b0);
        sts_f32(outB_s + (c + 1) * 128 + lane * 4, b1);
        acc = f2_make(0.f, 0.f);
      }
      fence_async_shared();
      __syncwarp();
      if (lane == 0) {
        tma_reduce_add_4d_s(&tmDB, outB_s, j0 + q4 * 32, i0 + H * HT + QT * cb2 + 16 * sub, h, b);
        tma_commit_group();
      }
    };
    // dK (cb2 = 0) or dV (1) of row-group slot g, 32 keys, by a bulk store from the staging area.  Done by the warps of
    // half 0: they are the ones whose arrival lets the next item's first MMAs overwrite the slot.  (Straight from
    // registers, sixteen bytes of 32 rows an instruction, it took 900 to 1 700 cycles at each of an item's first steps.)
    auto send_dk_or_dv = [&](int g, bool all) {
      uint32_t r[DP];
      tmem_ld<DP>(t_lane + (cb2 ? L::colDV : L::colDK) + g * DP, r);
      staging_free(all);
      tmem_wait_ld();
      const float f = cb2 ? 1.f : a.scale;
      const int x = DP == 16 ? (lane >> 2) & 1 : (lane >> 1) & 3;  // (swizzled as wide as a row)
#pragma unroll
      for (int c = 0; c < DP / 8; ++c) {
        uint32_t w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) w[u] = Pack2<T>::pack(__uint_as_float(r[8 * c + 2 * u]) * f, __uint_as_float(r[8 * c + 2 * u + 1]) * f);
        sts_v4(outB_s + lane * (DP * 2) + ((c ^ x) << 4), w[0], w[1], w[2], w[3]);
      }
      fence_async_shared();
      __syncwarp();
      if (lane == 0) {
        const int j = pj0 + q4 * 32, s = ps0 + g;
        if (j < a.R && s < a.S) tma_store_5d_s(cb2 ? &tmDV : &tmDK, outB_s, 0, j, s, ph, pb);
        tma_commit_group();
      }
    };

    int n = 0;          // running step
    uint32_t tile = 0;  // running (item, query tile)
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
        mj = mreg[0];  // (the rows take turns: chosen by g, the compiler made 44 instructions a step of it)
#pragma unroll
        for (int r = 0; r + 1 < G; ++r) mreg[r] = mreg[r + 1];
        mreg[G - 1] = mj;
      } else {
        if (it == 0) mbar_wait(mk_full + g, k & 1, abort_s, DEV_TIMEOUT_TMA);
        mj = lds_f32(mask_s + g * (BT * 4));
      }
      if (g == 0) mbar_wait(b_full + H, tile & 1, abort_s, DEV_TIMEOUT_TMA);
      mbar_wait(sd_full + 2 * H, n & 1, abort_s, DEV_TIMEOUT_MMA);  // S^T and dP^T, statistics
      tc_fence_after();
      // A row whose keys are all dropped has this nl for every query (the mask row is shared by all queries of the MSA
      // row).  Its S and dP are cleared before they are read: their NaNs and infinities would stay in bacc, which the
      // group's other rows share.  (As a branch around the arithmetic it costs 6 to 7 %.  This way forward and backward of
      // [1,128,384,8,32] take 244 us with an fp32 bias and 246 with a 16-bit one, unguarded 243 and 243.)
      const bool dead = __any_sync(0xffffffffu, lds_f32(vec_s) == kDeadRow);
      if (dead) {
        uint32_t z[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) z[e] = 0u;
        tmem_st32(cS, z);
        tmem_st32(cP, z);
        tmem_wait_st();
      }
      const F2 mj2 = f2_make(mj, mj);
      // dK and dV of the item before, ahead of this step's MMAs into them.  (All of the other half's MMAs into them were
      // issued before the S^T and dP^T of this step.)
      const bool drain = H == 0 && it == 0 && k > 0;
      if (drain) send_dk_or_dv(g, false);
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
        score_chunk<T, true>(
            sr, dr, vnl, vdl,
            [&](int e) { return staged_bias<T, kBias16>(brow + e * kBRow); }, c12, mj2, pk, dk + 8 * sub,
            [&](int e, F2 ds) { bacc[8 * sub + e] = f2_add(bacc[8 * sub + e], ds); });
        // P^T and dS^T, two 16-bit values per column, over the columns this thread has just read:
        // the A operands of the dV and dK MMAs (16 queries = 8 packed columns each)
        tmem_st8(cS + 16 * sub, pk);
        tmem_st8(cP + 16 * sub, *reinterpret_cast<uint32_t(*)[8]>(&dk[sub * 8]));
        if (sub == 0) {
          if (last_of_group) flush_half(0, it * BT, cur.j0, cur.h, cur.b, drain);
          if (g == 0 && tile > 0) {
            const bool turn = it == 0;
            flush_half(1, (turn ? NT - 1 : it - 1) * BT, turn ? pj0 : cur.j0, turn ? ph : cur.h, turn ? pb : cur.b, drain);
          }
        }
      }
      if (dead) {  // P is 1/N_res, dS 0
        const float pu = (cur.j0 + jrow < a.R) ? inv_r : 0.f;
        uint32_t w[8], z[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) { w[e] = Pack2<T>::pack(pu, pu); z[e] = 0u; }
        tmem_wait_st();
#pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
          tmem_st8(cS + 16 * sub, w);
          tmem_st8(cP + 16 * sub, z);
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) dk[e] = 0u;
      }
      if (last_of_group) {  // (every value read has been worked on, so the loads are through)
        __syncwarp();
        if (lane == 0) mbar_arrive(b_done + H);
      }
      // P^T and dS^T are in tensor memory: the dV / dK MMAs and the next S^T and dP^T may go, under what follows
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(cdone + 2 * H);
      // dQ of the step before is complete, so the dS tile has been read as well.  Its MMAs ran underneath this step.
      mbar_wait(dq_full, n & 1, abort_s, DEV_TIMEOUT_MMA);
      tc_fence_after();
      // dS^T -> shared memory, [key][query] rows of 128 bytes per half, 128-byte swizzle
#pragma unroll
      for (int c = 0; c < 4; ++c)  // dk[4 * c ..]: queries 32 * cb2 + 8 * c .. of this half
        sts_v4(drow + (((4 * cb2 + c) ^ (jrow & 7)) << 4), dk[4 * c], dk[4 * c + 1], dk[4 * c + 2], dk[4 * c + 3]);
      if (takes_dq) {
        uint32_t qr[QC];
        tmem_ld<QC>(t_lane + L::colDQ + qcol, qr);
        if (lane == 0) {
          if (last_of_group || g == 0) tma_wait_group_read1();  // (d(pair_bias) left since the last dQ)
          else tma_wait_group_read0();
        }
        __syncwarp();
        tmem_wait_ld();
        store_dq(qr);
      }
      fence_async_shared();
      tc_fence_before();  // (the next MMAs into the dQ columns just read follow from this arrival)
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(sdone + H);
        send_dq(p_row0, p_slab);
      }
      p_row0 = it * BT + q4 * 32;
      p_slab = cur.s + g < a.S ? (cur.b * a.H + cur.h) * a.S + cur.s + g : -1;
    }
    pb = cur.b; ph = cur.h; ps0 = cur.s; pj0 = cur.j0;
    }

    if (total_steps > 0) {
      flush_half(1, (NT - 1) * BT, pj0, ph, pb, true);
      mbar_wait(dq_full, total_steps & 1, abort_s, DEV_TIMEOUT_MMA);
      tc_fence_after();
      if (takes_dq) {
        uint32_t qr[QC];
        tmem_ld<QC>(t_lane + L::colDQ + qcol, qr);
        staging_free(true);
        tmem_wait_ld();
        store_dq(qr);
        fence_async_shared();
        __syncwarp();
        if (lane == 0) send_dq(p_row0, p_slab);
      }
      if (H == 0) {
        // every dV / dK MMA of this CTA has completed once the last step's tile stage has been released
        const int last = total_steps - 1;
        mbar_wait(st_empty + (last & 1), (last >> 1) & 1, abort_s, DEV_TIMEOUT_MMA);
        tc_fence_after();
#pragma unroll 1
        for (int g = 0; g < G; ++g) send_dk_or_dv(g, true);
      }
    }
    if (lane == 0) tma_wait_group0();  // this warp's reductions have completed before the CTA may exit
  }

  end_of_cta(abort_flag, a.status);
  if (warp == 0) tmem_dealloc(tmem, L::kTmemCols);
}

size_t align_up(size_t x, size_t al) { return (x + al - 1) / al * al; }

// One vector of row statistics: [B,H,S,delta_ld] fp32.
size_t stats_bytes(const Args& a) { return align_up((size_t)a.B * a.H * a.S * a.delta_ld * sizeof(float), 256); }

// Above a head dimension of 32: whether d(pair_bias) comes from a kernel that computes S and dP again (bwd_dbias.cuh), or
// leaves the kernel that gives dQ, dK and dV as reductions, 64 KB a step.  An item of the former costs its rows and about
// two more, so it takes many rows (and tiles, for there to be an item for every SM without cutting the rows up) to save
// what the reductions cost.  Forward and backward, us, apart and as reductions, fp32 bias:
//   one row:    [4,1,2048,32,64] 3 192 and 1 973, [4,1,300,32,64] 124 and 84, [1,1,300,8,64] 39 and 33
//   few:        [1,4,768,8,64] 86 and 76, [1,8,2048,8,64] 635 and 579, [1,16,512,8,64] 107 and 101
//   about even: [1,64,384,8,64] 219 and 219, [1,64,300,8,64] 198 and 197, [1,96,640,4,64] 378 and 376, [1,24,1536,4,64] 480
//               and 479
//   many:       [1,32,768,8,64] 352 and 364, [1,128,384,8,64] 401 and 405, [1,512,257,8,64] 1 277 and 1 310,
//               [1,56,1536,4,64] 1 027 and 1 083
//   two tiles:  [1,512,128,8,64] 330 and 304, [1,128,200,4,64] 115 and 107, [2,512,256,8,64] 1 564 and 1 553
bool apart_pays(const Args& a) {
  const long long NT = (a.R + BT - 1) / BT;
  return NT > 2 && a.S * NT >= 192;
}

template <class T, int DP>
int launch_t(const Args& a0, void* ws, size_t ws_bytes, cudaStream_t st, int* launches) {
  constexpr int G = RowsPerItem<DP>::G;
  Args a = a0;
  const size_t rows = (size_t)a.B * a.H * a.S * a.R;
  const size_t vec_bytes = stats_bytes(a);
  if (ws_bytes < sm100_bwd_workspace_bytes(0, a)) return EVOATTN_ERR_WORKSPACE;
  a.delta = reinterpret_cast<float*>(ws);
  float* nl = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ws) + vec_bytes);
  float* dq_acc = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ws) + 2 * vec_bytes);
  if (a.dgate) {
    launch_prep<T, true>(a, nl, dq_acc, st);
    use_effective_d_o(&a);
  } else {
    launch_prep<T, false>(a, nl, dq_acc, st);
  }

  CUtensorMap tq, tk, tv, tdo, tb, tdb, tdq, tnl, tdl, tdk, tdv;
  if (!make_qkv_map(&tq, a.q, a.sq, a.B, a.H, a.S, a.R, a.D, DP, BT)) return EVOATTN_ERR_CUDA;
  if (!make_qkv_map(&tk, a.k, a.sk, a.B, a.H, a.S, a.R, a.D, DP, BT)) return EVOATTN_ERR_CUDA;
  if (!make_qkv_map(&tv, a.v, a.sv, a.B, a.H, a.S, a.R, a.D, DP, BT)) return EVOATTN_ERR_CUDA;
  if (!make_qkv_map(&tdo, a.d_o, a.sdo, a.B, a.H, a.S, a.R, a.D, DP, BT)) return EVOATTN_ERR_CUDA;
  constexpr bool kApart = DP == 64;  // d(pair_bias) may have a kernel of its own
  const bool nodbias = kApart || !a.dbias;
  const long long slabs = (long long)a.B * a.H * a.S;
  if (!(nodbias ? make_rows_f32_map(&tdq, dq_acc, a.D, a.R, slabs, DP < 32 ? DP : 32, BT, /*swizzle=*/true)
                : make_rows_f32_map(&tdq, dq_acc, a.D, a.R, slabs, DP / 2, 32, /*swizzle=*/true)))
    return EVOATTN_ERR_CUDA;
  if (!make_stats_map(&tnl, nl, a.B * a.H, a.S, a.R, a.delta_ld, BT)) return EVOATTN_ERR_CUDA;
  if (!make_stats_map(&tdl, a.delta, a.B * a.H, a.S, a.R, a.delta_ld, BT)) return EVOATTN_ERR_CUDA;
  tb = tq;
  tdb = tq;
  tdk = tdv = tq;
  const int box_kv = nodbias ? BT : 32;
  if ((G == 1 || !nodbias) && (!make_qkv_map(&tdk, a.dk, a.sdk, a.B, a.H, a.S, a.R, a.D, DP, box_kv) ||
                               !make_qkv_map(&tdv, a.dv, a.sdv, a.B, a.H, a.S, a.R, a.D, DP, box_kv)))
    return EVOATTN_ERR_CUDA;
  if (a.bias) {
    const bool ok = a.bias16 ? make_bias16_map(&tb, a.bias, a.sbias, a.B, a.H, a.R, HT, BT, /*swizzle=*/false)
                             : make_bias_plain_map(&tb, a.bias, a.sbias, a.B, a.H, a.R, HT, BT);
    if (!ok) return EVOATTN_ERR_CUDA;
    const Str3 dense{(long long)a.H * a.R * a.dbias_ld, (long long)a.R * a.dbias_ld, (long long)a.dbias_ld};
    if (!nodbias && !make_bias_plain_map(&tdb, a.dbias, dense, a.B, a.H, a.R, 16, 32)) return EVOATTN_ERR_CUDA;
  }
  const int NT = (a.R + BT - 1) / BT;
  const long long items = (long long)a.B * a.H * NT * ((a.S + G - 1) / G);
  if (items > 0x7fffffffLL / (G * NT)) return EVOATTN_ERR_SHAPE;
  const int sms = sm_count();
  if (sms <= 0) return EVOATTN_ERR_CUDA;
  const long long ctas = items < sms ? items : sms;
  auto kern_n = !a.bias ? evo_bwd_nodbias_sm100_kernel<T, DP, BIAS_NONE, false>
                : a.bias16 ? evo_bwd_nodbias_sm100_kernel<T, DP, BIAS_16, false> : evo_bwd_nodbias_sm100_kernel<T, DP, BIAS_F32, false>;
  bool apart = false;
  if constexpr (kApart) {
    apart = a.dbias && apart_pays(a);
    if (a.dbias && !apart) kern_n = a.bias16 ? evo_bwd_nodbias_sm100_kernel<T, DP, BIAS_16, true> : evo_bwd_nodbias_sm100_kernel<T, DP, BIAS_F32, true>;
  }
  const void* entry = reinterpret_cast<const void*>(kern_n);
  size_t smem = !a.bias ? SmemN<DP, BIAS_NONE>::bytes : a.bias16 ? SmemN<DP, BIAS_16>::bytes : SmemN<DP, BIAS_F32>::bytes;
  if constexpr (!kApart) {
    if (!nodbias) {
      entry = a.bias16 ? reinterpret_cast<const void*>(evo_bwd_sm100_kernel<T, DP, true>) : reinterpret_cast<const void*>(evo_bwd_sm100_kernel<T, DP, false>);
      smem = SmemT<DP>::bytes;
    }
  }
  // setmaxnreg.inc waits until the scheduler's register pool (five warps at the launch-time count)
  // has what it asks for: never launch a build whose pool cannot hold the warps' requests.
  int num_regs = 0;
  if (!kernel_ready(entry, (int)smem, &num_regs)) return EVOATTN_ERR_CUDA;
  if ((kThreadsT / 128) * num_regs < 4 * kComputeRegs + kServiceRegs) return EVOATTN_ERR_UNSUPPORTED;
  if (nodbias) launch_dependent(kern_n, dim3((unsigned)ctas), kThreadsT, smem, st, a, (int)items, tq, tk, tv, tdo, tb, tdq, tnl, tdl, tdk, tdv);
  if constexpr (kApart) {
    if (apart) {
      const auto kern_b = a.bias16 ? evo_bwd_dbias_sm100_kernel<T, DP, true> : evo_bwd_dbias_sm100_kernel<T, DP, false>;
      if (!kernel_ready(reinterpret_cast<const void*>(kern_b), (int)SmemB<DP>::bytes, &num_regs)) return EVOATTN_ERR_CUDA;
      if ((kThreadsT / 128) * num_regs < 4 * kComputeRegs + kServiceRegs) return EVOATTN_ERR_UNSUPPORTED;
      const WalkB walk = walk_b(a, sms);
      launch_dependent(kern_b, dim3((unsigned)(walk.n_items < sms ? walk.n_items : sms)), kThreadsT, SmemB<DP>::bytes, st, a, walk, tq, tk, tv, tdo, tnl, tdl);
      *launches += 1;
    }
  } else {
    const auto kern = a.bias16 ? evo_bwd_sm100_kernel<T, DP, true> : evo_bwd_sm100_kernel<T, DP, false>;
    if (!nodbias) launch_dependent(kern, dim3((unsigned)ctas), kThreadsT, smem, st, a, (int)items, tq, tk, tv, tdo, tb, tdb, tdq, tnl, tdl, tdk, tdv);
  }
  if (a.dbias_out) {
    const int rc = launch_dbias_out(a, st, launches);
    if (rc) return rc;
  }
  // d(pair_bias) is complete: its sum over the GPUs of the node, if the caller asked for one, runs on
  // a stream of its own next to the dQ store below; the caller's stream waits for it at the end
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  if (a.exchange) {
    if (!exchange_lane(&side, &fork, &join)) return EVOATTN_ERR_CUDA;
    if (cudaEventRecord(fork, st) != cudaSuccess || cudaStreamWaitEvent(side, fork, 0) != cudaSuccess) return EVOATTN_ERR_CUDA;
    const int rc = launch_peer_allreduce(reinterpret_cast<const evoattn_peer_allreduce_params*>(a.exchange), side);
    if (cudaEventRecord(join, side) != cudaSuccess) return EVOATTN_ERR_CUDA;  // (join even after a failed launch)
    if (rc) { cudaStreamWaitEvent(st, join, 0); return rc; }
    *launches += 1;
  }
  const long long n8 = (long long)rows * (a.D / 8);
  const dim3 store_grid((unsigned)((n8 + 255) / 256));
  const auto store = n8 <= 0x7fffffffLL ? dq_store_kernel<T, uint32_t> : dq_store_kernel<T, unsigned long long>;
  if (a.exchange) store<<<store_grid, 256, 0, st>>>(a, dq_acc);  // (another launch lies between)
  else launch_dependent(store, store_grid, 256, 0, st, a, static_cast<const float*>(dq_acc));
  if (a.exchange && cudaStreamWaitEvent(st, join, 0) != cudaSuccess) return EVOATTN_ERR_CUDA;
  *launches += 3;
  return cudaGetLastError() == cudaSuccess ? EVOATTN_OK : EVOATTN_ERR_CUDA;
}

// Head dimensions up to 16: items of seven rows (padded to 16 columns) flush d(pair_bias) and reload the bias
// tile every seventh step instead of every third, but there are fewer of them and the last group of rows is
// padded further.  They are taken where the CTA with the most steps gets no more than 15 % more of them, or 5 % with
// an fp32 bias that wants no gradient (whose third half tile then pays for itself at three rows already).  Time of
// the backward call, seven rows over three, by how many more steps that CTA gets (D = 8 and 16, N_res 200 to 1000, 26
// shapes):
//                                as many    5 % more   10 %       17 %       27 %
//   with d(pair_bias):           0.86-0.89  0.91-0.94  0.94-0.98  0.99-1.03  1.11-1.12
//   with an fp32 bias alone:     0.90-0.95  0.95-0.99  0.97-1.03  1.03-1.09  1.15-1.18
//   with a 16-bit bias alone:    0.83-0.87  0.89-0.92  0.88-0.95  0.96-1.01  1.09-1.10
//   without a bias:              0.80-0.85  0.85-0.91  0.88-0.92  0.94-0.98  1.03-1.05
bool seven_rows_pay(const Args& a, int sms) {
  const auto steps = [&](int G) {
    const long long items = (long long)a.B * a.H * ((a.R + BT - 1) / BT) * ((a.S + G - 1) / G);
    return (items + sms - 1) / sms * G;
  };
  return 100 * steps(7) <= (a.bias && !a.bias16 && !a.dbias ? 105 : 115) * steps(3);
}

}  // namespace

bool sm100_bwd_supported(int dtype, const Args& a) {
  if (!sm100_fwd_supported(dtype, a)) return false;
  const long long NT = (a.R + BT - 1) / BT;
  if ((long long)a.B * a.H * NT * a.S > 2147483647LL) return false;
  return true;
}

size_t sm100_bwd_workspace_bytes(int, const Args& a) {
  const size_t rows = (size_t)a.B * a.H * a.S * a.R;
  return 2 * stats_bytes(a) + align_up(rows * a.D * sizeof(float), 256);
}

int launch_sm100_bwd(int dtype, const Args& a, void* workspace, size_t workspace_bytes, cudaStream_t st,
                     int* launches) {
  const int sms = sm_count();
  if (sms <= 0) return EVOATTN_ERR_CUDA;
  if (a.D <= 16 && seven_rows_pay(a, sms)) {
    if (dtype == EVOATTN_BF16) return launch_t<__nv_bfloat16, 16>(a, workspace, workspace_bytes, st, launches);
    return launch_t<__half, 16>(a, workspace, workspace_bytes, st, launches);
  }
  if (a.D <= 32) {
    if (dtype == EVOATTN_BF16) return launch_t<__nv_bfloat16, 32>(a, workspace, workspace_bytes, st, launches);
    return launch_t<__half, 32>(a, workspace, workspace_bytes, st, launches);
  }
  if (dtype == EVOATTN_BF16) return launch_t<__nv_bfloat16, 64>(a, workspace, workspace_bytes, st, launches);
  return launch_t<__half, 64>(a, workspace, workspace_bytes, st, launches);
}

}  // namespace evo
