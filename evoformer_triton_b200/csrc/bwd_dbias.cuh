// d(pair_bias) by itself, for head dimensions above 32 and many MSA rows (apart_pays): the sum over the rows of dS, from S
// and dP computed again.
//
// Up to a head dimension of 32 d(pair_bias) leaves the fused kernel (bwd_sm100.cu) as fp32 reductions, 64 KB a tile and row
// group.  Above, tensor memory holds the dK and dV of one row only, so that is 64 KB a step next to 32 KB of dQ, at the 21
// bytes a cycle and SM that reductions leave at (5.9 TB/s, the chip over): 4 600 cycles of a step's 7 200 when the fused
// kernel served these too.  Here a CTA keeps a 128 x 128 tile of d(pair_bias) in registers while it walks the MSA rows, and
// so does its tile of the bias: dS costs two products, two FMAs, an exponential and a third FMA an element, and nothing is
// written before the last row.  dQ, dK and dV come from the kernel without a d(pair_bias) (bwd_nodbias.cuh).  Bound by the
// exponentials (68 % of their unit's rate, 1 500 cycles a step).  Forward and backward, us, fused and now:
// [1,128,384,8,64] 446 and 401, [1,512,257,8,64] 1 464 and 1 277, [1,32,768,8,64] 389 and 352.
//
// Replaces the d_pair_bias half of dsevoformer-triton/evoformer.py:329-476 (the atomic of :458).
//
// Work item = (b, h, run of rows, query tile, key tile), tiles fastest, so that the CTAs that work side by side read
// the same rows out of L2.  Warps 0-15 compute (warp w: queries 32*(w%4).., keys 32*(w/4)..; a thread owns a query, its
// TMEM lane, and 32 keys), 16 loads tiles, 17 issues the MMAs, 18 stages the residue mask.  Bias and sum are 64 of a
// compute thread's 112 registers, and eight bytes of the rest are spilled.
#pragma once

#include "bwd_common.cuh"

namespace evo {
namespace {

template <int DP>
struct SmemB {
  static_assert(DP == 64, "up to 32 columns d(pair_bias) leaves the fused kernel");
  static constexpr int kTile = BT * DP * 2;
  static constexpr int kStage = 4 * kTile;                   // Q, dO, K, V of a row
  static constexpr int kStages3 = 3;
  static constexpr int kSlots = 8;                           // of statistics and masks: more than the steps in flight
  static constexpr int kVecs = 2 * BT * 4;                   // -lse*log2e and -delta of the row's queries
  static constexpr int offStage = 0;
  static constexpr int offVecs = offStage + kStages3 * kStage;
  static constexpr int offMask = offVecs + kSlots * kVecs;   // [slot][128 keys]: what the mask adds to a score
  static constexpr int offDirty = offMask + kSlots * BT * 4; // [slot]: bit u: the mask changes one of keys 32 u ..
  static constexpr int offBars = offDirty + kSlots * 4;
  static constexpr size_t bytes = offBars + 512 + 1024;
  static_assert(kStage % 1024 == 0, "swizzled tiles need 1024-byte alignment");
  static_assert(bytes <= 232448, "shared memory budget of one CTA");
};

struct ItemB {
  int b, h, i0, j0, s0, s1;
};
// The items of this CTA: blockIdx.x, blockIdx.x + gridDim.x, ...
struct WalkB {
  int n_items, runs, rows;  // rows: of a run (the last one may have fewer)
};
__device__ __forceinline__ ItemB item_b(const Args& a, const WalkB& w, int idx) {
  const int NT = (a.R + BT - 1) / BT;
  ItemB t;
  t.j0 = (idx % NT) * BT; idx /= NT;
  t.i0 = (idx % NT) * BT; idx /= NT;
  t.s0 = (idx % w.runs) * w.rows; idx /= w.runs;
  t.s1 = min(t.s0 + w.rows, a.S);
  t.h = idx % a.H;
  t.b = idx / a.H;
  return t;
}

template <class T, int DP, bool kBias16>
__global__ void __launch_bounds__(kThreadsT, 1)
evo_bwd_dbias_sm100_kernel(const Args a, const WalkB walk, const __grid_constant__ CUtensorMap tmQ,
                           const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                           const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ CUtensorMap tmNL,
                           const __grid_constant__ CUtensorMap tmDL) {
  using L = SmemB<DP>;
  constexpr int NS = L::kStages3, SLOTS = L::kSlots, RB = DP * 2;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t smem_s = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::offBars);
  const uint32_t bars_s = smem_u32(bars);
  const Bar st_full{bars_s + 8 * 0};    // [NS] the tiles and statistics of a step landed
  const Bar st_empty{bars_s + 8 * 8};   // [NS] ... its MMAs have read the tiles
  const Bar sd_full{bars_s + 8 * 16};   // [2] S and dP of a step are in TMEM, its statistics and mask in shared memory
  const Bar t_empty{bars_s + 8 * 18};   // [2] ... have been read by every compute warp
  const Bar m_full{bars_s + 8 * 20};    // [SLOTS] the mask of a step is in shared memory
  const Bar m_empty{bars_s + 8 * 28};   // [SLOTS] ... has been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 40);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 41);
  const uint32_t abort_s = smem_u32(const_cast<int*>(abort_flag));

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform, and known to be)

  grid_dependency_wait();
  grid_launch_dependents();
  if (tid == 0) *abort_flag = (a.status && *reinterpret_cast<volatile int*>(a.status) != 0) ? 1 : 0;
  __syncthreads();
  if (*abort_flag) return;

  if (tid == 0) {
    for (int i = 0; i < NS; ++i) { mbar_init(bars + 0 + i, 1); mbar_init(bars + 8 + i, 1); }  // st_full, st_empty
    for (int i = 0; i < 2; ++i) { mbar_init(bars + 16 + i, 2); mbar_init(bars + 18 + i, kCW); }  // sd_full: a commit, a warp; t_empty
    for (int i = 0; i < SLOTS; ++i) { mbar_init(bars + 20 + i, 1); mbar_init(bars + 28 + i, 1); }  // m_full, m_empty
    fence_mbar_init();
    prefetch_tmap(&tmQ); prefetch_tmap(&tmK); prefetch_tmap(&tmV); prefetch_tmap(&tmDO);
    prefetch_tmap(&tmNL); prefetch_tmap(&tmDL);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  constexpr int kBuf = 2 * BT;  // columns of a (S, dP) buffer

  if (warp >= kCW) {
    setmaxnreg_dec<kServiceRegs>();
    if (warp == kCW) {
      // =============================== tile loader ===============================
      uint32_t n = 0, st = 0, par = 1;  // step, stage and its parity
#pragma unroll 1
      for (int idx = blockIdx.x; idx < walk.n_items; idx += gridDim.x) {
        const ItemB it = item_b(a, walk, idx);
#pragma unroll 1
        for (int s = it.s0; s < it.s1; ++s, ++n) {
          mbar_wait(st_empty + (int)st, par, abort_s, DEV_TIMEOUT_MMA);
          if (elect_one()) {
            // (The MMAs of step n - NS have completed, for which every warp had to be through with step n - NS - 3.)
            static_assert(SLOTS >= NS + 3, "a slot is free before its turn comes");
            const uint32_t dst = smem_s + L::offStage + st * L::kStage, bar = (st_full + (int)st).a;
            const uint32_t vec = smem_s + L::offVecs + (n % SLOTS) * L::kVecs;
            mbar_expect_tx(st_full + (int)st, L::kStage + L::kVecs);
            tma_load_5d_s(dst, &tmQ, bar, 0, it.i0, s, it.h, it.b);
            tma_load_5d_s(dst + 2 * L::kTile, &tmK, bar, 0, it.j0, s, it.h, it.b);
            tma_load_5d_s(dst + L::kTile, &tmDO, bar, 0, it.i0, s, it.h, it.b);
            tma_load_5d_s(dst + 3 * L::kTile, &tmV, bar, 0, it.j0, s, it.h, it.b);
            tma_load_3d_s(vec, &tmNL, bar, it.i0, s, it.b * a.H + it.h);
            tma_load_3d_s(vec + BT * 4, &tmDL, bar, it.i0, s, it.b * a.H + it.h);
          }
          __syncwarp();
          if (++st == (uint32_t)NS) { st = 0; par ^= 1; }
        }
      }
    } else if (warp == kCW + 1) {
      // =============================== tensor-core issuer ===============================
      constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
      constexpr uint32_t SWZ = swizzle_code_for_row_bytes(RB);
      constexpr uint32_t kIdesc = make_idesc(kBf16, false, false, BT, BT);
      constexpr uint32_t kHi = static_cast<uint32_t>(make_sdesc_const(16, 8 * RB, SWZ) >> 32);
      constexpr uint32_t kLoLbo = static_cast<uint32_t>(make_sdesc_const(16, 0, 0) & 0xffffffffu);
      uint32_t n = 0, st = 0, par = 0;
#pragma unroll 1
      for (int idx = blockIdx.x; idx < walk.n_items; idx += gridDim.x) {
        const ItemB it = item_b(a, walk, idx);
#pragma unroll 1
        for (int s = it.s0; s < it.s1; ++s, ++n) {
          const int buf = n & 1;
          const uint32_t base = ((smem_s + L::offStage + st * L::kStage) >> 4) | kLoLbo;
          const uint32_t tS = tmem + buf * kBuf;
          // (the first two steps find their buffers free)
          mbar_wait(t_empty + buf, ((n >> 1) & 1) ^ 1, abort_s, DEV_TIMEOUT_SYNC);
          // A warp arrives there with the last of S and dP in registers, and is through with the step before.
          if (n >= 3) {
            if (elect_one()) mbar_arrive(m_empty + (int)((n - 3) % SLOTS));
            __syncwarp();
          }
          mbar_wait(st_full + (int)st, par, abort_s, DEV_TIMEOUT_TMA);
          tc_fence_after();
          const uint32_t el = elect_one();
#pragma unroll
          for (int kk = 0; kk < DP / 16; ++kk)  // S = Q K^T
            mma_ss_e(el, tS, pack_desc(base + 2 * kk, kHi), pack_desc(base + (2 * L::kTile >> 4) + 2 * kk, kHi), kIdesc, kk > 0 ? 1u : 0u);
#pragma unroll
          for (int kk = 0; kk < DP / 16; ++kk)  // dP = dO V^T
            mma_ss_e(el, tS + BT, pack_desc(base + (L::kTile >> 4) + 2 * kk, kHi), pack_desc(base + (3 * L::kTile >> 4) + 2 * kk, kHi), kIdesc,
                     kk > 0 ? 1u : 0u);
          mma_commit_if_s(el, (sd_full + buf).a);
          mma_commit_if_s(el, (st_empty + (int)st).a);
          mbar_wait(m_full + (int)(n % SLOTS), (n / SLOTS) & 1, abort_s, DEV_TIMEOUT_SYNC);
          if (elect_one()) mbar_arrive(sd_full + buf);
          __syncwarp();
          if (++st == (uint32_t)NS) { st = 0; par ^= 1; }
        }
      }
    } else if (warp == kCW + 2) {
      // =============================== residue-mask stager ===============================
      const uint32_t mask_s = smem_s + L::offMask, dirty_s = smem_s + L::offDirty;
      uint32_t n = 0;
#pragma unroll 1
      for (int idx = blockIdx.x; idx < walk.n_items; idx += gridDim.x) {
        const ItemB it = item_b(a, walk, idx);
#pragma unroll 1
        for (int s = it.s0; s < it.s1; ++s, ++n) {
          const uint32_t slot = n % SLOTS;
          float mk[4];
          uint32_t dirty = 0;
          if (a.mask_kind != EVOATTN_MASK_NONE) {
#pragma unroll
            for (int u = 0; u < 4; ++u) mk[u] = mask_term<T>(a, it.b, s, min(it.j0 + lane + 32 * u, a.R - 1));
          }
          mbar_wait(m_empty + (int)slot, ((n / SLOTS) & 1) ^ 1, abort_s, DEV_TIMEOUT_SYNC);
          if (a.mask_kind != EVOATTN_MASK_NONE) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              sts_f32(mask_s + (slot * BT + 32 * u + lane) * 4, mk[u]);
              if (__any_sync(0xffffffffu, mk[u] != 0.f)) dirty |= 1u << u;
            }
          }
          if (lane == 0) sts_u32(dirty_s + 4 * slot, dirty);
          __syncwarp();
          if (lane == 0) mbar_arrive(m_full + (int)slot);
        }
      }
    }
  } else {
    // =============================== compute warps ===============================
    setmaxnreg_inc<kComputeRegs>();
    const int q4 = warp & 3, kg = warp >> 2;
    const int row = q4 * 32 + lane;
    const uint32_t t_base = tmem + (static_cast<uint32_t>(q4 * 32) << 16) + 32 * kg;
    const float c1 = a.scale * kLog2e;
    const F2 c12 = f2_make(c1, c1), l2e2 = f2_make(kLog2e, kLog2e);
    uint32_t n = 0;
#pragma unroll 1
    for (int idx = blockIdx.x; idx < walk.n_items; idx += gridDim.x) {
      const ItemB it = item_b(a, walk, idx);
      const int i = it.i0 + row, j = it.j0 + 32 * kg;  // this thread's query and its first key
      // The bias of the query and the 32 keys, in registers for the whole item; zeros beyond the last ones.
      F2 bias[16], acc[16];
      {
        const size_t es = kBias16 ? 2 : 4;
        const unsigned char* p = reinterpret_cast<const unsigned char*>(a.bias) +
                                 (it.b * a.sbias.a + it.h * a.sbias.b + (long long)min(i, a.R - 1) * a.sbias.c + j) * es;
        const int left = i < a.R ? a.R - j : 0;
        constexpr int V = kBias16 ? 8 : 4;  // values of sixteen bytes (rows start on such a boundary)
#pragma unroll
        for (int g = 0; g < 32 / V; ++g) {
          uint32_t w[4] = {0u, 0u, 0u, 0u};
          if (g * V + V <= left) {
            const uint4 v = *reinterpret_cast<const uint4*>(p + 16 * g);
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
          } else if (g * V < left) {
            for (int u = 0; u < 4; ++u) {
              if constexpr (kBias16) {
                w[u] = ldg_u16_if(p + 16 * g + 4 * u, g * V + 2 * u < left);
                w[u] |= ldg_u16_if(p + 16 * g + 4 * u + 2, g * V + 2 * u + 1 < left) << 16;
              } else {
                w[u] = ldg_u32_if(p + 16 * g + 4 * u, g * V + u < left);
              }
            }
          }
          if constexpr (kBias16) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              float lo, hi;
              unpack2<T>(w[u], lo, hi);
              bias[4 * g + u] = f2_make(lo, hi);
            }
          } else {
            bias[2 * g] = f2_from_bits(w[0], w[1]);
            bias[2 * g + 1] = f2_from_bits(w[2], w[3]);
          }
        }
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) acc[e] = f2_make(0.f, 0.f);

#pragma unroll 1
      for (int s = it.s0; s < it.s1; ++s, ++n) {
        const int buf = n & 1;
        const uint32_t slot = n % SLOTS;
        const uint32_t vec_s = smem_s + L::offVecs + slot * L::kVecs;
        const uint32_t tS = t_base + buf * kBuf;
        mbar_wait(sd_full + buf, (n >> 1) & 1, abort_s, DEV_TIMEOUT_MMA);
        tc_fence_after();
        const float nl = lds_f32(vec_s + row * 4), dl = lds_f32(vec_s + BT * 4 + row * 4);
        const uint32_t dirty = __shfl_sync(0xffffffffu, lds_u32(smem_s + L::offDirty + 4 * slot), 0);
        const F2 nl2 = f2_make(nl, nl), dl2 = f2_make(dl, dl);
        auto accumulate = [&](auto masked) {
          const uint32_t mk_s = smem_s + L::offMask + (slot * BT + 32 * kg) * 4;
#pragma unroll
          for (int sub = 0; sub < 2; ++sub) {
            uint32_t sr[16], dr[16];
            tmem_ld16(tS + 16 * sub, sr);
            tmem_ld16(tS + BT + 16 * sub, dr);
            tmem_wait_ld();
            if (sub == 1) {  // S and dP have been read
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(t_empty + buf);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              F2 x = f2_fma(f2_from_bits(sr[2 * e], sr[2 * e + 1]), c12, f2_fma(bias[8 * sub + e], l2e2, nl2));
              if constexpr (decltype(masked)::value) {
                const float2 mk = lds_v2f(mk_s + (16 * sub + 2 * e) * 4);
                x = f2_add(x, f2_make(mk.x, mk.y));
              }
              float x0, x1;
              f2_get(x, x0, x1);
              const F2 p = f2_make(ex2(x0), ex2(x1));
              acc[8 * sub + e] = f2_fma(p, f2_add(f2_from_bits(dr[2 * e], dr[2 * e + 1]), dl2), acc[8 * sub + e]);
            }
          }
        };
        if (__all_sync(0xffffffffu, nl == kDeadRow || i >= a.R)) {  // a row whose keys are all dropped adds nothing
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(t_empty + buf);
        } else if ((dirty >> kg) & 1u) {
          accumulate(std::true_type{});
        } else {
          accumulate(std::false_type{});
        }
      }
      // The sum over the run's rows is added to d(pair_bias), which the first pass of the call has cleared.  (Its rows
      // are whole sixteen-byte pieces; the padding of a row may be written.)
      if (i < a.R) {
        float* out = a.dbias + (((long long)it.b * a.H + it.h) * a.R + i) * a.dbias_ld + j;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          if (j + 4 * g < a.R) {
            float x0, x1, x2, x3;
            f2_get(acc[2 * g], x0, x1);
            f2_get(acc[2 * g + 1], x2, x3);
            red_add_v4(out + 4 * g, x0, x1, x2, x3);
          }
        }
      }
      __syncwarp();
    }
  }

  end_of_cta(abort_flag, a.status);
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// How many runs the rows are cut into: the time of the busiest CTA, an item costing its rows and about two more (the
// bias tile in, the sum out).
inline WalkB walk_b(const Args& a, int sms) {
  const long long NT = (a.R + BT - 1) / BT, tiles = (long long)a.B * a.H * NT * NT;
  WalkB w{0, 1, a.S};
  long long best = 0;
  for (int runs = 1; runs <= a.S && runs <= 64; ++runs) {
    const int rows = (a.S + runs - 1) / runs, n = (a.S + rows - 1) / rows;  // (no empty run)
    const long long cost = (tiles * n + sms - 1) / sms * (rows + 2);
    if (tiles * n <= 0x7fffffffLL && (best == 0 || cost < best)) {
      best = cost;
      w = WalkB{(int)(tiles * n), n, rows};
    }
  }
  return w;
}

}  // namespace
}  // namespace evo
