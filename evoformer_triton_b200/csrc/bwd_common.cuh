// What the two forms of the fused backward kernel share (with a d(pair_bias): bwd_sm100.cu; without:
// bwd_nodbias.cuh): tiles, items and steps, the layout of tensor memory, the warps that issue S^T, dP^T, dV and dK,
// the mask, the arithmetic of a score, and the way of dK and dV to global memory.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"

namespace evo {
namespace {

using namespace ptx;

constexpr int BT = 128;   // tile edge (queries and keys)
constexpr int HT = 64;    // queries per half of a step (one warp group)
constexpr int QT = 32;    // queries per quarter of a step
// MSA rows per work item: each keeps a dK and a dV accumulator of DP columns in tensor memory for the
// whole item, next to 256 columns of score buffers and two dQ partials
template <int DP> struct RowsPerItem { static constexpr int G = (DP == 64) ? 1 : (DP == 32) ? 3 : 7; };
constexpr int kCW = 16;   // compute warps
constexpr int kThreadsT = 640;  // 16 compute + 4 service warps, five warps per scheduler
constexpr int kComputeRegs = 112, kServiceRegs = 32;  // after setmaxnreg; the launch-time pool must hold their sum
constexpr int kStages = 2;  // (three or four stages measured no faster: the loads are not what a step waits for)
constexpr float kLog2e = 1.4426950408889634f;
constexpr int BIAS_NONE = 0, BIAS_F32 = 1, BIAS_16 = 2;
// -lse*log2e of the queries of an MSA row whose keys are all dropped.  Its scores are constants: P is 1/N_res and dS 0
// whatever its Q, K, V and dO hold, which may be memory that was never written.  2^x of a finite score is 0 with it
// already; for the others each kernel says how.
constexpr float kDeadRow = -FLT_MAX;

template <int DP>
struct TilesT {
  static_assert(DP == 16 || DP == 32 || DP == 64, "padded head dimension");
  static_assert(kStages == 2, "steps alternate between two stages");
  static constexpr int G = RowsPerItem<DP>::G;
  static constexpr int RB = DP * 2;                          // bytes per staged row
  static constexpr int kTile = BT * RB;                      // one Q, dO, K or V tile
  static constexpr int kVec = BT * 4;                        // one vector of row statistics
  static constexpr int kStage = 2 * kTile + 2 * kVec;        // Q, dO, -lse*log2e, delta of one step
  static constexpr int kDS = BT * BT * 2;                    // dS^T: two halves of [128 keys][64 queries]
  // Tensor memory: two (S^T, dP^T) half-tile buffers, the per-row dV and dK accumulators, two dQ partials
  static constexpr int kTmemCols = 512;
  static constexpr int colS0 = 0, colDP0 = HT, colS1 = 2 * HT, colDP1 = 3 * HT;
  static constexpr int colDV = 4 * HT, colDK = colDV + G * DP, colDQ = colDK + G * DP;
  static_assert(colDQ + 2 * DP <= kTmemCols, "TMEM budget");
};

// An mbarrier named by its 32-bit shared-window address (8 bytes apart in the barrier array).
struct Bar {
  uint32_t a;
};
__device__ __forceinline__ Bar operator+(Bar b, int i) { return Bar{b.a + 8u * static_cast<uint32_t>(i)}; }
__device__ __forceinline__ void mbar_wait(Bar b, uint32_t parity, uint32_t abort_s, int code) {
  mbar_wait_s(b.a, parity, abort_s, code);
}
__device__ __forceinline__ void mbar_arrive(Bar b) { mbar_arrive_s(b.a); }
__device__ __forceinline__ void mbar_expect_tx(Bar b, uint32_t bytes) { mbar_expect_tx_s(b.a, bytes); }

struct StepT {
  int b, h, s, it, g, j0;
};
// Persistent CTAs: CTA c owns the items c, c + gridDim.x, ..., NT * G steps per item.  A short last
// row group (S % G != 0) is padded with rows >= S: their tiles and statistics arrive as zeros and
// their mask is -inf, so P = dS = 0, and nothing of them is stored.
// Key tiles are the fastest: the CTAs that work side by side share Q, dO and the dQ accumulator of the same rows, which
// come from DRAM once.  With row groups the fastest a large (b,h) came back for every key tile (four times the bytes
// at [1,512,768,2,64]; forward and backward of [1,512,768,8,32] 3 514 us, now 3 384, [2,512,768,8,64] 12 580, now
// 12 000).  Padded to sixteen columns a (b,h) is small, and there the shared bias tile is what counts:
// [1,1024,384,8,8] 1 475 us with row groups the fastest and 1 489 with key tiles, [1,1024,1024,8,8] 9 352 and 9 520.
template <int G>
struct Steps {
  int NT, NC, H;   // query (and key) tiles, row groups, heads
  int items, total;  // of this CTA
  __device__ __forceinline__ Steps(const Args& a, int n_items)
      : NT((a.R + BT - 1) / BT), NC((a.S + G - 1) / G), H(a.H),
        items((n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x), total(items * NT * G) {}
  __device__ __forceinline__ StepT decode(int N) const {
    StepT d;
    const int k = N / (NT * G), n = N - k * (NT * G);
    d.it = n / G;
    d.g = n - d.it * G;
    int idx = (int)blockIdx.x + k * (int)gridDim.x;
    int chunk = 0;
    if constexpr (G == 7) { chunk = idx % NC; idx /= NC; }
    d.j0 = (idx % NT) * BT; idx /= NT;
    if constexpr (G != 7) { chunk = idx % NC; idx /= NC; }
    d.h = idx % H;
    d.b = idx / H;
    d.s = chunk * G + d.g;
    return d;
  }
  // Position of step n = the one after c (no divisions inside an item).
  __device__ __forceinline__ StepT advance(const StepT& c, int n) const {
    StepT d = c;
    if (++d.g == G) {
      d.g = 0;
      if (++d.it == NT) return decode(n);
    }
    d.s = c.s - c.g + d.g;
    return d;
  }
};

// What the mask adds to a score of (b, s, key j) in the log2 domain: 0 keeps it, -inf drops it (a dropped score
// gives P = 0 exactly, as exp(-FLT_MAX - lse) does in evoformer.py:69,600).
template <class T>
__device__ __forceinline__ float mask_term(const Args& a, int b, int s, int j) {
  if (s >= a.S || j >= a.R) return -__int_as_float(0x7f800000);
  if (a.mask_kind == EVOATTN_MASK_NONE) return 0.f;
  const long long mi = (long long)b * a.smask.a + (long long)s * a.smask.b + (long long)j * a.smask.c;
  if (a.mask_kind == EVOATTN_MASK_BOOL) return reinterpret_cast<const unsigned char*>(a.mask)[mi] ? 0.f : -__int_as_float(0x7f800000);
  if (a.mask_kind == EVOATTN_MASK_ADD_F32) return reinterpret_cast<const float*>(a.mask)[mi] * kLog2e;
  return to_float<T>(reinterpret_cast<const T*>(a.mask)[mi]) * kLog2e;
}

// Tensor-core issuers: warp 16 (S^T, dV), warp 17 (dP^T, dK).
// Issuing a tcgen05.mma costs the issuing warp fifty cycles and more, so the 32 MMAs of a step
// are spread over three warps on three schedulers.  A thread's MMAs run in issue order, MMAs of
// different threads in no particular order, so the split follows the data: warp 16 owns the
// S^T columns of both buffers (S^T = K_j Q_i^T in, dV_j += P^T dO_i out), warp 17 the dP^T columns
// (dP^T = V_j dO_i^T in, dK_j += dS^T Q_i out): the MMA that overwrites a buffer is always issued
// by the thread that issued the MMAs reading it.  Warp 18 issues dQ_i = dS K_j, which depends on
// neither.  The warps walk their loops converged (see elect_one).
// The compute warps wait for S^T, dP^T and the statistics at once, and warp 16, which has seen these land, arrives on
// their barrier for them.
// With one row per item (G = 1) every item boundary would be a gap of a load and more: K and V have a barrier each
// (kv_full, kv_empty: [0] K, [1] V).  V is replaced as soon as the item's last dP^T is through, by load_v() of warp 17;
// K, which dQ reads too, by warp 18.  The outputs of an item's last step do not wait for the next K, and the compute
// warps read dK and dV meanwhile; `drained` lets the next item's first outputs overwrite them.
struct IssueBars {
  Bar kv_full, kv_empty, st_full, st_empty, sd_full, cdone, drained;
};
template <class T, int DP, class LoadV>
__device__ __forceinline__ void issue_scores_and_outputs(bool isA, uint32_t tmem, uint32_t sKV_s, uint32_t sStage_s, int NT,
                                                         int total_steps, const IssueBars& bar, uint32_t abort_s, LoadV load_v) {
  using L = TilesT<DP>;
  constexpr int G = L::G, RB = L::RB;
  constexpr uint32_t SWZ = swizzle_code_for_row_bytes(RB);
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  constexpr uint32_t kIdescSD = make_idesc(kBf16, false, false, BT, HT);   // S^T, dP^T: K-major operands, N = 64
  constexpr uint32_t kIdescOut = make_idesc(kBf16, false, true, BT, DP);   // dV, dK: A from TMEM, B MN-major
  constexpr uint32_t kHiOp = static_cast<uint32_t>(make_sdesc_const(16, 8 * RB, SWZ) >> 32);
  constexpr uint32_t kLoLbo = static_cast<uint32_t>(make_sdesc_const(16, 0, 0) & 0xffffffffu);
  constexpr uint32_t kRowBlk = (16 * RB) >> 4;  // 16 tile rows, in descriptor address units
  // warp 16 reads K (A operand) and Q (B), then dO (B of dV); warp 17 reads V and dO, then Q (B of dK)
  const uint32_t kv_lo = (sKV_s >> 4) + (isA ? 0 : (L::kTile >> 4));
  const uint32_t in_lo = (sStage_s >> 4) + (isA ? 0 : (L::kTile >> 4));
  const uint32_t out_lo = (sStage_s >> 4) + (isA ? (L::kTile >> 4) : 0);
  const uint32_t col_in0 = isA ? L::colS0 : L::colDP0, col_in1 = isA ? L::colS1 : L::colDP1;
  const uint32_t col_acc = isA ? L::colDV : L::colDK;

  // Position of a step inside this CTA's list, advanced without divisions: row g of the group,
  // query tile it, ring stage and the parities of the stage ring and of the item.
  struct Pos { int g, it; uint32_t stg, ring_par, item_par; };
  auto after = [&](Pos p) {
    if (++p.g == G) { p.g = 0; if (++p.it == NT) { p.it = 0; p.item_par ^= 1u; } }
    if (++p.stg == (uint32_t)kStages) { p.stg = 0; p.ring_par ^= 1u; }
    return p;
  };
  // Everything an MMA group needs is computed before the wait it follows: this thread shares its
  // scheduler with four arithmetic warps, so every instruction between the wake-up and the MMA is
  // paid several times over, and it sits on the critical path of the half that waits for it.
  auto issue_in = [&](const Pos& p, uint32_t ka, uint32_t qb, int h) {
    // (the second commit: the item's last read of this warp's K or V tile of row g)
    const uint32_t bar2 = (h == 1 && p.it == NT - 1 && !(G == 1 && isA)) ? (bar.kv_empty + (G == 1 ? 1 : p.g)).a : 0u;
    const uint32_t tD = tmem + (h ? col_in1 : col_in0), qa = qb + h * HT * (RB >> 4);
    const uint32_t el = elect_one();
#pragma unroll
    for (int kk = 0; kk < DP / 16; ++kk)
      mma_ss_e(el, tD, pack_desc(ka + 2 * kk, kHiOp), pack_desc(qa + 2 * kk, kHiOp), kIdescSD, kk > 0 ? 1u : 0u);
    mma_commit_if_s(el, (bar.sd_full + 2 * h).a);
    if (bar2) mma_commit_if_s(el, bar2);
    if (isA) {
      if (el) mbar_arrive(bar.sd_full + 2 * h);
      __syncwarp();
    }
    if (G == 1 && !isA && bar2) load_v();
  };
  Pos cur{0, 0, 0u, 0u, 0u};
  if (total_steps > 0) {
    mbar_wait(bar.st_full + 0, 0, abort_s, DEV_TIMEOUT_TMA);
    mbar_wait(bar.kv_full + (G == 1 && !isA ? 1 : 0), 0, abort_s, DEV_TIMEOUT_TMA);
    tc_fence_after();
    const uint32_t ka = (kv_lo + 0) | kLoLbo, qb = in_lo | kLoLbo;
    issue_in(cur, ka, qb, 0);
    issue_in(cur, ka, qb, 1);
  }
#pragma unroll 1
  for (int n = 0; n < total_steps; ++n) {
    const Pos nxt = after(cur);
    const bool more = n + 1 < total_steps;
    // this step: dV_j[g] += P^T dO_i (warp 16) or dK_j[g] += dS^T Q_i (warp 17);
    // A = 16 queries of P^T / dS^T (8 packed TMEM columns), B = their dO / Q rows
    const uint32_t acc = tmem + col_acc + cur.g * DP;
    const uint32_t ob = (out_lo + cur.stg * (L::kStage >> 4)) | kLoLbo;
    const uint32_t first0 = (cur.it == 0) ? 0u : 1u;  // the item's first MMA of row g overwrites
    const uint32_t st_empty_bar = (bar.st_empty + (int)cur.stg).a;
    // next step: S^T = K_j Q_i^T (warp 16) or dP^T = V_j dO_i^T (warp 17) into the buffer just read
    const uint32_t ka = (kv_lo + (2 * nxt.g) * (L::kTile >> 4)) | kLoLbo;
    const uint32_t qb = (in_lo + nxt.stg * (L::kStage >> 4)) | kLoLbo;
    const uint32_t st_full_bar = (bar.st_full + (int)nxt.stg).a, kv_full_bar = (bar.kv_full + (G == 1 ? (isA ? 0 : 1) : nxt.g)).a;
    auto outputs = [&](int h) {
      mbar_wait(bar.cdone + 2 * h, n & 1, abort_s, DEV_TIMEOUT_SYNC);
      if (G == 1 && h == 0 && cur.it == 0 && n > 0) mbar_wait(bar.drained, cur.item_par ^ 1u, abort_s, DEV_TIMEOUT_SYNC);
      tc_fence_after();
      const uint32_t tA = tmem + (h ? col_in1 : col_in0);
      const uint32_t el = elect_one();
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        mma_ts_e(el, acc, tA + 16 * kk, pack_desc(ob + (4 * h + kk) * kRowBlk, kHiOp), kIdescOut, h == 0 && kk == 0 ? first0 : 1u);
      if (h == 1) mma_commit_if_s(el, st_empty_bar);
    };
    auto inputs = [&](int h) {
      if (!more) return;
      if (h == 0 && nxt.it == 0) {
        mbar_wait_s(kv_full_bar, nxt.item_par, abort_s, DEV_TIMEOUT_TMA);
        tc_fence_after();
      }
      issue_in(nxt, ka, qb, h);
    };
    // (the next step's tiles are long there as a rule: waited for here, where nobody waits for this warp)
    if (more) mbar_wait_s(st_full_bar, nxt.ring_par, abort_s, DEV_TIMEOUT_TMA);
    outputs(0);
    if (G == 1 && nxt.it == 0) {
      outputs(1);
      inputs(0);
    } else {
      inputs(0);
      outputs(1);
    }
    inputs(1);
    cur = nxt;
  }
}

// dQ_i partial = dS K_j of a step: A = the dS^T tile [key][query] read MN-major (M = query), K runs over the keys.
// One warp, converged; returns the elected lane for the commits.
template <class T, int DP>
__device__ __forceinline__ uint32_t issue_dq(uint32_t d_tmem, uint32_t sDS_s, uint32_t k_tile_s) {
  constexpr int RB = TilesT<DP>::RB;
  constexpr uint32_t SWZ = swizzle_code_for_row_bytes(RB);
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  constexpr uint32_t kIdescDQ = make_idesc(kBf16, true, true, BT, DP);     // A = dS^T read MN-major, B = K MN-major
  constexpr uint32_t kHiOp = static_cast<uint32_t>(make_sdesc_const(16, 8 * RB, SWZ) >> 32);
  constexpr uint32_t kHiDS = static_cast<uint32_t>(make_sdesc_const(16, 1024, SWZ_128B) >> 32);
  constexpr uint32_t kLoLbo = static_cast<uint32_t>(make_sdesc_const(16, 0, 0) & 0xffffffffu);
  constexpr uint32_t kLoLboDS = static_cast<uint32_t>(make_sdesc_const(BT * 128, 0, 0) & 0xffffffffu);
  constexpr uint32_t kRowBlk = (16 * RB) >> 4;
  const uint32_t ka = (k_tile_s >> 4) | kLoLbo, ds = (sDS_s >> 4) | kLoLboDS;
  const uint32_t el = elect_one();
#pragma unroll
  for (int kk = 0; kk < 8; ++kk)
    mma_ss_e(el, d_tmem, pack_desc(ds + 128 * kk, kHiDS), pack_desc(ka + kk * kRowBlk, kHiOp), kIdescDQ, kk > 0 ? 1u : 0u);
  return el;
}

// A pair-bias value of a staged tile, widened.
template <class T, bool BIAS16>
__device__ __forceinline__ float staged_bias(uint32_t at) {
  if constexpr (BIAS16) {
    const uint16_t raw = lds_u16(at);
    return to_float<T>(*reinterpret_cast<const T*>(&raw));
  } else {
    return lds_f32(at);
  }
}

// P^T and dS^T of a key and 16 queries, packed, from S^T and dP^T: x = S*(scale*log2e) + (bias*log2e - lse*log2e) +
// mask, P = 2^x, dS = P (dP - delta), two queries per instruction (the pairs lie side by side in every operand).
// vnl, vdl: the queries' statistics; bias_at(e): the bias value of query e; take(e, dS): the dS of pair e.
template <class T, bool HAS_BIAS, class BiasAt, class Take>
__device__ __forceinline__ void score_chunk(const uint32_t (&sr)[16], const uint32_t (&dr)[16], uint32_t vnl, uint32_t vdl,
                                            BiasAt bias_at, F2 c12, F2 mj2, uint32_t (&pk)[8], uint32_t* dk, Take take) {
  const F2 l2e2 = f2_make(kLog2e, kLog2e);
#pragma unroll
  for (int c4 = 0; c4 < 4; ++c4) {
    const float4 nl = lds_v4f(vnl + 16 * c4);
    const float4 dl = lds_v4f(vdl + 16 * c4);
    F2 t[2] = {f2_make(nl.x, nl.y), f2_make(nl.z, nl.w)};
    const F2 de[2] = {f2_make(dl.x, dl.y), f2_make(dl.z, dl.w)};
    if constexpr (HAS_BIAS) {
      float bv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) bv[u] = bias_at(4 * c4 + u);
      t[0] = f2_fma(f2_make(bv[0], bv[1]), l2e2, t[0]);
      t[1] = f2_fma(f2_make(bv[2], bv[3]), l2e2, t[1]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = 4 * c4 + 2 * u;
      float x0, x1;
      f2_get(f2_add(f2_fma(f2_from_bits(sr[e], sr[e + 1]), c12, t[u]), mj2), x0, x1);
      const float p0 = ex2(x0), p1 = ex2(x1);
      const F2 ds = f2_mul(f2_make(p0, p1), f2_add(f2_from_bits(dr[e], dr[e + 1]), de[u]));
      take(e / 2, ds);
      float d0, d1;
      f2_get(ds, d0, d1);
      pk[2 * c4 + u] = Pack2<T>::pack(p0, p1);
      dk[2 * c4 + u] = Pack2<T>::pack(d0, d1);
    }
  }
}

// dK, dV of row-group slot g (MSA row s of (b,h), keys j0..): TMEM -> registers -> global.  For the kernel without a
// d(pair_bias) up to DP = 32: with an fp32 bias its shared memory is full, so that nothing can be staged for bulk stores.
// Done by the warps of half 0 (half of the DP columns each, 16 at a time): they are the ones
// whose arrival lets the next item's first MMAs overwrite the slot.
template <class T, int DP>
__device__ __forceinline__ void drain_dkdv(const Args& a, uint32_t t_lane, int cb2, int jrow, int b, int h, int s, int j0, int g) {
  using L = TilesT<DP>;
  const float scale = a.scale;
  const int j = j0 + jrow;
  constexpr int W = DP == 16 ? 8 : 16;  // columns at a time
#pragma unroll
  for (int part = 0; part < DP / 2 / W; ++part) {
    const int c0 = cb2 * (DP / 2) + part * W;
    uint32_t kr[W], vr[W];
    tmem_ld<W>(t_lane + L::colDK + g * DP + c0, kr);
    tmem_ld<W>(t_lane + L::colDV + g * DP + c0, vr);
    tmem_wait_ld();
    if (j < a.R && s < a.S) {
      T* kd = reinterpret_cast<T*>(a.dk) + off4(a.sdk, b, h, s, j) + c0;
      T* vd = reinterpret_cast<T*>(a.dv) + off4(a.sdv, b, h, s, j) + c0;
#pragma unroll
      for (int d8 = 0; d8 < W / 8; ++d8) {
        if (c0 + d8 * 8 < a.D) {
          uint4 pk, pv;
          pk.x = Pack2<T>::pack(__uint_as_float(kr[d8 * 8 + 0]) * scale, __uint_as_float(kr[d8 * 8 + 1]) * scale);
          pk.y = Pack2<T>::pack(__uint_as_float(kr[d8 * 8 + 2]) * scale, __uint_as_float(kr[d8 * 8 + 3]) * scale);
          pk.z = Pack2<T>::pack(__uint_as_float(kr[d8 * 8 + 4]) * scale, __uint_as_float(kr[d8 * 8 + 5]) * scale);
          pk.w = Pack2<T>::pack(__uint_as_float(kr[d8 * 8 + 6]) * scale, __uint_as_float(kr[d8 * 8 + 7]) * scale);
          pv.x = Pack2<T>::pack(__uint_as_float(vr[d8 * 8 + 0]), __uint_as_float(vr[d8 * 8 + 1]));
          pv.y = Pack2<T>::pack(__uint_as_float(vr[d8 * 8 + 2]), __uint_as_float(vr[d8 * 8 + 3]));
          pv.z = Pack2<T>::pack(__uint_as_float(vr[d8 * 8 + 4]), __uint_as_float(vr[d8 * 8 + 5]));
          pv.w = Pack2<T>::pack(__uint_as_float(vr[d8 * 8 + 6]), __uint_as_float(vr[d8 * 8 + 7]));
          *reinterpret_cast<uint4*>(kd + d8 * 8) = pk;
          *reinterpret_cast<uint4*>(vd + d8 * 8) = pv;
        }
      }
    }
  }
}

// The same with one row per item, where all sixteen warps do it: 32 columns of dK (half 0) or dV (half 1) each, to the
// swizzled tile at dst, which leaves by one bulk store.  (Sixteen bytes a lane straight to global memory, 32 rows an
// instruction, took 3 800 cycles at every item boundary.)
template <class T>
__device__ __forceinline__ void stage_dk_or_dv(uint32_t t_src, uint32_t dst, float f, int jrow, int cb2) {
  uint32_t r[32];
  tmem_ld32(t_src, r);
  tmem_wait_ld();
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) w[u] = Pack2<T>::pack(__uint_as_float(r[8 * c + 2 * u]) * f, __uint_as_float(r[8 * c + 2 * u + 1]) * f);
    sts_v4(dst + jrow * 128 + (((4 * cb2 + c) ^ (jrow & 7)) << 4), w[0], w[1], w[2], w[3]);
  }
}

}  // namespace
}  // namespace evo
