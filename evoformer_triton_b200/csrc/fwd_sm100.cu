// Evoformer attention forward for sm_100a: TMA-staged tiles, tcgen05 MMAs with the
// accumulators in TMEM, online softmax with pair bias and residue mask in registers.
//
// Computes what dsevoformer-triton/evoformer.py:23-100 (_attn_fwd_inner) and :103-297
// (_attn_fwd) compute:  O = softmax(scale*Q K^T + bias, masked) V  and the row
// log-sum-exp, without ever writing the R x R scores to memory.
//
// Persistent, warp-specialised kernel, one CTA per SM, NW = 2, 3 or 4 softmax warpgroups:
//   warp 0      TMA producer: Q tiles, K/V tiles (64 keys each) and pair-bias tiles
//   warp 1, 2   issue the tcgen05.mma of half of the warpgroups each
//   warp 3      stages the residue-mask rows of the next item in shared memory
//   warps 4..   softmax warpgroups
// A work item is one 128-row query tile of NW consecutive MSA rows s of one (b,h), one row for each
// warpgroup.  All of them use the same pair-bias tile, which is staged in shared memory once.  Inside a
// warpgroup thread t owns score row t (= TMEM lane t) and all 64 columns of the current key tile, so the row
// sum needs no exchange between threads.
//
// With a single MSA row (N_seq = 1, the shape of the reference's own benchmark sweep) there is no
// second row to pair: the kernel is then instantiated in query-pair mode, where an item is two
// consecutive query tiles of the same row, the warpgroups share the K/V tiles and each has its own
// pair-bias tile in a stage.
//
// Per warpgroup and key tile n:  S_n = Q K_n^T lands in TMEM; the warpgroup turns it into P_n (rounded to
// the storage type as evoformer.py:84 does) and writes it back over S_n in TMEM, from where it feeds the P V
// MMA as the A operand; O accumulates in TMEM over the item.  With two warpgroups S is double buffered; with
// three or four (152 and 112 registers a thread) it is not, and the other warpgroups hide the hand-over.
//
// The exponentials of a tile do not wait for its maximum: they are taken against the running maximum m of the
// tiles before (of the first tile, its own), straight from the scores: load, two FMAs, ex2, row sum, pack.  Only
// if a row's sum of the tile shows that some exp2(x - m) may be too large (its sum is) is the tile's maximum
// taken, m and O follow it, and the tile is done again.  So the maximum pass costs one tile in T_TILES instead of
// every one, and no score is held in a register.  Where the scores rise from tile to tile by more than m may lag
// (Lag), the next tile's maximum is taken first, and its exponentials only once.
//
// Bound by the issue slots and hand-overs around the exponentials (16 a cycle and SM: [1,256,1024,4,32] would
// take 236 us).  That shape takes 378 us with four warpgroups, and 540 with the form before, which had the
// maximum in line, two warpgroups taking turns, one TMA copy per row and MMAs issued from a single-lane branch;
// [1,128,384,8,32] 97 -> 77, [1,1024,384,8,8] fp16 703 -> 505, [1,128,768,8,64] 349 -> 295 us.
#include <type_traits>

#include "common.cuh"
#include "launch.h"
#include "ptx.cuh"
#include "tmap.h"

namespace evo {
namespace {

using namespace ptx;

constexpr int BM = 128;  // query rows per warpgroup tile
constexpr int BN = 64;   // keys per tile
constexpr int kTmemCols = 512;
constexpr size_t kMaxSmem = 232448;  // of one CTA
constexpr int kMaxRes = 2048;        // longest N_res: two mask rows for each warpgroup are staged in shared memory
constexpr float kLog2e = 1.4426950408889634f;
// How far the running maximum may lag.  kMaxSum: sum of a tile's exponentials up to which they serve; kRise: rise of a
// tile's maximum above the running one up to which the sum of its 64 cannot be more.  fp16 ends at 2^16; bf16 and the
// fp32 sums do not care how large P is (2^84 is left for the values of V).  A line at 2^8, with a maximum that followed
// only where it had grown by that much, made every tile after a moderate rise pay for both passes.  Forward, us, with
// that, with the line here, and of the kernel that took every tile's maximum; a bias that rises along the keys by
// 8 bits / by 64 bits / by 7 bits once: [1,128,768,8,32] bf16 373 / 469 / 467, 227 / 262 / 226, 317 / 345 / 343;
// [1,64,768,8,64] bf16 265 / 330 / 325, 168 / 189 / 168, 193 / 208 / 208 (fp16, which may lag less: 260 at 64 bits).
template <class T> struct Lag;
template <> struct Lag<__half> { static constexpr float kMaxSum = 32768.f, kRise = 9.f / kLog2e; };
template <> struct Lag<__nv_bfloat16> { static constexpr float kMaxSum = 4294967296.f, kRise = 26.f / kLog2e; };
constexpr float kFar = 65536.f;        // running maximum up to which an exponent is formed in one FMA (see far_tile)
constexpr int MASK_MIN = 0;  // boolean keep-mask (or none): score = min(score, m), m = +-FLT_MAX
constexpr int MASK_ADD = 1;  // additive mask
constexpr int BIAS_NONE = 0, BIAS_F32 = 1, BIAS_16 = 2;

// NW softmax warpgroups per CTA, each with a query tile of one MSA row at a time.  QP: query-pair mode.
template <int DP, int NW, bool QP, int BIAS>
struct Cfg {
  static_assert(!QP || NW == 2, "query-pair mode has two warpgroups");
  static constexpr int RB = DP * 2;                    // bytes per staged row
  static constexpr int QST = (DP == 64 || NW > 2) ? 1 : 2;  // Q stages
  static constexpr int SB = NW > 2 ? 1 : 2;            // score buffers per warpgroup
  // Query pairs with an fp32 bias: a stage of V and the bias is 64 KB and more, so there are two of them, and at
  // DP = 64 two of K, which leaves room for the masks of every length.  Bound by reading the bias (332 us of it at
  // 2 048).  Forward of [4,1,R,32,D] bf16, us, as query pairs and as items of two rows, the second of which does not
  // exist: R = 2048, D = 8 343 and 426, D = 32 354 and 447, D = 64 376 and 538; R = 300, D = 8 18.5 and 22.6, D = 32
  // 20.6 and 22.6.  (At D = 64 up to 1 472 query pairs fitted with three stages of K as well: 24 and 114 either way.)
  static constexpr bool kWide = QP && BIAS == BIAS_F32;
  static constexpr int NK = DP == 64 && NW > 2 ? 1 : DP == 64 && kWide ? 2 : SB + 1;  // K stages (S is through with one early in a tile)
  static constexpr int NV = (DP == 64 || NW > 2 || kWide) ? 2 : 3;  // stages of V and the pair bias
  static constexpr int KVR = QP ? 1 : NW;              // rows of K and V in a stage: one per warpgroup, or one shared
  static constexpr int BTL = QP ? 2 : 1;               // pair-bias tiles in a stage: one shared, or one per warpgroup
  static constexpr int kThreads = 128 + 128 * NW;
  static constexpr int kServiceRegs = NW == 2 ? 40 : NW == 3 ? 56 : 32, kSoftmaxRegs = NW == 2 ? 232 : NW == 3 ? 152 : 112;
  static constexpr int kQ = BM * RB;
  static constexpr int kKV = BN * RB;
  static constexpr int kBias = BIAS == BIAS_NONE ? 0 : BM * BN * (BIAS == BIAS_16 ? 2 : 4);  // one tile; fp32: two 128x32 boxes
  static constexpr int kVB = KVR * kKV + BTL * kBias;  // a stage: V, then the bias
  static constexpr int kOnes = 16 * RB;                // 16 keys by DP columns of ones
  static constexpr int offQ = 0;
  static constexpr int offK = offQ + NW * QST * kQ;
  static constexpr int offV = offK + NK * KVR * kKV;
  static constexpr int offOnes = offV + NV * kVB;
  static constexpr int offMask = offOnes + (kOnes < 1024 ? 1024 : kOnes);
  static constexpr int PER = 3 * SB + 4;               // barriers of a warpgroup
  static constexpr int kNumBars = NW * PER + 2 * (QST + NK + NV);
  // Slack for aligning the tiles to 1024 bytes; where it does not fit the kernel checks that the base address
  // needs none (the dynamic shared memory of a kernel without static shared memory starts on such a boundary on
  // this architecture) and gives up with a status code otherwise.
  static constexpr int kSlack = DP == 64 && kWide ? 0 : 1024;
  static constexpr size_t bytes(int r_pad) {
    return (size_t)offMask + (size_t)2 * NW * (r_pad * 4 + 4) + kNumBars * 8 + 64 + kSlack;
  }
  static_assert(!QP || bytes(kMaxRes) <= kMaxSmem, "query-pair mode is there for every length");
  // TMEM columns of a warpgroup: S buffers, then O, then the row sum of P (16 equal columns)
  static constexpr int colO = SB * BN, colL = colO + DP, tmemWg = colL + 16;
  static_assert(NW * tmemWg <= kTmemCols, "TMEM budget");
  static_assert(offK % 1024 == 0 && offV % 1024 == 0 && kVB % 1024 == 0 && offOnes % 1024 == 0, "swizzled tiles");
};

// n / d by a multiplication, exact for n < 2^31: m = ceil(2^(31 + s) / d), s = ceil(log2 d).
struct FastDiv {
  uint32_t m, s, d;
};
FastDiv fast_div(uint32_t d) {
  uint32_t s = 0;
  while ((1ull << s) < d) ++s;
  return FastDiv{static_cast<uint32_t>(((1ull << (31 + s)) + d - 1) / d), 31 + s, d};
}
__device__ __forceinline__ uint32_t div_mod(uint32_t n, const FastDiv& f, uint32_t& rem) {
  const uint32_t q = static_cast<uint32_t>((static_cast<unsigned long long>(n) * f.m) >> f.s);
  rem = n - q * f.d;
  return q;
}
// Work items (b, h, inner, outer) in one of two orders (see rows_first).  Row mode: warpgroup w works on MSA row
// NW * inner + w, query tile `outer`.  Query-pair mode: on row `inner`, query tile 2 * outer + w.
struct Walk {
  int n_items;
  bool rows_first;               // inner is the fastest, else outer
  FastDiv first, second, heads;  // (the fastest and the other one)
};
struct Item {
  uint32_t b, h, outer, inner;
};
// (Two selects: query tiles fastest without a choice is 1 % faster at D = 64; a branch, or divisions by strides, 1 % slower.)
__device__ __forceinline__ Item decode_item(int idx, const Walk& wk) {
  Item it;
  uint32_t fast, slow;
  uint32_t n = div_mod(static_cast<uint32_t>(idx), wk.first, fast);
  n = div_mod(n, wk.second, slow);
  it.outer = wk.rows_first ? slow : fast;
  it.inner = wk.rows_first ? fast : slow;
  it.b = div_mod(n, wk.heads, it.h);
  return it;
}

// Eight scores of query row `row`, the g8-th eight of a key tile: x = scale*S + bias, then the mask.
template <class T, int MASKMODE, int BIAS, int BOXES, bool MASKED>
__device__ __forceinline__ void row_scores8(const uint32_t* s8, int g8, int row, F2 scale2, uint32_t brow_s, uint32_t mtile_s,
                                            float (&v)[8]) {
  float bvv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, mkv[8];
  if constexpr (BIAS == BIAS_16) {
    // eight 16-bit values of my row (rows of 128 bytes, 128-byte swizzle), widened here
    const uint4 wv = lds_v4(brow_s + ((g8 ^ (row & 7)) << 4));
    unpack2<T>(wv.x, bvv[0], bvv[1]); unpack2<T>(wv.y, bvv[2], bvv[3]);
    unpack2<T>(wv.z, bvv[4], bvv[5]); unpack2<T>(wv.w, bvv[6], bvv[7]);
  } else if constexpr (BIAS == BIAS_F32) {  // (two boxes of 32 columns, BOXES bytes apart)
    const int c = g8 >> 2, q4 = (g8 & 3) * 2;
    const float4 b0 = lds_v4f(brow_s + c * BOXES + ((q4 ^ (row & 7)) << 4));
    const float4 b1 = lds_v4f(brow_s + c * BOXES + (((q4 + 1) ^ (row & 7)) << 4));
    bvv[0] = b0.x; bvv[1] = b0.y; bvv[2] = b0.z; bvv[3] = b0.w;
    bvv[4] = b1.x; bvv[5] = b1.y; bvv[6] = b1.z; bvv[7] = b1.w;
  }
  if constexpr (MASKED) {
    const float4 k0 = lds_v4f(mtile_s + g8 * 32);
    const float4 k1 = lds_v4f(mtile_s + g8 * 32 + 16);
    mkv[0] = k0.x; mkv[1] = k0.y; mkv[2] = k0.z; mkv[3] = k0.w;
    mkv[4] = k1.x; mkv[5] = k1.y; mkv[6] = k1.z; mkv[7] = k1.w;
  }
#pragma unroll
  for (int u = 0; u < 8; u += 2) {  // two elements per instruction
    F2 x = f2_fma(f2_from_bits(s8[u], s8[u + 1]), scale2, f2_make(bvv[u], bvv[u + 1]));
    if constexpr (MASKED && MASKMODE == MASK_ADD) x = f2_add(x, f2_make(mkv[u], mkv[u + 1]));
    f2_get(x, v[u], v[u + 1]);
  }
  if constexpr (MASKED && MASKMODE == MASK_MIN) {
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = fminf(v[u], mkv[u]);
  }
}

// P of a key tile against a maximum m beyond kFar.  (x - m) log2 e in one FMA carries the rounding of m log2 e, half a
// unit in its last place: 2^-8 at kFar, but 64 at 1e9, where all scores of a query lie whose bias drops it whole; its
// probabilities came out at 2^18 (infinite in fp16) or at 0.  Here the difference is formed first.  (So it is in the
// key tiles that an additive mask changes, where the packed instruction more is the one that a packed mask saves.)
// Sixteen keys at a time and straight into place: P_n lies over columns of S_n that have been read.  Returns the row
// sum.  Not inlined, which leaves the registers of the tile loop as they are; inlined, the forward of
// [1,128,768,8,64] took 314 us instead of 306, of [1,128,384,8,32] without a bias 74 instead of 72.
template <class T, int BIAS, int BOXES>
__device__ __noinline__ float far_tile(uint32_t tS, float m, int row, float scale, uint32_t brow_s, uint32_t mtile_s) {
  const F2 scale2 = f2_make(scale, scale);
  float sum = 0.f;
#pragma unroll 1
  for (int h = 0; h < BN / 16; ++h) {
    uint32_t s16[16], p8[8];
    tmem_ld16(tS + 16 * h, s16);
    tmem_wait_ld();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      float v[8];
      row_scores8<T, MASK_MIN, BIAS, BOXES, true>(s16 + 8 * k, 2 * h + k, row, scale2, brow_s, mtile_s, v);
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        const float p0 = ex2((v[u] - m) * kLog2e), p1 = ex2((v[u + 1] - m) * kLog2e);
        sum += p0 + p1;
        p8[4 * k + u / 2] = Pack2<T>::pack(p0, p1);
      }
    }
    tmem_st8(tS + 8 * h, p8);
  }
  return sum;
}

template <class T, int DP, int MASKMODE, int BIAS, int NW, bool QP>
__global__ void __launch_bounds__(Cfg<DP, NW, QP, BIAS>::kThreads, 1)
evo_fwd_sm100_kernel(const Args a, const Walk wk, const __grid_constant__ CUtensorMap tmQ,
                     const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     const __grid_constant__ CUtensorMap tmB) {
  using C = Cfg<DP, NW, QP, BIAS>;
  constexpr int RB = C::RB, QST = C::QST, NK = C::NK, NV = C::NV, SB = C::SB;
  constexpr uint32_t SWZ = swizzle_code_for_row_bytes(RB);
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (static_cast<int>(smem - smem_raw) > C::kSlack) {  // the same for every thread of every CTA
    if (threadIdx.x == 0 && a.status) atomicCAS(a.status, 0, DEV_TIMEOUT_SYNC);
    return;
  }
  const uint32_t smem_s = smem_u32(smem);
  const int T_TILES = (a.R + BN - 1) / BN;
  const int r_pad = T_TILES * BN;
  float* sMask = reinterpret_cast<float*>(smem + C::offMask);  // [warpgroup][stage][r_pad]
  // one bit per key tile of a staged mask row (R <= 2048): the tile has a key that the mask changes
  uint32_t* sDirty = reinterpret_cast<uint32_t*>(sMask + 2 * NW * r_pad);  // [warpgroup][stage]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDirty + 2 * NW);
  const uint32_t bars_s = smem_u32(bars);
  // barriers: a block of PER for each warpgroup, then those of the rings
  // With two score buffers there are two of each of these for tiles in turn: the softmax warps may finish a
  // tile while the issuer still waits for the V of the one before, and a single barrier that is two phases on
  // looks the same as one that has not moved (a parity wait cannot tell).
  auto s_full = [&](int w, uint32_t i) { return bars_s + 8 * (w * C::PER + i); };
  auto p_full = [&](int w, uint32_t i) { return bars_s + 8 * (w * C::PER + SB + i); };
  auto o_full = [&](int w, uint32_t i) { return bars_s + 8 * (w * C::PER + 2 * SB + i); };
  auto m_full = [&](int w, int st) { return bars_s + 8 * (w * C::PER + 3 * SB + st); };
  auto m_empty = [&](int w, int st) { return bars_s + 8 * (w * C::PER + 3 * SB + 2 + st); };
  const uint32_t rings = bars_s + 8 * (NW * C::PER);
  auto q_full = [&](uint32_t st) { return rings + 8 * st; };
  auto q_empty = [&](uint32_t st) { return rings + 8 * (QST + st); };
  auto k_full = [&](uint32_t st) { return rings + 8 * (2 * QST + st); };
  auto k_empty = [&](uint32_t st) { return rings + 8 * (2 * QST + NK + st); };
  auto v_full = [&](uint32_t st) { return rings + 8 * (2 * (QST + NK) + st); };  // V and the pair bias
  auto v_empty = [&](uint32_t st) { return rings + 8 * (2 * (QST + NK) + NV + st); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + C::kNumBars + 1);
  const uint32_t abort_s = smem_u32(const_cast<int*>(abort_flag));

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform, and known to be)
  const int NQT = (a.R + BM - 1) / BM;
  // MSA row and query tile of warpgroup w (either may lie beyond the last one)
  auto row_of = [&](const Item& it, int w) { return (int)it.inner * (QP ? 1 : NW) + (QP ? 0 : w); };
  auto tile_of = [&](const Item& it, int w) { return (int)it.outer * (QP ? NW : 1) + (QP ? w : 0); };
  constexpr bool has_bias = BIAS != BIAS_NONE, BIAS16 = BIAS == BIAS_16;

  // A launch that follows a failed one returns at once (one reader, so the CTA agrees).
  grid_dependency_wait();
  grid_launch_dependents();
  if (tid == 0) *abort_flag = (a.status && *reinterpret_cast<volatile int*>(a.status) != 0) ? 1 : 0;
  __syncthreads();
  if (*abort_flag) return;

  if (tid == 0) {
#pragma unroll 1
    for (int w = 0; w < NW; ++w) {
      for (int i = 0; i < SB; ++i) {
        mbar_init_s(s_full(w, i), has_bias && SB == 1 ? 2 : 1);  // the MMA, and the bias tile (below)
        mbar_init_s(p_full(w, i), 4);  // one arrival per softmax warp
        mbar_init_s(o_full(w, i), 1);
      }
      for (int st = 0; st < 2; ++st) { mbar_init_s(m_full(w, st), 1); mbar_init_s(m_empty(w, st), 4); }
    }
    // (every warpgroup's issuer releases the stages that they share)
    for (int st = 0; st < QST; ++st) { mbar_init_s(q_full(st), 1); mbar_init_s(q_empty(st), NW); }
    for (int st = 0; st < NK; ++st) { mbar_init_s(k_full(st), 1); mbar_init_s(k_empty(st), NW); }
    for (int st = 0; st < NV; ++st) { mbar_init_s(v_full(st), 1); mbar_init_s(v_empty(st), NW); }
    fence_mbar_init();
    prefetch_tmap(&tmQ); prefetch_tmap(&tmK); prefetch_tmap(&tmV);
    if (has_bias) prefetch_tmap(&tmB);
  }
  if (tid < C::kOnes / 4) reinterpret_cast<uint32_t*>(smem + C::offOnes)[tid] = Pack2<T>::pack(1.f, 1.f);
  if (C::kOnes / 4 > C::kThreads && tid + C::kThreads < C::kOnes / 4)
    reinterpret_cast<uint32_t*>(smem + C::offOnes)[tid + C::kThreads] = Pack2<T>::pack(1.f, 1.f);
  fence_async_shared();
  if (warp == 0) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp < 4) {
    setmaxnreg_dec<C::kServiceRegs>();
    if (warp == 0) {
      // =============================== TMA producer ===============================
      // Few copies per tile (K, V of all rows and the bias: three or four), since issuing one, with its wait,
      // costs hundreds of cycles: with a copy per row this warp set the pace of the kernel.
      uint32_t n_item = 0, kt = 0, kp = 1, vt = 0, vp = 1;  // items; stage and parity of the rings
#pragma unroll 1
      for (int item = blockIdx.x; item < wk.n_items; item += gridDim.x, ++n_item) {
        const Item it = decode_item(item, wk);
        const int s0 = row_of(it, 0), i0 = tile_of(it, 0) * BM;  // (rows and query tiles beyond the last load as zeros)
        const uint32_t qs = n_item % QST;
        mbar_wait_s(q_empty(qs), ((n_item / QST) & 1) ^ 1, abort_s, DEV_TIMEOUT_SYNC);
        if (elect_one()) {
          mbar_expect_tx_s(q_full(qs), NW * C::kQ);
          tma_load_5d_s(smem_s + C::offQ + qs * (NW * C::kQ), &tmQ, q_full(qs), 0, i0, s0, it.h, it.b);
        }
        __syncwarp();
#pragma unroll 1
        for (int j0 = 0; j0 < r_pad; j0 += BN) {
          mbar_wait_s(k_empty(kt), kp, abort_s, DEV_TIMEOUT_SYNC);
          if (elect_one()) {
            mbar_expect_tx_s(k_full(kt), C::KVR * C::kKV);
            tma_load_5d_s(smem_s + C::offK + kt * (C::KVR * C::kKV), &tmK, k_full(kt), 0, j0, s0, it.h, it.b);
          }
          __syncwarp();
          mbar_wait_s(v_empty(vt), vp, abort_s, DEV_TIMEOUT_SYNC);
          if (elect_one()) {
            const uint32_t dst = smem_s + C::offV + vt * C::kVB;
            mbar_expect_tx_s(v_full(vt), C::kVB);
            if constexpr (has_bias) {  // rows of 64 16-bit values, or twice rows of 32 floats
              tma_load_4d_s(dst + C::KVR * C::kKV, &tmB, v_full(vt), j0, i0, it.h, it.b);
              if constexpr (!BIAS16)
                tma_load_4d_s(dst + C::KVR * C::kKV + C::BTL * (C::kBias / 2), &tmB, v_full(vt), j0 + 32, i0, it.h, it.b);
            }
            tma_load_5d_s(dst, &tmV, v_full(vt), 0, j0, s0, it.h, it.b);
          }
          __syncwarp();
          if (++kt == NK) { kt = 0; kp ^= 1; }
          if (++vt == NV) { vt = 0; vp ^= 1; }
        }
      }
    } else if (warp == 1 || warp == 2) {
      // =============================== MMA issuers: half of the warpgroups each ===============================
      constexpr int HALF = (NW + 1) / 2;
      const int w0 = (warp - 1) * HALF, w1 = warp == 1 ? HALF : NW;
      constexpr uint32_t kIdescS = make_idesc(kBf16, false, false, BM, BN);
      constexpr uint32_t kIdescO = make_idesc(kBf16, false, true, BM, DP + 16);
      // Descriptor halves that never change: the high word holds the stride offset, version and
      // swizzle; the low word is (address >> 4) plus the leading-offset field.
      constexpr uint32_t kHiOp = static_cast<uint32_t>(make_sdesc_const(16, 8 * RB, SWZ) >> 32);
      constexpr uint32_t kLoLbo = static_cast<uint32_t>(make_sdesc_const(16, 0, 0) & 0xffffffffu);
      const uint32_t q_lo0 = ((smem_s + C::offQ) >> 4) | kLoLbo, k_lo0 = ((smem_s + C::offK) >> 4) | kLoLbo;
      const uint32_t v_lo0 = (smem_s + C::offV) >> 4, ones = (smem_s + C::offOnes) >> 4;
      uint32_t n_item = 0;
      uint32_t gs = 0, kt = 0, kp = 0;  // next S: key tile, K stage and its parity
      uint32_t go = 0, vt = 0, vp = 0;  // next P V: key tile, V stage and its parity
      // S of the next key tile for the warpgroups of this warp.  With one score buffer the softmax warps wait
      // for S and the bias tile at once: this warp sees the tile land and arrives on their barrier too.
      auto issue_s = [&](int w, bool last) {
        const uint32_t qa = q_lo0 + (n_item % QST * NW + w) * (C::kQ >> 4);
        const uint32_t ka = k_lo0 + (kt * C::KVR + (QP ? 0 : w)) * (C::kKV >> 4);
        const uint32_t tS = tmem + w * C::tmemWg + (gs % SB) * BN, bar = s_full(w, gs % SB);
        mbar_wait_s(k_full(kt), kp, abort_s, DEV_TIMEOUT_TMA);
        tc_fence_after();
        const uint32_t el = elect_one();
#pragma unroll
        for (int kk = 0; kk < DP / 16; ++kk)
          mma_ss_e(el, tS, pack_desc(qa + kk * 2, kHiOp), pack_desc(ka + kk * 2, kHiOp), kIdescS, kk > 0 ? 1u : 0u);
        mma_commit_if_s(el, bar);
        mma_commit_if_s(el, k_empty(kt));
        if (last) mma_commit_if_s(el, q_empty(n_item % QST));
      };
      auto next_s = [&]() {
        ++gs;
        if (++kt == NK) { kt = 0; kp ^= 1; }
      };
      auto bias_landed = [&](int w, uint32_t st, uint32_t par) {
        if constexpr (has_bias && SB == 1) {
          mbar_wait_s(v_full(st), par, abort_s, DEV_TIMEOUT_TMA);
          if (elect_one()) mbar_arrive_s(s_full(w, 0));
          __syncwarp();
        }
      };
      // O += P V, and the row sums of P as it was rounded, by which O is divided (see the epilogue): the B
      // operand is DP columns of V followed by 16 of ones, which are simply its next block along N (the leading
      // offset leads from the V tile to them).
      auto issue_pv = [&](int w, bool first, bool last) {  // (the first of an item overwrites)
        const uint32_t va = v_lo0 + vt * (C::kVB >> 4) + (QP ? 0 : w) * (C::kKV >> 4);
        const uint32_t tW = tmem + w * C::tmemWg, tP = tW + (go % SB) * BN;
        const uint32_t d0 = va | ((ones - va) << 16);
        mbar_wait_s(v_full(vt), vp, abort_s, DEV_TIMEOUT_TMA);
        mbar_wait_s(p_full(w, go % SB), (go / SB) & 1, abort_s, DEV_TIMEOUT_SYNC);
        tc_fence_after();
        const uint32_t el = elect_one();
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)  // 16 keys = 8 packed columns of P per step
          mma_ts_e(el, tW + C::colO, tP + kk * 8, pack_desc(d0 + kk * (RB - (RB << 16)), kHiOp), kIdescO, (kk > 0 || !first) ? 1u : 0u);
        if (SB == 2 || last) mma_commit_if_s(el, o_full(w, go % SB));
        mma_commit_if_s(el, v_empty(vt));  // (P has arrived, so the bias tile has been read)
      };
#pragma unroll 1
      for (int item = blockIdx.x; item < wk.n_items; item += gridDim.x) {
        mbar_wait_s(q_full(n_item % QST), (n_item / QST) & 1, abort_s, DEV_TIMEOUT_TMA);
#pragma unroll 1
        for (int t = 0; t < SB && t < T_TILES; ++t) {
#pragma unroll 1
          for (int w = w0; w < w1; ++w) {
            issue_s(w, t == T_TILES - 1);
            bias_landed(w, vt, vp);
          }
          next_s();
        }
#pragma unroll 1
        for (int t = 0; t < T_TILES; ++t) {
          const bool more = t + SB < T_TILES;
          const uint32_t vt1 = vt + 1 == NV ? 0 : vt + 1, vp1 = vp ^ (vt + 1 == NV ? 1u : 0u);
#pragma unroll 1
          for (int w = w0; w < w1; ++w) {
            issue_pv(w, t == 0, t == T_TILES - 1);
            // (the score buffer was read before P was signalled, and P is read before it is overwritten: the MMAs
            // of one thread execute in order)
            if (more) {
              issue_s(w, t + SB == T_TILES - 1);
              bias_landed(w, vt1, vp1);
            }
          }
          vt = vt1;
          vp = vp1;
          ++go;
          if (more) next_s();
        }
        ++n_item;
      }
    } else if (warp == 3) {
      // =============================== residue-mask stager ===============================
      // One float per key for each warpgroup's MSA row, one item ahead of the softmax warps.
      // Keys beyond R are always excluded.  A lane takes eight consecutive keys: one address, then
      // independent loads.  (A chain of test, load and convert per key, as the compiler made of a branching
      // helper, took 18 000 cycles an item and set the pace of the whole kernel.)
      constexpr bool kMin = MASKMODE == MASK_MIN;
      const int kind = a.mask_kind;
      const int es = kind == EVOATTN_MASK_BOOL ? 1 : kind == EVOATTN_MASK_ADD_F32 ? 4 : 2;
      const long long step = a.smask.c * es;  // bytes from key to key
      uint32_t n = 0;
#pragma unroll 1
      for (int item = blockIdx.x; item < wk.n_items; item += gridDim.x, ++n) {
        const Item it = decode_item(item, wk);
        const int st = n & 1;
#pragma unroll 1
        for (int w = 0; w < NW; ++w) {
          const unsigned char* ptr = reinterpret_cast<const unsigned char*>(a.mask) +
                                     ((long long)it.b * a.smask.a + (long long)min(row_of(it, w), a.S - 1) * a.smask.b) * es;
          mbar_wait_s(m_empty(w, st), ((n >> 1) & 1) ^ 1, abort_s, DEV_TIMEOUT_SYNC);
          float* dst = sMask + (w * 2 + st) * r_pad;
          uint32_t dirty = 0;
#pragma unroll 1
          for (int j0 = 0; j0 < r_pad; j0 += 256) {
            const int j = j0 + lane * 8;
            const unsigned char* q = ptr + j * step;
            uint32_t raw[8];
            if (kind == EVOATTN_MASK_BOOL) {
#pragma unroll
              for (int u = 0; u < 8; ++u) raw[u] = ldg_u8_if(q + u * step, j + u < a.R);
            } else if (kind == EVOATTN_MASK_ADD_F32) {
#pragma unroll
              for (int u = 0; u < 8; ++u) raw[u] = ldg_u32_if(q + u * step, j + u < a.R);
            } else if (kind == EVOATTN_MASK_ADD_SAME) {
#pragma unroll
              for (int u = 0; u < 8; ++u) raw[u] = ldg_u16_if(q + u * step, j + u < a.R);
            }
            float m[8];
            bool any = false;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              float v = kMin ? FLT_MAX : 0.f;
              if constexpr (kMin) {
                if (kind == EVOATTN_MASK_BOOL && raw[u] == 0) v = -FLT_MAX;
              } else {
                if (kind == EVOATTN_MASK_ADD_F32) v = __uint_as_float(raw[u]);
                else unpack2<T>(raw[u], v, m[u]);
              }
              m[u] = j + u < a.R ? v : -FLT_MAX;
              any |= kMin ? m[u] < 0.f : m[u] != 0.f;
            }
            if (j < r_pad) {
              *reinterpret_cast<float4*>(dst + j) = make_float4(m[0], m[1], m[2], m[3]);
              *reinterpret_cast<float4*>(dst + j + 4) = make_float4(m[4], m[5], m[6], m[7]);
            }
            const uint32_t lanes_any = __ballot_sync(0xffffffffu, any);  // eight lanes to a key tile
            for (int k = 0; k < 4; ++k)
              if ((lanes_any >> (8 * k)) & 0xffu) dirty |= 1u << (j0 / BN + k);
          }
          if (lane == 0) sDirty[w * 2 + st] = dirty;
          __syncwarp();
          if (lane == 0) mbar_arrive_s(m_full(w, st));
        }
      }
    }
  } else {
    // =============================== softmax warpgroups ===============================
    setmaxnreg_inc<C::kSoftmaxRegs>();
    const int w = (warp >> 2) - 1;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t t_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + w * C::tmemWg;
    const float scale = a.scale;
    const F2 scale2 = f2_make(scale, scale);
    // this thread's row of a bias tile (in query-pair mode the two tiles of a box follow one another)
    constexpr int kBoxBias = BIAS16 ? C::kBias : C::kBias / 2;
    const uint32_t brow0_s = smem_s + C::offV + C::KVR * C::kKV + (QP ? w : 0) * kBoxBias + row * 128;
    uint32_t vt = 0, vp = 0;     // stage of the bias ring and its parity
    uint32_t g = 0, n_item = 0;  // running key-tile and item index
#pragma unroll 1
    for (int item = blockIdx.x; item < wk.n_items; item += gridDim.x, ++n_item) {
      const Item it = decode_item(item, wk);
      const bool active = row_of(it, w) < a.S && tile_of(it, w) < NQT;
      const int s = min(row_of(it, w), a.S - 1);
      const int i = tile_of(it, w) * BM + row;

      // residue-mask row of (b, s), staged by warp 3
      const uint32_t mst = n_item & 1;
      mbar_wait_s(m_full(w, mst), (n_item >> 1) & 1, abort_s, DEV_TIMEOUT_SYNC);
      const uint32_t mrow_s = smem_u32(sMask) + (w * 2 + mst) * r_pad * 4;
      uint32_t dirty = lds_u32(smem_u32(sDirty) + (w * 2 + mst) * 4);

      // The gate's row is wanted in the epilogue, where every cycle of its latency would be waited for.
      const T* grow = a.gate ? reinterpret_cast<const T*>(a.gate) + off4(a.sgate, it.b, it.h, s, i < a.R ? i : 0) : nullptr;
      if (grow != nullptr) prefetch_l2(grow);

      float m_run = -FLT_MAX, l_run = 0.f;
      bool alive = false;  // every row of this warp has a running maximum that the fast path below can take

#pragma unroll 1
      for (int t = 0; t < T_TILES; ++t, ++g) {
        const uint32_t tS = t_base + (g % SB) * BN;
        const uint32_t brow_s = brow0_s + vt * C::kVB;
        const uint32_t mtile_s = mrow_s + t * (BN * 4);
        mbar_wait_s(s_full(w, g % SB), (g / SB) & 1, abort_s, DEV_TIMEOUT_MMA);
        tc_fence_after();
        if (has_bias && SB == 2) mbar_wait_s(v_full(vt), vp, abort_s, DEV_TIMEOUT_TMA);

        auto scores8 = [&](const uint32_t* s8, int g8, auto with_mask, float (&v)[8]) {
          row_scores8<T, MASKMODE, BIAS, C::BTL * kBoxBias, decltype(with_mask)::value>(s8, g8, row, scale2, brow_s, mtile_s, v);
        };

        float lsum = 0.f;
        uint32_t pk[BN / 2];
        bool go = alive, settled = false;
#pragma unroll 1
        for (;;) {
          bool bad = true;
          if (go) {
            const float nm2 = -m_run * kLog2e;
            const F2 l2e2 = f2_make(kLog2e, kLog2e), nm22 = f2_make(nm2, nm2);
            F2 ls4[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) ls4[u] = f2_make(0.f, 0.f);
            auto exps = [&](auto with_mask) {
              uint32_t sr[2][16];  // S, sixteen columns ahead of the arithmetic
              tmem_ld16(tS, sr[0]);
#pragma unroll
              for (int g8 = 0; g8 < BN / 8; ++g8) {
                if (g8 % 2 == 0) {
                  tmem_wait_ld();
                  if (g8 + 2 < BN / 8) tmem_ld16(tS + 8 * g8 + 16, sr[(g8 / 2 + 1) & 1]);
                }
                float v[8];
                scores8(sr[(g8 / 2) & 1] + 8 * (g8 & 1), g8, with_mask, v);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const F2 x2 = f2_make(v[2 * u], v[2 * u + 1]);
                  float y0, y1;
                  if constexpr (decltype(with_mask)::value && MASKMODE == MASK_ADD)  // (see far_tile)
                    f2_get(f2_mul(f2_add(x2, f2_make(-m_run, -m_run)), l2e2), y0, y1);
                  else
                    f2_get(f2_fma(x2, l2e2, nm22), y0, y1);
                  const float p0 = ex2(y0), p1 = ex2(y1);
                  ls4[u] = f2_add(ls4[u], f2_make(p0, p1));
                  pk[g8 * 4 + u] = Pack2<T>::pack(p0, p1);
                }
              }
            };
            if (__builtin_expect((dirty >> t) & 1u, 0)) exps(std::true_type{});
            else exps(std::false_type{});
            float lsa[8];
#pragma unroll
            for (int u = 0; u < 4; ++u) f2_get(ls4[u], lsa[2 * u], lsa[2 * u + 1]);
            lsum = ((lsa[0] + lsa[1]) + (lsa[2] + lsa[3])) + ((lsa[4] + lsa[5]) + (lsa[6] + lsa[7]));
            bad = __any_sync(0xffffffffu, !(lsum <= Lag<T>::kMaxSum));
          }
          if (__builtin_expect(!bad || settled, 1)) break;
          // The tile's own maximum, and the running one follows it.
          float mx = -FLT_MAX;
#pragma unroll 1
          for (int h = 0; h < BN / 32; ++h) {
            uint32_t s32[32];
            tmem_ld32(tS + 32 * h, s32);
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              float v[8];
              scores8(s32 + 8 * k, 4 * h + k, std::true_type{}, v);
#pragma unroll
              for (int u = 0; u < 8; u += 2) mx = max3(mx, v[u], v[u + 1]);
            }
          }
          bool steep = false;  // the next tile may well rise as much again
          if (t == 0) {
            m_run = mx;
          } else {
            steep = mx > m_run + Lag<T>::kRise;
            if (__any_sync(0xffffffffu, mx > m_run)) {
              const float m_up = fmaxf(mx, m_run);
              const float alpha = ex2((m_run - m_up) * kLog2e);
              m_run = m_up;
              l_run *= alpha;
              // (P V of the tile before has to be complete: with one score buffer, S of this tile came after it)
              if constexpr (SB == 2) mbar_wait_s(o_full(w, (g - 1) & 1), ((g - 1) >> 1) & 1, abort_s, DEV_TIMEOUT_MMA);
              tc_fence_after();
#pragma unroll 1
              for (int d0 = 0; d0 < DP + 16; d0 += 16) {  // O and the row sum behind it
                uint32_t o[16];
                tmem_ld16(t_base + C::colO + d0, o);
                tmem_wait_ld();
#pragma unroll
                for (int u = 0; u < 16; ++u) o[u] = __float_as_uint(__uint_as_float(o[u]) * alpha);
                tmem_st16(t_base + C::colO + d0, o);
              }
            }
          }
          alive = !__any_sync(0xffffffffu, m_run == -FLT_MAX || steep);
          go = __any_sync(0xffffffffu, m_run != -FLT_MAX);
          settled = true;
          if (__any_sync(0xffffffffu, m_run != -FLT_MAX && fabsf(m_run) > kFar)) {  // (see far_tile)
            if constexpr (MASKMODE == MASK_ADD) dirty = ~0u;
            else alive = go = false;
          }
        }
        if (!alive) {
          if (!go && __any_sync(0xffffffffu, m_run != -FLT_MAX)) {
            lsum = far_tile<T, BIAS, C::BTL * kBoxBias>(tS, m_run, row, scale, brow_s, mtile_s);
            tmem_wait_st();
            tmem_ld32(tS, pk);
            tmem_wait_ld();
          }
          if (m_run == -FLT_MAX) {
            // every key seen so far was dropped: the scores are all -FLT_MAX and the softmax is
            // uniform over the real keys (test.py:54-55 semantics)
            const int real = min(BN, a.R - t * BN);
            lsum = (float)real;
#pragma unroll
            for (int e = 0; e < BN; e += 2) pk[e / 2] = Pack2<T>::pack(e < real ? 1.f : 0.f, e + 1 < real ? 1.f : 0.f);
          }
        }
        l_run += lsum;
        if (++vt == NV) { vt = 0; vp ^= 1; }

        // P_n -> TMEM, packed two 16-bit values per column, over the first half of the S_n
        // columns this thread has just consumed (lane = row, column j = keys 2j, 2j+1): the
        // A operand of P V comes straight from tensor memory.
        tmem_st32(tS, pk);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_s(p_full(w, g % SB));
      }
      uint4 gw[DP / 8];
      if (grow != nullptr) {
#pragma unroll
        for (int d8 = 0; d8 < DP / 8; ++d8) gw[d8] = d8 * 8 < a.D ? *reinterpret_cast<const uint4*>(grow + d8 * 8) : make_uint4(0, 0, 0, 0);
      }
      // O of the item, complete with its last P V
      if constexpr (SB == 2) mbar_wait_s(o_full(w, (g - 1) & 1), ((g - 1) >> 1) & 1, abort_s, DEV_TIMEOUT_MMA);
      else mbar_wait_s(o_full(w, 0), n_item & 1, abort_s, DEV_TIMEOUT_MMA);
      tc_fence_after();
      float acc[DP];
#pragma unroll
      for (int d0 = 0; d0 < DP; d0 += 16) tmem_ld16(t_base + C::colO + d0, *reinterpret_cast<uint32_t(*)[16]>(&acc[d0]));
      // O is divided by the sum of the P it was made of, rounded to the storage type.  The running maximum
      // may lag, so the largest P of a row is not exactly 1; with the sum of the unrounded values its
      // rounding would go into O in full (an fp16 O was off by 5.4e-4 instead of 2.7e-4).  The log-sum-exp
      // is that of the unrounded values.
      uint32_t lr[4];
      tmem_ld4(t_base + C::colL, lr);
      tmem_wait_ld();
      tc_fence_before();  // (the next item's first P V, which overwrites O, is released by a later arrival)
      if (active && i < a.R) {
        const float inv = 1.f / __uint_as_float(lr[0]);
        T* orow = reinterpret_cast<T*>(a.o) + off4(a.so, it.b, it.h, s, i);
#pragma unroll
        for (int d8 = 0; d8 < DP / 8; ++d8) {
          if (d8 * 8 < a.D) {
            float f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) f[u] = acc[d8 * 8 + u] * inv;
            if (grow != nullptr) {  // gated output: O * sigmoid(gate), in the epilogue
              const uint32_t w4[4] = {gw[d8].x, gw[d8].y, gw[d8].z, gw[d8].w};
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                float g0, g1;
                unpack2<T>(w4[u], g0, g1);
                f[2 * u] *= sigmoid16(g0);
                f[2 * u + 1] *= sigmoid16(g1);
              }
            }
            uint4 v4;
            v4.x = Pack2<T>::pack(f[0], f[1]);
            v4.y = Pack2<T>::pack(f[2], f[3]);
            v4.z = Pack2<T>::pack(f[4], f[5]);
            v4.w = Pack2<T>::pack(f[6], f[7]);
            *reinterpret_cast<uint4*>(orow + d8 * 8) = v4;
          }
        }
        const long long li = (((long long)it.b * a.H + it.h) * a.S + s) * a.R + i;
        a.lse[li] = (m_run == -FLT_MAX) ? -FLT_MAX : (m_run + logf(l_run));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive_s(m_empty(w, mst));
    }
  }

  end_of_cta(abort_flag, a.status);
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

// The order of the items.  With the query tiles fastest the CTAs that work side by side share the K and V of few rows,
// which then come from DRAM once; with the MSA rows fastest they share the bias tile and spread over the K and V of many
// rows, all of which come back for every query tile.  That is the better way where they are still in L2 then (126 MB, next
// to everything else) and there are more than a few query tiles.  Us, query tiles fastest and rows fastest, by the K and
// V of a (b,h):
//   64 MB and more: [1,1024,1024,8,32] fp32 bias 2 904 and 3 063, [1,512,1024,4,64] bf16 982 and 1 103,
//     [1,512,2048,4,64] 3 524 and 4 089, [1,128,2048,4,64] without a bias 842 and 895
//   48 MB: [1,512,768,8,32] bf16 856 and 877, [1,512,1024,8,24] 1 590 and 1 585, [1,128,2048,4,48] 1 011 and 992
//   32 MB and less, from six tiles on: [1,1024,1024,8,8] fp32 2 938 and 2 838, [1,128,1024,4,48] bf16 286 and 269,
//     [1,128,2048,8,8] fp32 1 439 and 1 369, [1,128,768,8,32] 236 and 230, [1,32,2048,4,64] without a bias 240 and 234
//   up to three tiles: [1,128,384,8,32] fp32 75 and 77, [1,1024,384,4,64] 354 and 381, [1,1024,384,8,8] 478 and 475,
//     [1,512,256,8,24] 143 and 141
bool rows_first(const Args& a, int query_tiles) {
  return query_tiles > 4 && 4LL * a.S * a.R * a.D < 40LL << 20;
}

template <class T, int DP, int BIAS, int NW, bool QP>
int launch_t(const Args& a, cudaStream_t st, int* launches) {
  using C = Cfg<DP, NW, QP, BIAS>;
  CUtensorMap tq, tk, tv, tb;
  if (!make_qkv_map(&tq, a.q, a.sq, a.B, a.H, a.S, a.R, a.D, DP, QP ? NW * BM : BM, C::KVR)) return EVOATTN_ERR_CUDA;
  if (!make_qkv_map(&tk, a.k, a.sk, a.B, a.H, a.S, a.R, a.D, DP, BN, C::KVR)) return EVOATTN_ERR_CUDA;
  if (!make_qkv_map(&tv, a.v, a.sv, a.B, a.H, a.S, a.R, a.D, DP, BN, C::KVR)) return EVOATTN_ERR_CUDA;
  if (a.bias) {
    const bool ok = a.bias16 ? make_bias16_map(&tb, a.bias, a.sbias, a.B, a.H, a.R, C::BTL * BM, BN)
                             : make_bias_map(&tb, a.bias, a.sbias, a.B, a.H, a.R, C::BTL * BM, 32);
    if (!ok) return EVOATTN_ERR_CUDA;
  } else {
    tb = tq;
  }
  const int sms = sm_count();
  if (sms <= 0) return EVOATTN_ERR_CUDA;
  const int T_TILES = (a.R + BN - 1) / BN;
  const int NQT = (a.R + BM - 1) / BM;
  const size_t smem = C::bytes(T_TILES * BN);
  const int inner = QP ? a.S : (a.S + NW - 1) / NW, outer = QP ? (NQT + NW - 1) / NW : NQT;
  const long long items = (long long)a.B * a.H * outer * inner;
  const bool rf = rows_first(a, NQT);
  const Walk wk{(int)items, rf, fast_div((uint32_t)(rf ? inner : outer)), fast_div((uint32_t)(rf ? outer : inner)), fast_div((uint32_t)a.H)};
  const int grid = (int)(items < sms ? items : sms);
  const bool add = a.mask_kind == EVOATTN_MASK_ADD_F32 || a.mask_kind == EVOATTN_MASK_ADD_SAME;
  auto kern = add ? evo_fwd_sm100_kernel<T, DP, MASK_ADD, BIAS, NW, QP> : evo_fwd_sm100_kernel<T, DP, MASK_MIN, BIAS, NW, QP>;
  // setmaxnreg.inc waits until the scheduler's register pool (1 + NW warps at the launch-time count) has what
  // it asks for: never launch a build whose pool cannot hold the warps' requests.
  int num_regs = 0;
  if (!kernel_ready(reinterpret_cast<const void*>(kern), (int)smem, &num_regs)) return EVOATTN_ERR_CUDA;
  if ((1 + NW) * num_regs < NW * C::kSoftmaxRegs + C::kServiceRegs) return EVOATTN_ERR_UNSUPPORTED;
  launch_dependent(kern, dim3((unsigned)grid), C::kThreads, smem, st, a, wk, tq, tk, tv, tb);
  *launches += 1;
  return cudaGetLastError() == cudaSuccess ? EVOATTN_OK : EVOATTN_ERR_CUDA;
}

// A single MSA row with several query tiles runs in query-pair mode (both warpgroups get work).  Several rows
// share the larger tile, the pair bias, two to four of them at a time.
template <class T, int DP, int BIAS>
int launch_mode(const Args& a, cudaStream_t st, int* launches) {
  const int r_pad = (a.R + BN - 1) / BN * BN;
  if (a.S == 1 && a.R > BM) return launch_t<T, DP, BIAS, 2, true>(a, st, launches);
  const int sms = sm_count();
  if (sms <= 0) return EVOATTN_ERR_CUDA;
  // Time of the busiest CTA: the items it walks, times what an item of two, three or four rows costs (each
  // measured with the CTAs evenly loaded, [1,148,1024,4,32] 17.6, 22.3 and 27.7 us, [1,64,768,8,64] 16.0 and 21.4).
  // What the rounding to whole items does to it: [1,128,384,8,32] 89.1, 76.9 and 78.1 us, [1,64,500,4,16] 41.1,
  // 41.0 and 37.3, [1,4,384,8,32] 12.4, 15.0 and 18.5, [1,96,384,8,64] 76.8 and 80.3.
  const auto cost = [&](int nw, long long item) {
    const long long items = (long long)a.B * a.H * ((a.R + BM - 1) / BM) * ((a.S + nw - 1) / nw);
    return (items + sms - 1) / sms * item;
  };
  int nw = 2;
  long long best = cost(2, 100);
  const long long three = cost(3, DP == 64 ? 137 : 130);
  if (Cfg<DP, 3, false, BIAS>::bytes(r_pad) <= kMaxSmem && three < best) {
    nw = 3;
    best = three;
  }
  if constexpr (DP <= 32) {
    if (Cfg<DP, 4, false, BIAS>::bytes(r_pad) <= kMaxSmem && cost(4, 158) < best) nw = 4;
  }
  if constexpr (DP <= 32) {
    if (nw == 4) return launch_t<T, DP, BIAS, 4, false>(a, st, launches);
  }
  if (nw == 3) return launch_t<T, DP, BIAS, 3, false>(a, st, launches);
  return launch_t<T, DP, BIAS, 2, false>(a, st, launches);
}
template <class T, int DP>
int launch_bias(const Args& a, cudaStream_t st, int* launches) {
  if (!a.bias) return launch_mode<T, DP, BIAS_NONE>(a, st, launches);
  if (a.bias16) return launch_mode<T, DP, BIAS_16>(a, st, launches);
  return launch_mode<T, DP, BIAS_F32>(a, st, launches);
}

template <class T>
int launch_d(const Args& a, cudaStream_t st, int* launches) {
  if (a.D <= 16) return launch_bias<T, 16>(a, st, launches);
  if (a.D <= 32) return launch_bias<T, 32>(a, st, launches);
  return launch_bias<T, 64>(a, st, launches);
}

}  // namespace

bool sm100_fwd_supported(int dtype, const Args& a) {
  if (dtype != EVOATTN_BF16 && dtype != EVOATTN_FP16) return false;
  if (a.D % 8 != 0 || a.D > 64) return false;
  if (a.R > kMaxRes) return false;
  if (a.bias) {
    const int es = a.bias16 ? 2 : 4;
    if ((reinterpret_cast<uintptr_t>(a.bias) & 15) != 0) return false;
    if ((a.sbias.a * es) % 16 || (a.sbias.b * es) % 16 || (a.sbias.c * es) % 16) return false;
  }
  if ((long long)a.B * a.H * a.S * ((a.R + BM - 1) / BM) > 2147483647LL) return false;
  return true;
}

int launch_sm100_fwd(int dtype, const Args& a, cudaStream_t st, int* launches) {
  if (dtype == EVOATTN_BF16) return launch_d<__nv_bfloat16>(a, st, launches);
  return launch_d<__half>(a, st, launches);
}

}  // namespace evo
