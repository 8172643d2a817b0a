// CUDA-core Evoformer attention kernels: any dtype (fp32 included), any D <= 128, any R.
//
// These serve fp32 inputs (tensor cores would lose bits there) and every shape the tcgen05 kernels do
// not cover.  fp32 math throughout, every sum in a fixed order: the pair-bias gradient is produced by
// one owner per element instead of the reference's fp32 atomics (dsevoformer-triton/evoformer.py:458),
// and dQ and dK/dV each compute the scores, so results are the same bits on every run.
//
// Math (evoformer.py:68-89 forward, :450-462 and :594-614 backward):
//   x_ij = scale * <q_i,k_j> + bias_ij ;  mask ;  P = softmax_j(x) ;  O = P V
//   delta_i = <dO_i,O_i> ; dP_ij = <dO_i,v_j> ; dS = P (dP - delta)
//   dV_j = sum_i P_ij dO_i ; dQ_i = scale sum_j dS_ij k_j ; dK_j = scale sum_i dS_ij q_i
//   dBias_ij = sum_s dS_ij
//
// Bound by the fp32 FMA rate.  A block of 256 threads works on 64 x 64 scores, 4 x 4 per thread, so that
// a 16-byte shared load feeds 16 multiply-adds: rows are strided over the threads (i = ty + 16 r,
// j = tx + 16 c) and a staged row has DP + 4 floats, which makes the 16-byte loads of eight
// neighbouring lanes hit all 32 banks once without transposing anything on the way in.
// [1,32,256,8,32] fp32: forward 115 us, backward 356 us (37 and 30 TFLOP/s of about 74); with one warp per
// score row, as before, 940 us and 6 ms.
#include "common.cuh"
#include "launch.h"
#include "ptx.cuh"

namespace evo {
namespace {

using ptx::F2;
using ptx::f2_fma;
using ptx::f2_get;
using ptx::f2_make;

constexpr int TT = 64;        // rows of a tile (queries and keys)
constexpr int NTH = 256;
constexpr int PLD = TT + 4;   // row stride of a staged score tile

struct Slab {
  int b, h, s;
};
__device__ __forceinline__ Slab slab_of(int idx, const Args& a) {
  Slab r;
  r.s = idx % a.S;
  r.h = (idx / a.S) % a.H;
  r.b = idx / (a.S * a.H);
  return r;
}

// `n` rows r0.. of slab (b,h,s) -> shared memory, widened, rows of DP + 4 floats; zeros beyond R and D.
// `t` of `nt` threads take part.
template <class T, int DP>
__device__ __forceinline__ void stage_rows(float* dst, const T* x, const Str4& st, const Slab& sl, int r0, int n, int R, int D,
                                           bool vec, int t, int nt) {
  constexpr int LD = DP + 4, C4 = DP / 4;
  const T* base = x + off4(st, sl.b, sl.h, sl.s, 0);
  for (int e = t; e < n * C4; e += nt) {
    const int rr = e / C4, d = (e - rr * C4) * 4, r = r0 + rr;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < R) {
      const T* p = base + (long long)r * st.r + d;
      if (vec && d + 4 <= D) {
        if constexpr (sizeof(T) == 4) {
          v = *reinterpret_cast<const float4*>(p);
        } else {
          const uint2 w = *reinterpret_cast<const uint2*>(p);
          const T* h = reinterpret_cast<const T*>(&w);
          v = make_float4(to_float<T>(h[0]), to_float<T>(h[1]), to_float<T>(h[2]), to_float<T>(h[3]));
        }
      } else {
        if (d < D) v.x = to_float<T>(p[0]);
        if (d + 1 < D) v.y = to_float<T>(p[1]);
        if (d + 2 < D) v.z = to_float<T>(p[2]);
        if (d + 3 < D) v.w = to_float<T>(p[3]);
      }
    }
    *reinterpret_cast<float4*>(dst + rr * LD + d) = v;
  }
}

// The same without waiting for the loads where they can be asynchronous (fp32 rows read 16 bytes at a time):
// the caller waits with async_wait() before the barrier that makes the rows visible.
template <class T, int DP>
__device__ __forceinline__ void stage_rows_ahead(float* dst, const T* x, const Str4& st, const Slab& sl, int r0, int n, int R, int D,
                                                 bool vec) {
  if constexpr (sizeof(T) == 4) {
    if (vec && D == DP) {
      constexpr int LD = DP + 4, C4 = DP / 4;
      const T* base = x + off4(st, sl.b, sl.h, sl.s, 0);
      for (int e = threadIdx.x; e < n * C4; e += NTH) {
        const int rr = e / C4, d = (e - rr * C4) * 4, r = r0 + rr;
        const int bytes = r < R ? 16 : 0;  // (rows beyond R are filled with zeros)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_u32(dst + rr * LD + d)),
                     "l"(base + (long long)min(r, R - 1) * st.r + d), "r"(bytes)
                     : "memory");
      }
      return;
    }
  }
  stage_rows<T, DP>(dst, x, st, sl, r0, n, R, D, vec, threadIdx.x, NTH);
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Whether the tiles of the inner loop are double-buffered: the next pair is loaded under the arithmetic
// of this one (at DP = 128 two pairs do not fit).
template <int DP> constexpr bool kAhead = DP <= 64;

// acc[r][c] = <A row ty + W r, B row tx + W c> over DP columns.  Two columns per instruction: the even
// and the odd ones are summed apart and added at the end.
template <int DP, int W>
__device__ __forceinline__ void dots(float (&acc)[4][4], const float* A, const float* B, int ty, int tx) {
  constexpr int LD = DP + 4;
  F2 s[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) s[r][c] = f2_make(0.f, 0.f);
#pragma unroll 1
  for (int d = 0; d < DP; d += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const float4*>(A + (ty + W * r) * LD + d);
#pragma unroll
    for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(B + (tx + W * c) * LD + d);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        s[r][c] = f2_fma(f2_make(a[r].x, a[r].y), f2_make(b[c].x, b[c].y), s[r][c]);
        s[r][c] = f2_fma(f2_make(a[r].z, a[r].w), f2_make(b[c].z, b[c].w), s[r][c]);
      }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float lo, hi;
      f2_get(s[r][c], lo, hi);
      acc[r][c] = lo + hi;
    }
}

// The columns of a [rows][DP] product that a thread owns: NC of them, in runs of VEC.
template <int DP>
struct Cols {
  static constexpr int NC = DP / 16, VEC = NC < 4 ? NC : 4;
  static __device__ __forceinline__ int at(int tx, int n) { return (n / VEC) * (16 * VEC) + tx * VEC + n % VEC; }
};

// acc[r][n] += sum_j P[ty + 16 r][j] * V[j][col n] over the 64 rows of V.
template <int DP>
__device__ __forceinline__ void weighted_rows(float (&acc)[4][DP / 16], const float* P, const float* V, int ty, int tx) {
  using C = Cols<DP>;
  constexpr int LD = DP + 4;
#pragma unroll 2
  for (int j = 0; j < TT; j += 4) {
    float p[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float4 t = *reinterpret_cast<const float4*>(P + (ty + 16 * r) * PLD + j);
      p[r][0] = t.x; p[r][1] = t.y; p[r][2] = t.z; p[r][3] = t.w;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float v[C::NC];
#pragma unroll
      for (int n = 0; n < C::NC; n += C::VEC) {
        const float* src = V + (j + u) * LD + C::at(tx, n);
        if constexpr (C::VEC == 4) {
          const float4 t = *reinterpret_cast<const float4*>(src);
          v[n] = t.x; v[n + 1] = t.y; v[n + 2] = t.z; v[n + 3] = t.w;
        } else if constexpr (C::VEC == 2) {
          const float2 t = *reinterpret_cast<const float2*>(src);
          v[n] = t.x; v[n + 1] = t.y;
        } else {
          v[n] = *src;
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int n = 0; n < C::NC; ++n) acc[r][n] += p[r][u] * v[n];
    }
  }
}

// What is added to the 4 x 4 scores of a thread (i = i0 + ty + W r, j = j0 + tx + W c) before the softmax.
// Read ahead of the dot products, whose arithmetic covers the latency of these loads.
struct Terms {
  float bias[4][4], add[4];
  unsigned replaced;  // bit c: a boolean mask dropped column c (its scores are constants)
};
template <class T, int W>
__device__ __forceinline__ void load_terms(Terms& t, const Args& a, const Slab& sl, int i0, int j0, int ty, int tx) {
  t.replaced = 0;
  const bool full = i0 + 4 * W <= a.R && j0 + 4 * W <= a.R;  // (one address per row, the same for the whole block)
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int j = min(j0 + tx + W * c, a.R - 1);
    const long long mi = (long long)sl.b * a.smask.a + (long long)sl.s * a.smask.b + (long long)j * a.smask.c;
    t.add[c] = 0.f;
    if (a.mask_kind == EVOATTN_MASK_BOOL) t.replaced |= (reinterpret_cast<const unsigned char*>(a.mask)[mi] == 0 ? 1u : 0u) << c;
    else if (a.mask_kind == EVOATTN_MASK_ADD_F32) t.add[c] = reinterpret_cast<const float*>(a.mask)[mi];
    else if (a.mask_kind == EVOATTN_MASK_ADD_SAME) t.add[c] = to_float<T>(reinterpret_cast<const T*>(a.mask)[mi]);
  }
  if (!a.bias) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) t.bias[r][c] = 0.f;
  } else if (full && !a.bias16) {
    const float* p = a.bias + (long long)sl.b * a.sbias.a + (long long)sl.h * a.sbias.b + (long long)(i0 + ty) * a.sbias.c + j0 + tx;
#pragma unroll
    for (int r = 0; r < 4; ++r, p += W * a.sbias.c)
#pragma unroll
      for (int c = 0; c < 4; ++c) t.bias[r][c] = __ldg(p + W * c);
  } else {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        t.bias[r][c] = load_bias<T>(a, sl.b, sl.h, min(i0 + ty + W * r, a.R - 1), min(j0 + tx + W * c, a.R - 1));
  }
}
__device__ __forceinline__ float score(const Terms& t, float scale, float dot, int r, int c) {
  return (t.replaced >> c & 1u) ? -FLT_MAX : (dot * scale + t.bias[r][c]) + t.add[c];
}

// P_ij from a stored log-sum-exp.  A row whose keys were all dropped has lse == -FLT_MAX
// exactly (the log of the row sum is absorbed); its softmax is uniform over the R keys.
__device__ __forceinline__ float prob_from_lse(float x, float lse, int R) {
  if (lse == -FLT_MAX) return 1.f / (float)R;
  return expf(x - lse);
}

// Which loads of a tensor may take 16 bytes (fp32) or 8 (16-bit) at a time.
enum : int { VEC_Q = 1, VEC_K = 2, VEC_V = 4, VEC_DO = 8 };

template <class T, int DP>
__global__ void __launch_bounds__(NTH, DP <= 64 ? 2 : 1) generic_fwd_kernel(const Args a, const int vec) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  extern __shared__ __align__(16) float sm[];
  constexpr int LD = DP + 4;
  float* Qs = sm;
  float* KV = Qs + TT * LD;  // one or two pairs of K and V tiles
  float* Ps = KV + (kAhead<DP> ? 4 : 2) * TT * LD;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const Slab sl = slab_of(blockIdx.x, a);
  const int i0 = blockIdx.y * TT;
  auto stage = [&](int j0) {
    float* dst = KV + (kAhead<DP> ? (j0 / TT & 1) * 2 * TT * LD : 0);
    stage_rows_ahead<T, DP>(dst, reinterpret_cast<const T*>(a.k), a.sk, sl, j0, TT, a.R, a.D, vec & VEC_K);
    stage_rows_ahead<T, DP>(dst + TT * LD, reinterpret_cast<const T*>(a.v), a.sv, sl, j0, TT, a.R, a.D, vec & VEC_V);
  };
  if (kAhead<DP>) stage(0);
  stage_rows<T, DP>(Qs, reinterpret_cast<const T*>(a.q), a.sq, sl, i0, TT, a.R, a.D, vec & VEC_Q, threadIdx.x, NTH);
  float m[4], l[4], acc[4][DP / 16];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int n = 0; n < DP / 16; ++n) acc[r][n] = 0.f;
  }
  for (int j0 = 0; j0 < a.R; j0 += TT) {
    if (!kAhead<DP>) {
      __syncthreads();
      stage(j0);
    }
    async_wait();
    __syncthreads();
    if (kAhead<DP> && j0 + TT < a.R) stage(j0 + TT);  // (the pair the last iteration read)
    const float* Ks = KV + (kAhead<DP> ? (j0 / TT & 1) * 2 * TT * LD : 0);
    const float* Vs = Ks + TT * LD;
    Terms terms;
    load_terms<T, 16>(terms, a, sl, i0, j0, ty, tx);
    float x[4][4];
    dots<DP, 16>(x, Qs, Ks, ty, tx);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        x[r][c] = j0 + tx + 16 * c < a.R ? score(terms, a.scale, x[r][c], r, c) : -INFINITY;
        mx = fmaxf(mx, x[r][c]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float mn = fmaxf(m[r], mx), alpha = expf(m[r] - mn);
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float p = (j0 + tx + 16 * c < a.R) ? expf(x[r][c] - mn) : 0.f;
        sum += p;
        Ps[(ty + 16 * r) * PLD + tx + 16 * c] = p;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l[r] = l[r] * alpha + sum;
      m[r] = mn;
#pragma unroll
      for (int n = 0; n < DP / 16; ++n) acc[r][n] *= alpha;
    }
    __syncwarp();  // (a row of P is written and read by the same half-warp)
    weighted_rows<DP>(acc, Ps, Vs, ty, tx);
    __syncwarp();
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + ty + 16 * r;
    if (i >= a.R) continue;
    T* o = reinterpret_cast<T*>(a.o) + off4(a.so, sl.b, sl.h, sl.s, i);
    const T* gate = a.gate ? reinterpret_cast<const T*>(a.gate) + off4(a.sgate, sl.b, sl.h, sl.s, i) : nullptr;
    const float inv = 1.f / l[r];
#pragma unroll
    for (int n = 0; n < DP / 16; ++n) {
      const int d = Cols<DP>::at(tx, n);
      if (d < a.D) o[d] = from_float<T>(acc[r][n] * inv * (gate ? sigmoidf_fast(to_float<T>(gate[d])) : 1.f));
    }
    if (tx == 0) a.lse[((long long)blockIdx.x) * a.R + i] = m[r] + logf(l[r]);
  }
}

// delta[b,h,s,i] = <dO_i, O_i>   (evoformer.py:299-326), eight lanes per row.
template <class T>
__global__ void __launch_bounds__(256) generic_delta_kernel(const Args a) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  const int lane = threadIdx.x & 7;
  const long long row = (long long)blockIdx.x * 32 + (threadIdx.x >> 3);
  const long long rows = (long long)a.B * a.H * a.S * a.R;
  const long long rc = row < rows ? row : rows - 1;
  const long long slab = rc / a.R;
  const int i = (int)(rc - slab * a.R);
  const Slab sl = slab_of((int)slab, a);
  const T* o = reinterpret_cast<const T*>(a.o) + off4(a.so, sl.b, sl.h, sl.s, i);
  const T* g = reinterpret_cast<const T*>(a.d_o) + off4(a.sdo, sl.b, sl.h, sl.s, i);
  float acc = 0.f;
  for (int d = lane; d < a.D; d += 8) acc += to_float<T>(o[d]) * to_float<T>(g[d]);
#pragma unroll
  for (int m = 4; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
  if (row < rows && lane == 0) a.delta[slab * a.delta_ld + i] = acc;
}

// Gated output Og = sigmoid(gate) * O.  With G = dOg (gradient of the gated output):
//   dO    = G * sigmoid(gate)                      (what the attention backward needs)
//   delta = sum_d dO * O = sum_d G * Og            (so the un-gated O is never needed)
//   dgate = G * O * sigmoid'(gate) = G * Og * (1 - sigmoid(gate))
// One warp per (b,h,s,i) row.  dO is written contiguously ([rows][D]) into scratch.
template <class T>
__global__ void __launch_bounds__(256) generic_gate_backward_kernel(Args a) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * 8 + warp;
  T* d_o_eff = reinterpret_cast<T*>(a.d_o_eff);
  const long long rows = (long long)a.B * a.H * a.S * a.R;
  if (row >= rows) return;
  const int i = (int)(row % a.R);
  long long sl = row / a.R;
  const int s = (int)(sl % a.S); sl /= a.S;
  const int h = (int)(sl % a.H);
  const int b = (int)(sl / a.H);
  const T* og = reinterpret_cast<const T*>(a.o) + off4(a.so, b, h, s, i);
  const T* g = reinterpret_cast<const T*>(a.d_o) + off4(a.sdo, b, h, s, i);
  const T* gt = reinterpret_cast<const T*>(a.gate) + off4(a.sgate, b, h, s, i);
  T* dg = reinterpret_cast<T*>(a.dgate) + off4(a.sdgate, b, h, s, i);
  float acc = 0.f;
  for (int d = lane; d < a.D; d += 32) {
    const float G = to_float<T>(g[d]), O = to_float<T>(og[d]);
    const float sg = sigmoidf_fast(to_float<T>(gt[d]));
    acc += G * O;
    d_o_eff[row * a.D + d] = from_float<T>(G * sg);
    dg[d] = from_float<T>(G * O * (1.f - sg));
  }
  acc = warp_sum(acc);
  if (lane == 0) a.delta[(row / a.R) * a.delta_ld + i] = acc;
}

// The row statistics of a thread's four query rows.
template <int W>
__device__ __forceinline__ void load_stats(float (&lse)[4], float (&delta)[4], const Args& a, long long slab, int i0, int ty) {
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = min(i0 + ty + W * r, a.R - 1);
    lse[r] = a.lse[slab * a.R + i];
    delta[r] = a.delta[slab * a.delta_ld + i];
  }
}

// P and dS of a 4 x 4 patch from its two dot products; both 0 outside the R x R scores.
template <int W>
__device__ __forceinline__ void probs(const Args& a, const Terms& t, const float (&lse)[4], const float (&delta)[4], int i0, int j0,
                                      int ty, int tx, float (&p)[4][4], float (&ds)[4][4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const bool in = i0 + ty + W * r < a.R && j0 + tx + W * c < a.R;
      p[r][c] = in ? prob_from_lse(score(t, a.scale, p[r][c], r, c), lse[r], a.R) : 0.f;
      ds[r][c] = (in && !(t.replaced >> c & 1u)) ? p[r][c] * (ds[r][c] - delta[r]) : 0.f;
    }
}

// dQ of 64 queries of the MSA rows s0 .. s1: walks the keys.  dS is at hand here, so d(pair_bias) of these
// queries and rows is summed on the way, in a buffer that no other block touches (`part`, [R][R] of this
// (b,h) and run of rows): the first row stores, the others add in turn.  That read and write of L2 costs a
// tenth of what a pass of its own did, which had to compute every score and dP once more.
template <class T, int DP>
__device__ __forceinline__ void dq_role(const Args& a, int vec, float* sm, int bh, int s0, int s1, int i0, float* part, int ld) {
  constexpr int LD = DP + 4;
  float* Qs = sm;
  float* Gs = Qs + TT * LD;
  float* KV = Gs + TT * LD;
  float* Ds = KV + (kAhead<DP> ? 4 : 2) * TT * LD;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int srow = s0; srow < s1; ++srow) {
    const Slab sl{bh / a.H, bh % a.H, srow};
    const long long slab = (long long)bh * a.S + srow;
    auto stage = [&](int j0) {
      float* dst = KV + (kAhead<DP> ? (j0 / TT & 1) * 2 * TT * LD : 0);
      stage_rows_ahead<T, DP>(dst, reinterpret_cast<const T*>(a.k), a.sk, sl, j0, TT, a.R, a.D, vec & VEC_K);
      stage_rows_ahead<T, DP>(dst + TT * LD, reinterpret_cast<const T*>(a.v), a.sv, sl, j0, TT, a.R, a.D, vec & VEC_V);
    };
    if (srow > s0) __syncthreads();  // the tiles of the row before have been read
    if (kAhead<DP>) stage(0);
    stage_rows_ahead<T, DP>(Qs, reinterpret_cast<const T*>(a.q), a.sq, sl, i0, TT, a.R, a.D, vec & VEC_Q);
    stage_rows_ahead<T, DP>(Gs, reinterpret_cast<const T*>(a.d_o), a.sdo, sl, i0, TT, a.R, a.D, vec & VEC_DO);
    float acc[4][DP / 16] = {}, lse[4], delta[4];
    load_stats<16>(lse, delta, a, slab, i0, ty);
    for (int j0 = 0; j0 < a.R; j0 += TT) {
      if (!kAhead<DP>) {
        __syncthreads();
        stage(j0);
      }
      async_wait();
      __syncthreads();
      if (kAhead<DP> && j0 + TT < a.R) stage(j0 + TT);
      const float* Ks = KV + (kAhead<DP> ? (j0 / TT & 1) * 2 * TT * LD : 0);
      const float* Vs = Ks + TT * LD;
      Terms terms;
      load_terms<T, 16>(terms, a, sl, i0, j0, ty, tx);
      float p[4][4], ds[4][4];
      dots<DP, 16>(p, Qs, Ks, ty, tx);
      dots<DP, 16>(ds, Gs, Vs, ty, tx);
      probs<16>(a, terms, lse, delta, i0, j0, ty, tx, p, ds);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) Ds[(ty + 16 * r) * PLD + tx + 16 * c] = ds[r][c];
      if (part != nullptr) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int i = i0 + ty + 16 * r;
          float* out = part + (long long)i * ld + j0 + tx;
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (i < a.R && j0 + tx + 16 * c < a.R) out[16 * c] = srow == s0 ? ds[r][c] : out[16 * c] + ds[r][c];
        }
      }
      __syncwarp();  // (a row of dS is written and read by the same half-warp)
      weighted_rows<DP>(acc, Ds, Ks, ty, tx);
      __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = i0 + ty + 16 * r;
      if (i >= a.R) continue;
      T* o = reinterpret_cast<T*>(a.dq) + off4(a.sdq, sl.b, sl.h, sl.s, i);
#pragma unroll
      for (int n = 0; n < DP / 16; ++n) {
        const int d = Cols<DP>::at(tx, n);
        if (d < a.D) o[d] = from_float<T>(acc[r][n] * a.scale);
      }
    }
  }
}

// dK, dV of 64 keys (and their share of an additive mask's gradient): walks the queries.
template <class T, int DP>
__device__ __forceinline__ void dkdv_role(const Args& a, int vec, float* sm, int slab, int j0) {
  constexpr int LD = DP + 4;
  float* Ks = sm;
  float* Vs = Ks + TT * LD;
  float* QG = Vs + TT * LD;
  float* Pt = QG + (kAhead<DP> ? 4 : 2) * TT * LD;  // P^T and dS^T: [key][query]
  float* Dt = Pt + TT * PLD;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const Slab sl = slab_of(slab, a);
  auto stage = [&](int i0) {
    float* dst = QG + (kAhead<DP> ? (i0 / TT & 1) * 2 * TT * LD : 0);
    stage_rows_ahead<T, DP>(dst, reinterpret_cast<const T*>(a.q), a.sq, sl, i0, TT, a.R, a.D, vec & VEC_Q);
    stage_rows_ahead<T, DP>(dst + TT * LD, reinterpret_cast<const T*>(a.d_o), a.sdo, sl, i0, TT, a.R, a.D, vec & VEC_DO);
  };
  if (kAhead<DP>) stage(0);
  stage_rows<T, DP>(Ks, reinterpret_cast<const T*>(a.k), a.sk, sl, j0, TT, a.R, a.D, vec & VEC_K, threadIdx.x, NTH);
  stage_rows<T, DP>(Vs, reinterpret_cast<const T*>(a.v), a.sv, sl, j0, TT, a.R, a.D, vec & VEC_V, threadIdx.x, NTH);
  float accK[4][DP / 16] = {}, accV[4][DP / 16] = {}, dm[4] = {};
  for (int i0 = 0; i0 < a.R; i0 += TT) {
    if (!kAhead<DP>) {
      __syncthreads();
      stage(i0);
    }
    async_wait();
    __syncthreads();
    if (kAhead<DP> && i0 + TT < a.R) stage(i0 + TT);
    const float* Qs = QG + (kAhead<DP> ? (i0 / TT & 1) * 2 * TT * LD : 0);
    const float* Gs = Qs + TT * LD;
    Terms terms;
    load_terms<T, 16>(terms, a, sl, i0, j0, ty, tx);
    float p[4][4], ds[4][4], lse[4], delta[4];
    load_stats<16>(lse, delta, a, slab, i0, ty);
    dots<DP, 16>(p, Qs, Ks, ty, tx);
    dots<DP, 16>(ds, Gs, Vs, ty, tx);
    probs<16>(a, terms, lse, delta, i0, j0, ty, tx, p, ds);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        Pt[(tx + 16 * c) * PLD + ty + 16 * r] = p[r][c];
        Dt[(tx + 16 * c) * PLD + ty + 16 * r] = ds[r][c];
        dm[c] += ds[r][c];
      }
    __syncthreads();
    weighted_rows<DP>(accV, Pt, Gs, ty, tx);
    weighted_rows<DP>(accK, Dt, Qs, ty, tx);
  }
  if (a.dmask != nullptr) {  // one addition per (b,h,s,j): the sum over heads
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 4; ++c) Pt[(tx + 16 * c) * PLD + ty] = dm[c];
    __syncthreads();
    if (threadIdx.x < TT && j0 + threadIdx.x < a.R) {
      float tot = 0.f;
      for (int u = 0; u < 16; ++u) tot += Pt[threadIdx.x * PLD + u];
      atomicAdd(a.dmask + ((long long)sl.b * a.S + sl.s) * a.R + j0 + threadIdx.x, tot);
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int j = j0 + ty + 16 * r;
    if (j >= a.R) continue;
    T* ok = reinterpret_cast<T*>(a.dk) + off4(a.sdk, sl.b, sl.h, sl.s, j);
    T* ov = reinterpret_cast<T*>(a.dv) + off4(a.sdv, sl.b, sl.h, sl.s, j);
#pragma unroll
    for (int n = 0; n < DP / 16; ++n) {
      const int d = Cols<DP>::at(tx, n);
      if (d < a.D) {
        ok[d] = from_float<T>(accK[r][n] * a.scale);
        ov[d] = from_float<T>(accV[r][n]);
      }
    }
  }
}

// How the MSA rows are dealt out to the blocks that compute dQ and d(pair_bias): runs of `rows`, each run
// with a partial d(pair_bias) of its own unless there is only one.  Long enough that the partial sums
// stay few (600 tiles' worth, 150 KB times R, at most), short enough for some four blocks per SM; fewer
// where the scratch has no room for them.
struct Runs {
  int rows, n;
};
Runs plan_runs(const Args& a) {
  if (!a.dbias) return Runs{1, a.S};
  const long long tiles = (long long)a.B * a.H * ((a.R + TT - 1) / TT);
  int want = (int)min((long long)a.S, (600 + tiles - 1) / tiles);
  if (a.max_runs > 0) want = min(want, a.max_runs);
  const int rows = (a.S + want - 1) / want;
  return Runs{rows, (a.S + rows - 1) / rows};
}

// The two parts of a backward call read the same inputs and write different outputs: one launch, the
// blocks that walk several MSA rows first.
template <class T, int DP>
__global__ void __launch_bounds__(NTH, DP <= 32 ? 2 : 1) generic_bwd_kernel(const Args a, const int vec, const Runs runs, float* part,
                                                                          const long long n_dq, const long long n_total) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  extern __shared__ __align__(16) float sm[];
  long long idx = (long long)blockIdx.y * gridDim.x + blockIdx.x;
  if (idx >= n_total) return;
  const int nt = (a.R + TT - 1) / TT;
  const int i0 = (int)(idx % nt) * TT;
  if (idx >= n_dq) {
    idx -= n_dq;
    dkdv_role<T, DP>(a, vec, sm, (int)(idx / nt), (int)(idx % nt) * TT);
    return;
  }
  const int run = (int)(idx / nt % runs.n), bh = (int)(idx / nt / runs.n);
  float* mine = nullptr;
  const int ld = runs.n == 1 ? a.dbias_ld : a.R;
  if (a.dbias) mine = (runs.n == 1 ? a.dbias : part + (long long)run * a.B * a.H * a.R * ld) + (long long)bh * a.R * ld;
  dq_role<T, DP>(a, vec, sm, bh, run * runs.rows, min(a.S, (run + 1) * runs.rows), i0, mine, ld);
}

// d(pair_bias) = the partial sums, added in order.
__global__ void __launch_bounds__(256) generic_dbias_sum_kernel(const float* __restrict__ part, int n, long long rows, int R, float* __restrict__ dst,
                                                                int ld) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  const long long total = rows * R;
  for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < total; e += (long long)gridDim.x * 256) {
    float t = part[e];
    for (int k = 1; k < n; ++k) t += part[k * total + e];
    dst[ld == R ? e : e / R * ld + e % R] = t;
  }
}

template <int DP> constexpr int fwd_smem() { return ((kAhead<DP> ? 5 : 3) * TT * (DP + 4) + TT * PLD) * 4; }
template <int DP> constexpr int bwd_smem() { return ((kAhead<DP> ? 6 : 4) * TT * (DP + 4) + 2 * TT * PLD) * 4; }

template <class T>
bool vec_ok(const void* p, const Str4& s) {
  const long long n = 4;  // elements of a vector load
  return reinterpret_cast<uintptr_t>(p) % (n * sizeof(T)) == 0 && s.b % n == 0 && s.h % n == 0 && s.s % n == 0 && s.r % n == 0;
}
template <class T>
int vec_flags(const Args& a, bool bwd) {
  return (vec_ok<T>(a.q, a.sq) ? VEC_Q : 0) | (vec_ok<T>(a.k, a.sk) ? VEC_K : 0) | (vec_ok<T>(a.v, a.sv) ? VEC_V : 0) |
         (bwd && vec_ok<T>(a.d_o, a.sdo) ? VEC_DO : 0);
}

template <class T, int DP>
cudaError_t launch_fwd_t(const Args& a, cudaStream_t st, int* launches) {
  auto kern = generic_fwd_kernel<T, DP>;
  if (!kernel_ready(reinterpret_cast<const void*>(kern), fwd_smem<DP>(), nullptr)) return cudaErrorUnknown;
  launch_dependent(kern, dim3(a.B * a.H * a.S, (a.R + TT - 1) / TT), NTH, fwd_smem<DP>(), st, a, vec_flags<T>(a, false));
  *launches += 1;
  return cudaGetLastError();
}

size_t delta_bytes(const Args& a) { return ((size_t)a.B * a.H * a.S * a.delta_ld * sizeof(float) + 255) / 256 * 256; }

template <class T, int DP>
cudaError_t launch_bwd_t(Args a, cudaStream_t st, int* launches) {
  const long long rows = (long long)a.B * a.H * a.S * a.R;
  if (a.dgate) {
    launch_dependent(generic_gate_backward_kernel<T>, dim3((unsigned)((rows + 7) / 8)), 256, 0, st, a);
    use_effective_d_o(&a);
  } else {
    launch_dependent(generic_delta_kernel<T>, dim3((unsigned)((rows + 31) / 32)), 256, 0, st, a);
  }
  auto kern = generic_bwd_kernel<T, DP>;
  if (!kernel_ready(reinterpret_cast<const void*>(kern), bwd_smem<DP>(), nullptr)) return cudaErrorUnknown;
  const Runs runs = plan_runs(a);
  float* part = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(a.delta) + delta_bytes(a));
  const long long nt = (a.R + TT - 1) / TT;
  const long long n_dq = (long long)a.B * a.H * runs.n * nt, n_total = n_dq + (long long)a.B * a.H * a.S * nt;
  const long long gx = n_total < (1 << 30) ? n_total : (1 << 30);
  launch_dependent(kern, dim3((unsigned)gx, (unsigned)((n_total + gx - 1) / gx)), NTH, bwd_smem<DP>(), st, a, vec_flags<T>(a, true), runs, part, n_dq,
                   n_total);
  *launches += 2;
  if (a.dbias && runs.n > 1) {
    const long long drows = (long long)a.B * a.H * a.R, blocks = (drows * a.R + 1023) / 1024;
    launch_dependent(generic_dbias_sum_kernel, dim3((unsigned)(blocks < 1184 ? blocks : 1184)), 256, 0, st, static_cast<const float*>(part), runs.n,
                     drows, a.R, a.dbias, a.dbias_ld);
    *launches += 1;
  }
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_fwd_d(const Args& a, cudaStream_t st, int* launches) {
  if (a.D <= 16) return launch_fwd_t<T, 16>(a, st, launches);
  if (a.D <= 32) return launch_fwd_t<T, 32>(a, st, launches);
  if (a.D <= 64) return launch_fwd_t<T, 64>(a, st, launches);
  return launch_fwd_t<T, 128>(a, st, launches);
}
template <class T>
cudaError_t launch_bwd_d(const Args& a, cudaStream_t st, int* launches) {
  if (a.D <= 16) return launch_bwd_t<T, 16>(a, st, launches);
  if (a.D <= 32) return launch_bwd_t<T, 32>(a, st, launches);
  if (a.D <= 64) return launch_bwd_t<T, 64>(a, st, launches);
  return launch_bwd_t<T, 128>(a, st, launches);
}

}  // namespace

size_t generic_bwd_workspace_bytes(const Args& a) {
  const Runs runs = plan_runs(a);
  return delta_bytes(a) + (a.dbias && runs.n > 1 ? (size_t)runs.n * a.B * a.H * a.R * a.R * sizeof(float) : 0);
}

cudaError_t launch_generic_fwd(int dtype, const Args& a, cudaStream_t st, int* launches) {
  switch (dtype) {
    case EVOATTN_BF16: return launch_fwd_d<__nv_bfloat16>(a, st, launches);
    case EVOATTN_FP16: return launch_fwd_d<__half>(a, st, launches);
    default: return launch_fwd_d<float>(a, st, launches);
  }
}

cudaError_t launch_generic_bwd(int dtype, const Args& a, cudaStream_t st, int* launches) {
  switch (dtype) {
    case EVOATTN_BF16: return launch_bwd_d<__nv_bfloat16>(a, st, launches);
    case EVOATTN_FP16: return launch_bwd_d<__half>(a, st, launches);
    default: return launch_bwd_d<float>(a, st, launches);
  }
}

}  // namespace evo
