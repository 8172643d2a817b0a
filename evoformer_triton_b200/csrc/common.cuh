// Shared device-side definitions for the Evoformer attention kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "evoattn.h"

namespace evo {

// Device status codes written to evoattn_fwd_params::status.
enum : int {
  DEV_OK = 0,
  DEV_TIMEOUT_TMA = 1,   // a wait for a TMA copy ran out
  DEV_TIMEOUT_MMA = 2,   // a wait for tcgen05.commit ran out
  DEV_TIMEOUT_SYNC = 3   // a wait between warps ran out
};

struct Str4 {
  long long b, h, s, r;
};
struct Str3 {
  long long a, b, c;
};

// Kernel arguments (by value).  Attention view [B,H,S,R,D]; D contiguous.
struct Args {
  int B, H, S, R, D;
  float scale;
  const void* q;
  const void* k;
  const void* v;
  void* o;          // forward: out; backward: in
  float* lse;       // [B,H,S,R]
  Str4 sq, sk, sv, so;
  const void* mask; // [B,S,R]
  int mask_kind;
  Str3 smask;       // (b,s,r)
  const float* bias;  // [B,H,R,R]; fp32, or (bias16 != 0) the q/k/v 16-bit type behind this pointer
  Str3 sbias;         // (b,h,i), in elements of the bias type
  int bias16;
  // backward only
  const void* d_o;
  void* dq;
  void* dk;
  void* dv;
  float* dbias;     // [B,H,R,dbias_ld] fp32: where the kernels sum d(pair_bias), or null
  int dbias_ld;
  // where it goes from there, if it is not the caller's own fp32 buffer already
  void* dbias_out;      // [B,H,R,R], or [B,R,R,H] if dbias_out_last
  int dbias_out_dtype;
  int dbias_out_last;
  float* delta;     // [B,H,S,delta_ld] (workspace)
  int delta_ld;     // R, or R rounded up to whole 16-byte rows where a tensor map reads it
  Str4 sdo, sdq, sdk, sdv;
  int* status;
  // gated output (optional): forward multiplies O by sigmoid(gate); backward gets dO of the gated output
  const void* gate;
  Str4 sgate;
  // backward of a gated output: d_o and o are the gated ones; the first kernel of a family writes the
  // gradient of the gate and the effective dO (contiguous), which the later ones read
  void* dgate;
  Str4 sdgate;
  void* d_o_eff;
  const void* exchange;  // backward: evoattn_peer_allreduce_params of the d(pair_bias) exchange, or null
  int max_runs;     // backward (CUDA-core kernels only): at most this many partial sums of d(pair_bias); 0: no limit
  float* dmask;     // backward (CUDA-core kernels only): gradient of an additive mask, [B,S,R] fp32
};

template <class T> __device__ __forceinline__ float to_float(T x);
template <> __device__ __forceinline__ float to_float<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <> __device__ __forceinline__ float to_float<__half>(__half x) { return __half2float(x); }

template <class T> __device__ __forceinline__ T from_float(float x);
template <> __device__ __forceinline__ float from_float<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_float<__half>(float x) { return __float2half_rn(x); }

// Two floats rounded to the 16-bit storage type, packed into one 32-bit word (first value low).
template <class T> struct Pack2;
template <> struct Pack2<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
};
template <> struct Pack2<__half> {
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
};

// The two 16-bit values of a 32-bit word, widened.
template <class T> __device__ __forceinline__ void unpack2(uint32_t w, float& lo, float& hi);
template <> __device__ __forceinline__ void unpack2<__nv_bfloat16>(uint32_t w, float& lo, float& hi) {
  lo = __uint_as_float(w << 16);
  hi = __uint_as_float(w & 0xffff0000u);
}
template <> __device__ __forceinline__ void unpack2<__half>(uint32_t w, float& lo, float& hi) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  lo = f.x;
  hi = f.y;
}

__device__ __forceinline__ long long off4(const Str4& s, int b, int h, int ss, int r) {
  return (long long)b * s.b + (long long)h * s.h + (long long)ss * s.s + (long long)r * s.r;
}

// Pair-bias element (b, h, i, j) in either storage type.
template <class T>
__device__ __forceinline__ float load_bias(const Args& a, int b, int h, int i, int j) {
  const long long idx = (long long)b * a.sbias.a + (long long)h * a.sbias.b + (long long)i * a.sbias.c + j;
  if (a.bias16) return to_float<T>(reinterpret_cast<const T*>(a.bias)[idx]);
  return a.bias[idx];
}
template <>
__device__ __forceinline__ float load_bias<float>(const Args& a, int b, int h, int i, int j) {
  return a.bias[(long long)b * a.sbias.a + (long long)h * a.sbias.b + (long long)i * a.sbias.c + j];
}

__device__ __forceinline__ float sigmoidf_fast(float x) { return 1.f / (1.f + __expf(-x)); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace evo
