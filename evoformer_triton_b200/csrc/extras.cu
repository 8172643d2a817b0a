// Small device passes around the attention kernels: the conversion of a pair bias (and its gradient)
// between the layout a linear layer emits, [B, R, R, H], and the [B, H, R, R] the kernels (and
// dsevoformer-triton/evoformer.py:638,652) use, and between dense and padded rows.
// None of this exists in the reference: it takes the bias heads-first.
#include <string.h>

#include "common.cuh"
#include "launch.h"
#include "ptx.cuh"

namespace evo {
namespace {

// [B,R,R,H] -> [B,H,R,ld >= R]: a block takes 128 keys of one (b, i) row: 128*H contiguous elements in,
// H runs of 128 contiguous elements out.
template <class E>
__global__ void __launch_bounds__(256) heads_first_kernel(const E* __restrict__ src, E* __restrict__ dst, int H, int R,
                                                          int ld) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  extern __shared__ unsigned char sm_raw[];
  E* sm = reinterpret_cast<E*>(sm_raw);
  const int j0 = blockIdx.x * 128, i = blockIdx.y, b = blockIdx.z;
  const int nj = min(128, R - j0);
  const E* in = src + (((long long)b * R + i) * R + j0) * H;
  for (int e = threadIdx.x; e < nj * H; e += 256) sm[e] = in[e];
  __syncthreads();
  for (int e = threadIdx.x; e < nj * H; e += 256) {
    const int h = e / nj, j = e - h * nj;
    dst[(((long long)b * H + h) * R + i) * ld + j0 + j] = sm[j * H + h];
  }
}

// fp32 [B,H,R,ld] -> [B,R,R,H] in type E (the one cast of the gradient happens here).
template <class E>
__global__ void __launch_bounds__(256) heads_last_kernel(const float* __restrict__ src, int ld, E* __restrict__ dst, int H,
                                                         int R) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  extern __shared__ unsigned char sm_raw[];
  float* sm = reinterpret_cast<float*>(sm_raw);
  const int j0 = blockIdx.x * 128, i = blockIdx.y, b = blockIdx.z;
  const int nj = min(128, R - j0);
  for (int e = threadIdx.x; e < nj * H; e += 256) {
    const int h = e / nj, j = e - h * nj;
    sm[j * H + h] = src[(((long long)b * H + h) * R + i) * ld + j0 + j];
  }
  __syncthreads();
  E* out = dst + (((long long)b * R + i) * R + j0) * H;
  for (int e = threadIdx.x; e < nj * H; e += 256) out[e] = from_float<E>(sm[e]);
}

// A pair bias with arbitrary (b, h, i) strides -> rows of R values with a row stride of `ld`, the form
// the tensor maps can read (whole 16-byte pieces).  All sizes in words of type W: the widest that divides
// rows, strides and addresses.  Bound by memory; a warp per row, four loads in flight per lane.  The last
// ld - R columns are never read and stay unwritten.
template <class W>
__global__ void __launch_bounds__(256) pad_rows_kernel(const W* __restrict__ src, Str3 st, W* __restrict__ dst, long long n_rows, int H,
                                                       int rows, int cols, int ld) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);  // (b, h, i): any number of (b, h)
  if (row >= n_rows) return;
  const int bh = (int)(row / rows), i = (int)(row - (long long)bh * rows);
  const W* in = src + (long long)(bh / H) * st.a + (long long)(bh % H) * st.b + (long long)i * st.c;
  W* out = dst + row * ld;
  for (int j = threadIdx.x & 31; j < cols; j += 128) {
    W v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (j + 32 * u < cols) v[u] = in[j + 32 * u];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (j + 32 * u < cols) out[j + 32 * u] = v[u];
  }
}
template <class W>
void pad_rows_t(const void* src, const int64_t* stride, void* dst, int es, int B, int H, int R, int ld, cudaStream_t st) {
  const int n = (int)sizeof(W) / es;  // elements per word
  const Str3 s{stride[0] / n, stride[1] / n, stride[2] / n};
  const long long rows = (long long)B * H * R;
  launch_dependent(pad_rows_kernel<W>, dim3((unsigned)((rows + 7) / 8)), 256, 0, st, static_cast<const W*>(src), s, static_cast<W*>(dst), rows, H, R, R / n, ld / n);
}

template <class E>
__global__ void __launch_bounds__(256) dbias_dense_kernel(const float* __restrict__ src, int ld, E* __restrict__ dst,
                                                          long long rows, int cols) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);  // a warp per row
  if (row >= rows) return;
  for (int j = threadIdx.x & 31; j < cols; j += 32) dst[row * cols + j] = from_float<E>(src[row * ld + j]);
}

template <class E>
void dbias_out_t(const Args& a, cudaStream_t st) {
  E* dst = reinterpret_cast<E*>(a.dbias_out);
  if (a.dbias_out_last) {
    dim3 grid((a.R + 127) / 128, a.R, a.B);
    launch_dependent(heads_last_kernel<E>, grid, 256, (size_t)128 * a.H * 4, st, static_cast<const float*>(a.dbias), a.dbias_ld, dst, a.H, a.R);
  } else {
    const long long rows = (long long)a.B * a.H * a.R;
    launch_dependent(dbias_dense_kernel<E>, dim3((unsigned)((rows + 7) / 8)), 256, 0, st, static_cast<const float*>(a.dbias), a.dbias_ld, dst, rows, a.R);
  }
}

}  // namespace

int launch_dbias_out(const Args& a, cudaStream_t st, int* launches) {
  switch (a.dbias_out_dtype) {
    case EVOATTN_BF16: dbias_out_t<__nv_bfloat16>(a, st); break;
    case EVOATTN_FP16: dbias_out_t<__half>(a, st); break;
    default: dbias_out_t<float>(a, st); break;
  }
  *launches += 1;
  return cudaGetLastError() == cudaSuccess ? EVOATTN_OK : EVOATTN_ERR_CUDA;
}

}  // namespace evo

extern "C" {

int evoattn_bias_to_heads_first(const void* src, void* dst, int dtype, int B, int H, int R, void* cuda_stream) {
  return evoattn_bias_to_heads_first_ld(src, dst, dtype, B, H, R, R, cuda_stream);
}

int evoattn_bias_pad_rows(const void* src, const int64_t* stride, void* dst, int dtype, int B, int H, int R, int ld,
                          void* cuda_stream) {
  if (!src || !dst || !stride) return EVOATTN_ERR_NULL;
  if (B <= 0 || H <= 0 || R <= 0 || ld < R || (long long)B * H > 0x7fffffffLL) return EVOATTN_ERR_SHAPE;
  if (((long long)B * H * R + 7) / 8 > 0x7fffffffLL) return EVOATTN_ERR_SHAPE;  // (blocks of eight rows)
  cudaStream_t st = reinterpret_cast<cudaStream_t>(cuda_stream);
  if (dtype != EVOATTN_FP32 && dtype != EVOATTN_BF16 && dtype != EVOATTN_FP16) return EVOATTN_ERR_DTYPE;
  const int es = dtype == EVOATTN_FP32 ? 4 : 2;
  const auto fits = [&](int bytes) {
    const uint64_t all = (uint64_t)(uintptr_t)src | (uintptr_t)dst | (uint64_t)(stride[0] * es) | (uint64_t)(stride[1] * es) |
                         (uint64_t)(stride[2] * es) | (uint64_t)(R * es) | (uint64_t)(ld * es);
    return all % bytes == 0;
  };
  if (fits(8)) evo::pad_rows_t<uint2>(src, stride, dst, es, B, H, R, ld, st);
  else if (fits(4)) evo::pad_rows_t<uint32_t>(src, stride, dst, es, B, H, R, ld, st);
  else evo::pad_rows_t<uint16_t>(src, stride, dst, es, B, H, R, ld, st);
  return cudaGetLastError() == cudaSuccess ? EVOATTN_OK : EVOATTN_ERR_CUDA;
}

int evoattn_bias_to_heads_first_ld(const void* src, void* dst, int dtype, int B, int H, int R, int ld, void* cuda_stream) {
  if (!src || !dst) return EVOATTN_ERR_NULL;
  if (ld < R) return EVOATTN_ERR_SHAPE;
  if (B <= 0 || H <= 0 || R <= 0 || H > 96 || B > 65535 || R > 65535) return EVOATTN_ERR_SHAPE;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(cuda_stream);
  dim3 grid((R + 127) / 128, R, B);
  if (dtype == EVOATTN_FP32)
    evo::launch_dependent(evo::heads_first_kernel<float>, grid, 256, (size_t)128 * H * 4, st, static_cast<const float*>(src), static_cast<float*>(dst), H, R, ld);
  else if (dtype == EVOATTN_BF16 || dtype == EVOATTN_FP16)
    evo::launch_dependent(evo::heads_first_kernel<uint16_t>, grid, 256, (size_t)128 * H * 2, st, static_cast<const uint16_t*>(src), static_cast<uint16_t*>(dst), H, R, ld);
  else
    return EVOATTN_ERR_DTYPE;
  return cudaGetLastError() == cudaSuccess ? EVOATTN_OK : EVOATTN_ERR_CUDA;
}

int evoattn_dbias_to_heads_last(const float* src, void* dst, int dtype, int B, int H, int R, void* cuda_stream) {
  if (!src || !dst) return EVOATTN_ERR_NULL;
  if (B <= 0 || H <= 0 || R <= 0 || H > 96 || B > 65535 || R > 65535) return EVOATTN_ERR_SHAPE;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(cuda_stream);
  dim3 grid((R + 127) / 128, R, B);
  const size_t smem = (size_t)128 * H * 4;
  if (dtype == EVOATTN_FP32) evo::launch_dependent(evo::heads_last_kernel<float>, grid, 256, smem, st, src, R, static_cast<float*>(dst), H, R);
  else if (dtype == EVOATTN_BF16) evo::launch_dependent(evo::heads_last_kernel<__nv_bfloat16>, grid, 256, smem, st, src, R, static_cast<__nv_bfloat16*>(dst), H, R);
  else if (dtype == EVOATTN_FP16) evo::launch_dependent(evo::heads_last_kernel<__half>, grid, 256, smem, st, src, R, static_cast<__half*>(dst), H, R);
  else return EVOATTN_ERR_DTYPE;
  return cudaGetLastError() == cudaSuccess ? EVOATTN_OK : EVOATTN_ERR_CUDA;
}

}  // extern "C"
