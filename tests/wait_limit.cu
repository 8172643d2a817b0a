// A CTA as the attention kernels have them (abort flag, bounded waits, one end), reduced to a single wait: thread 0
// goes straight to the end, and one warp waits on a barrier that is arrived on or not.
#include "common.cuh"
#include "ptx.cuh"

using namespace evo;

__global__ void wait_kernel(int waiting_warp, int arrive, int* status) {
  __shared__ uint64_t bar;
  __shared__ int flag;
  volatile int* abort_flag = &flag;
  if (threadIdx.x == 0) {
    ptx::mbar_init(&bar, 1);
    flag = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0 && arrive) ptx::mbar_arrive_s(ptx::smem_u32(&bar));
  if (static_cast<int>(threadIdx.x / 32) == waiting_warp) {
    ptx::mbar_wait_s(ptx::smem_u32(&bar), 0, ptx::smem_u32(&flag), DEV_TIMEOUT_MMA);
    // once one has run out, the others fall through
    for (int i = 0; !arrive && i < 8; ++i) ptx::mbar_wait_s(ptx::smem_u32(&bar), 0, ptx::smem_u32(&flag), DEV_TIMEOUT_SYNC);
  }
  ptx::end_of_cta(abort_flag, status);
}

extern "C" int run_wait_kernel(int waiting_warp, int arrive, int* status) {
  wait_kernel<<<1, 128>>>(waiting_warp, arrive, status);
  return static_cast<int>(cudaGetLastError());
}
