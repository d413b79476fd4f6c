// Test kernel for the whole-warp bounded wait: warp 0 of every block waits on a barrier with a limit given by the host, one
// thread of warp 1 completes it after a delay given per block (negative: never).  What each lane was told goes to `verdicts`.
#include "common.cuh"

namespace {

__global__ void wait_kernel(const long long* delays_ns, unsigned long long limit_ns, int* verdicts, int* flags) {
  __shared__ alignas(8) unsigned long long barrier;
  __shared__ int flag;
  const uint32_t bar = aima::smem_u32(&barrier);
  if (threadIdx.x == 0) {
    aima::mbar_init(bar, 1);
    flag = 0;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    verdicts[blockIdx.x * 32 + threadIdx.x] = aima::mbar_wait_bounded_warp(bar, 0, &flag, limit_ns) ? 1 : 0;
  } else if (threadIdx.x == 32 && delays_ns[blockIdx.x] >= 0) {
    const unsigned long long start = aima::global_timer_ns();
    for (int i = 0; i < 1000000 && aima::global_timer_ns() - start < static_cast<unsigned long long>(delays_ns[blockIdx.x]); ++i) {}
    aima::mbar_arrive(bar);
  }
  __syncthreads();
  if (threadIdx.x == 0) flags[blockIdx.x] = flag;
}

}  // namespace

extern "C" __attribute__((visibility("default"))) int run_wait_probe(const long long* delays_ns, unsigned long long limit_ns,
                                                                     int blocks, int* verdicts, int* flags) {
  wait_kernel<<<blocks, 64>>>(delays_ns, limit_ns, verdicts, flags);
  const cudaError_t launched = cudaGetLastError();
  return static_cast<int>(launched != cudaSuccess ? launched : cudaDeviceSynchronize());
}
