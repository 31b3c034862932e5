// A grid barrier that a block never reaches (grid_barrier, csrc/common.cuh, compiled with a short
// bound): every waiting block gets false and the flag is set.  Prints how many did, the flag, and
// how long the bound that the library is built with would last, in seconds.
#include <cstdio>

#include "common.cuh"

using namespace psc;

__global__ void k_wait(uint32_t* st, uint32_t* gave_up) {
  uint32_t target = 0;
  if (!grid_barrier(&st[0], &st[1], target)) return;  // all arrive here
  if (blockIdx.x == 0) return;                         // and not here
  if (!grid_barrier(&st[0], &st[1], target) && threadIdx.x == 0) atomicAdd(gave_up, 1u);
}

int main() {
  int sms = 0;
  uint32_t* st;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0) || cudaMalloc(&st, 64)) return 2;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  float ms = 0;
  uint32_t h[3] = {};
  for (int run = 0; run < 2; run++) {
    cudaMemset(st, 0, 64);
    uint32_t* gave_up = st + 8;
    void* args[] = {&st, &gave_up};
    cudaEventRecord(a);
    cudaLaunchCooperativeKernel((const void*)k_wait, dim3(sms), dim3(384), args, 0, nullptr);
    cudaEventRecord(b);
    if (cudaEventSynchronize(b) != cudaSuccess) return 3;
    cudaEventElapsedTime(&ms, a, b);
    cudaMemcpy(h, st, 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(h + 2, gave_up, 4, cudaMemcpyDeviceToHost);
  }
  std::printf("gave_up %u of %d failed %u seconds %.1f\n", h[2], sms - 1, h[1],
              1e-3 * ms / kGridSpin * kGridSpinDefault);
  return 0;
}
