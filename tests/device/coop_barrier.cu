// The grid barrier of closure_coop.cuh: when a bounded wait ran out in one CTA,
// every CTA has to learn of it at the next barrier.  Every CTA arrives, so no wait
// runs out here.  Exit code 0, or the number of the case that failed.
#include <cstdio>

#include "../../simd2_b200/csrc/closure_coop.cuh"

using namespace simd2;

__global__ void probe(CoopCtl* ctl, int which, int* seen) {
  __shared__ int failed;
  if (threadIdx.x == 0) failed = (int)blockIdx.x == which;  // as sk_wait leaves it
  __syncthreads();
  coop_barrier(ctl, gridDim.x, &failed);
  if (threadIdx.x == 0) seen[blockIdx.x] = failed;
}

int main() {
  constexpr int kCtas = 12;
  CoopCtl* ctl;
  int* seen;
  if (cudaMalloc(&ctl, sizeof(CoopCtl)) != cudaSuccess || cudaMalloc(&seen, kCtas * sizeof(int)) != cudaSuccess) return 10;
  int c = 0;
  for (int which : {-1, 0, 5, kCtas - 1}) {
    c++;
    if (cudaMemset(ctl, 0, sizeof(CoopCtl)) != cudaSuccess) return 10;
    void* args[] = {&ctl, &which, &seen};
    if (cudaLaunchCooperativeKernel((void*)probe, dim3(kCtas), dim3(kSimtThreads), args, 0, 0) != cudaSuccess) return 10;
    int h[kCtas];
    if (cudaMemcpy(h, seen, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 10;
    for (int i = 0; i < kCtas; i++)
      if (h[i] != (which >= 0)) {
        std::printf("case %d: CTA %d of %d saw %d\n", c, i, kCtas, h[i]);
        return c;
      }
  }
  return 0;
}
