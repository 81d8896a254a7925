// A refused chained launch returns its error and leaves none behind for the
// launch check of an unrelated later call. The runtime refuses the launch (a
// block of 2048 threads): nothing reaches the GPU.
#include <cstdio>

#include "../perf_libs_sparse_b200/csrc/common.cuh"

__global__ void kernel(int) {}

int main() {
  const cudaError_t e = pls::launch_chained(kernel, 1, 2048, cudaStream_t(0), 0);
  const cudaError_t left = cudaGetLastError();
  std::printf("%s, left %s\n", cudaGetErrorName(e), cudaGetErrorName(left));
  return e != cudaSuccess && left == cudaSuccess ? 0 : 1;
}
