// launch_pdl() of the library over a fake of the runtime's launch call, for test_launch_host.py.
#include <cuda_runtime.h>

#include "p2r_launch.cuh"

namespace {
cudaError_t answer, pending;  // what the next launch returns; the thread's last error
int launches;
void kernel(int) {}
}  // namespace

extern "C" {

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) {
  ++launches;
  if (answer != cudaSuccess) pending = answer;
  return answer;
}

cudaError_t cudaGetLastError(void) {
  const cudaError_t e = pending;
  pending = cudaSuccess;
  return e;
}

// Launches once; returns launch_pdl's result and, in *left, the error that is pending afterwards.
int fake_launch(int result, int pending_before, int* left) {
  answer = (cudaError_t)result;
  pending = (cudaError_t)pending_before;
  launches = 0;
  const cudaError_t e = p2r::launch_pdl(kernel, dim3(1), 32, 0, nullptr, 1);
  *left = (int)pending;
  return launches == 1 ? (int)e : -1;
}

}  // extern "C"
