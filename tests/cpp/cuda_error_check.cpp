// A CUDA call that the library reports as an error is not left behind as the
// thread's last error, which a later, unrelated check would take for its own.
#include <cstdio>

#include "../../lsim_b200/csrc/fsimb_internal.h"

int main() {
  bool threw = false;
  try {
    CK(cudaSetDevice(4096));  // no such device
  } catch (const fsimb::CudaError& e) {
    threw = !e.msg.empty();
  }
  const cudaError_t left = cudaGetLastError();
  std::printf("%d %s\n", (int)threw, cudaGetErrorName(left));
  return threw && left == cudaSuccess ? 0 : 1;
}
