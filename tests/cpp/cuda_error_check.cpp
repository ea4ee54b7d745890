// A CUDA call that the library reports as an error is not left behind as the
// thread's last error, which a later, unrelated check would take for its
// own.  The runtime's error state is faked here: no GPU, no driver.
#include <cstdio>

#include "../../lsim_b200/csrc/fsimb_internal.h"

static cudaError_t last = cudaSuccess;

extern "C" {
cudaError_t CUDARTAPI cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* CUDARTAPI cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "refused"; }
}

static cudaError_t refused() { return last = cudaErrorInvalidValue; }

int main() {
  bool threw = false;
  try {
    CK(refused());
  } catch (const fsimb::CudaError& e) {
    threw = e.msg.find("refused") != std::string::npos;
  }
  std::printf("%d %d\n", (int)threw, (int)last);
  return threw && last == cudaSuccess ? 0 : 1;
}
