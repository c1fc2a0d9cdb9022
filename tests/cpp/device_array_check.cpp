// A device array whose allocation fails (no device, or far more memory than there is) is empty and
// leaves no error behind; the same array after a good allocation gives back what it held.
#include <cstdio>
#include <vector>

#include "synthesis.h"

int main() {
  sb::DeviceArray<double> a;
  int device = 0;
  const bool have = cudaGetDeviceCount(&device) == cudaSuccess && device > 0;
  cudaGetLastError();
  if (have) {
    a.allocate(100);
    if (a.p == nullptr || a.n != 100) {
      std::printf("a good allocation holds %zu values\n", a.n);
      return 1;
    }
  }
  bool thrown = false;
  try {
    a.allocate(static_cast<size_t>(1) << 58);
  }
  catch (const sb::Error &) {
    thrown = true;
  }
  if (!thrown || a.p != nullptr || a.n != 0) {
    std::printf("after a failed allocation: thrown %d, pointer %p, n %zu\n", thrown ? 1 : 0,
                static_cast<void*>(a.p), a.n);
    return 1;
  }
  std::printf("device array check passed\n");
  return 0;
}
