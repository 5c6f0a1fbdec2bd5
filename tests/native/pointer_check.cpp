// Host check of which caller pointers a kernel takes directly
// (csrc/kernels.cuh).  Built and run by tests/test_pointer_host.py.
#include <cstdio>

#include <cuda_runtime_api.h>

#include "../../gpu-spectral-channel-dns_b200/csrc/kernels.cuh"

static int takes(cudaMemoryType type, int owner, int dev, unsigned long long p) {
  cudaPointerAttributes a{};
  a.type = type;
  a.device = owner;
  return kernel_memory((const void*)p, a, dev);
}

int main() {
  for (int owner = 0; owner < 2; ++owner)
    for (int dev = 0; dev < 2; ++dev)
      for (unsigned long long p : {0x1000ull, 0x1008ull})
        printf("%d %d %d %d %d %d %d\n", owner, dev, (int)(p % 16), takes(cudaMemoryTypeDevice, owner, dev, p),
               takes(cudaMemoryTypeManaged, owner, dev, p), takes(cudaMemoryTypeHost, owner, dev, p),
               takes(cudaMemoryTypeUnregistered, owner, dev, p));
  return 0;
}
