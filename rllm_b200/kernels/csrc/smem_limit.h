// A kernel that takes more than 48 KB of dynamic shared memory has to be allowed to, and the permission holds for the
// device that is current when it is given.  One SmemLimit a kernel, static at the launch: it remembers for every device how
// much was allowed there, so that a launch costs no more than asking for the current device.
#pragma once
#include <cuda_runtime.h>

struct SmemLimit {
  enum { DEVICES = 64 };
  int allowed[DEVICES] = {};
  // 0, or the CUDA error code.  Threads that meet here set the same limit twice at most.
  template <typename K> int allow(K kernel, size_t bytes) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    const bool known = dev >= 0 && dev < DEVICES;
    if (known && allowed[dev] >= (int)bytes) return 0;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    if (known) allowed[dev] = (int)bytes;
    return 0;
  }
};
