// Host-side state shared by the entry points of libattn_b200.so.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

// One status word per device, allocated on first use and kept until process
// exit.  Kernels record the id of a wait that ran out here; a non-zero word
// makes every later kernel of this library return at once, until
// attn_b200_last_device_status() has read (and thereby cleared) it.
int* device_status_word(int device);

// SMs of the current device, 0 if it cannot be asked.
inline int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return sms;
}

// Launches a kernel that passes pdl_wait() before it touches memory (sm100.cuh has the rules): it may be made ready while the
// one in front of it in the stream still runs (behind anything but a kernel that calls pdl_launch_dependents() it starts as
// usual).  Two calls of 1 x 16 / 4 x 333 x 64 one after the other: 10.4 us each without, 8.2 with; the launches inside a
// training step likewise.
template <class... Expected, class... Actual>
inline bool launch_pdl(void (*kernel)(Expected...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Actual&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kernel, static_cast<Actual&&>(args)...) == cudaSuccess) return true;
  cudaGetLastError();
  return false;
}

}  // namespace b200
