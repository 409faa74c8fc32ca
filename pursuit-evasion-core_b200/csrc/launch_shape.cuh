// Launch shape of kernels whose dynamic shared memory depends on the call.
#pragma once
#include <cuda_runtime.h>

namespace pe {

// Let launches of `kernel` take all the dynamic shared memory a CTA can have.
// The limit belongs to the kernel and the device: were it set to one launch's
// size, a smaller launch of another handle or thread would lower it under a
// larger one that was configured before.
inline cudaError_t allow_all_smem(const void *kernel) {
  int device = 0, most = 0;
  cudaFuncAttributes attr{};
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, kernel);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             most - (int)attr.sharedSizeBytes);
  return e;
}

// SMs of the current device, and CTAs of `kernel` resident on each, for one
// block size and dynamic shared memory.
struct LaunchShape {
  int device = -1, threads = 0, sms = 0, resident = 0;
  size_t smem = 0;
};

// Bring `last` (a kernel's shape that this thread launched last) up to this
// launch's.
inline cudaError_t launch_shape(const void *kernel, int threads, size_t smem,
                                LaunchShape &last) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  if (last.device == device && last.threads == threads && last.smem == smem) return cudaSuccess;
  LaunchShape s{device, threads, 0, 0, smem};
  e = allow_all_smem(kernel);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&s.resident, kernel, threads, smem);
  if (e != cudaSuccess) return e;
  if (s.resident < 1) return cudaErrorInvalidConfiguration;
  last = s;
  return cudaSuccess;
}

// CTAs of one cooperative launch (0: the launch is not possible).
inline int cooperative_ctas(const void *kernel, int threads, size_t smem) {
  LaunchShape s;
  if (launch_shape(kernel, threads, smem, s) == cudaSuccess) return s.sms * s.resident;
  cudaGetLastError();  // the caller reports the refusal
  return 0;
}

}  // namespace pe
