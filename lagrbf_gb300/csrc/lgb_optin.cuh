/*
 * lgb_optin.cuh -- the opt-in of a kernel to more than 48 KB of dynamic shared memory, per device.
 */
#pragma once

/* Opts the kernel in on the current device, once for each device of the process: `done` holds a bit per device and
   kernel.  Threads racing on it set the same attribute to the same value. */
template <typename Kernel> static inline int lgb_opt_in(Kernel kernel, int bytes, unsigned long long *done)
{
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (__atomic_load_n(done, __ATOMIC_ACQUIRE) & bit) return 0;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) __atomic_fetch_or(done, bit, __ATOMIC_RELEASE);
  return (int)e;
}
