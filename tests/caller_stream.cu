// What a caller may have queued on its stream before a call: a slow kernel that starts its
// dependents at once and writes a field only at its end, and behind it a kernel that takes
// part in programmatic dependent launch without waiting for anything.
#include <cuda_runtime.h>

__global__ void slow_copy(double* dst, const double* src, long long n, long long cycles) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long t0 = clock64();
  while (clock64() - t0 < cycles) {  // bounded: the clock goes on
  }
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

__global__ void early() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

extern "C" int queue_slow_copy(double* dst, const double* src, long long n, long long cycles,
                               void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  slow_copy<<<32, 256, 0, st>>>(dst, src, n, cycles);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(32);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, early);
  return (int)cudaGetLastError();
}
