// Two kernels around a library call: one ahead of it that lets its successor
// start at once and ends after a while, and one behind it that looks, before its
// own wait, at what has been done.
#include <cuda_runtime.h>

namespace {

__global__ void ahead(int* done, long long cycles) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const long long t0 = clock64();
  for (int i = 0; i < 1000000 && clock64() - t0 < cycles; ++i) {
  }
  *reinterpret_cast<volatile int*>(done) = 1;
}

__global__ void behind(const int* done, const double* v, double* seen) {
  seen[0] = *reinterpret_cast<const volatile int*>(done);
  seen[1] = *reinterpret_cast<const volatile double*>(v);
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  seen[2] = *reinterpret_cast<const volatile double*>(v);
}

}  // namespace

extern "C" int probe_ahead(int* done, long long cycles, cudaStream_t s) {
  ahead<<<1, 1, 0, s>>>(done, cycles);
  return cudaGetLastError();
}

extern "C" int probe_behind(const int* done, const double* v, double* seen, cudaStream_t s) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(1);
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, behind, done, v, seen);
  return cudaGetLastError();
}
