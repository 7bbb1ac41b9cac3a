// Included before the library's sources (nvcc -include): the CUDA calls that
// set a kernel's shared memory limit and that launch it are recorded, nothing
// runs.  A device of 152 SMs is reported.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <vector>

struct RecordedCall {
  const void *fn;
  long long bytes;  // the limit, or the dynamic shared memory of the launch
  int launch;
};
inline std::vector<RecordedCall> recorded;
inline std::mutex recorded_mutex;

inline cudaError_t record(const void *fn, long long bytes, int launch) {
  std::lock_guard<std::mutex> lock(recorded_mutex);
  recorded.push_back({fn, bytes, launch});
  return cudaSuccess;
}
template <typename F>
inline cudaError_t record_limit(F *fn, cudaFuncAttribute, int bytes) { return record((const void *)fn, bytes, 0); }
template <typename F>
inline cudaError_t record_launch(F *fn, dim3, dim3, void **, size_t smem, cudaStream_t) {
  return record((const void *)fn, (long long)smem, 1);
}
inline cudaError_t record_launch_ex(const cudaLaunchConfig_t *c, const void *fn, void **) {
  return record(fn, (long long)c->dynamicSmemBytes, 1);
}
template <typename F>
inline cudaError_t record_occupancy(int *blocks, F *, int, size_t) { *blocks = 2; return cudaSuccess; }
inline cudaError_t record_device(int *d) { *d = 0; return cudaSuccess; }
inline cudaError_t record_attribute(int *v, cudaDeviceAttr attr, int) {
  *v = attr == cudaDevAttrL2CacheSize ? 129 << 20 : 152;
  return cudaSuccess;
}

#define cudaFuncSetAttribute record_limit
#define cudaLaunchKernel record_launch
#define cudaLaunchKernelExC record_launch_ex
#define cudaOccupancyMaxActiveBlocksPerMultiprocessor record_occupancy
#define cudaGetDevice record_device
#define cudaDeviceGetAttribute record_attribute
#define cudaGetLastError() cudaSuccess
#define cudaMemsetAsync(...) cudaSuccess
#define cudaMemcpyAsync(...) cudaSuccess
#define cudaStreamSynchronize(...) cudaSuccess
#define cudaGetSymbolAddress(...) cudaErrorNotSupported

extern "C" inline __attribute__((used, visibility("default"))) long long recorded_count() { return (long long)recorded.size(); }
extern "C" inline __attribute__((used, visibility("default"))) void recorded_get(long long i, const void **fn, long long *bytes, int *launch) {
  *fn = recorded[i].fn;
  *bytes = recorded[i].bytes;
  *launch = recorded[i].launch;
}
