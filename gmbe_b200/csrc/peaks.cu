// Measured memory peaks for the benchmark's roofline: the rate at which the
// SMs read a buffer that stays resident in L2.  No counterpart in the
// reference.  One launch makes `passes` grid-stride sweeps over the buffer
// with 16-byte loads that bypass L1 (ld.global.cg), so after a warm-up sweep
// every load is an L2 hit and the launch time is L2 read time.
#include <cuda_runtime.h>

#include <algorithm>

#include "engine.h"
#include "internal.h"
#include "mbe.h"

using namespace gmbe;

namespace {

__global__ void l2_read_kernel(const uint4* __restrict__ p, size_t n16, int passes,
                               unsigned* sink) {
  uint32_t acc = 0;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (int k = 0; k < passes; ++k) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride) {
      const uint4 v = __ldcg(p + i);
      acc ^= v.x ^ v.y ^ v.z ^ v.w;
    }
  }
  if (acc == 0x9e3779b9u) sink[0] = acc;  // keeps the loads; the buffer never holds it
}

}  // namespace

extern "C" int mbe_measure_l2_read(int32_t device, int64_t bytes, int32_t passes, double* gbs) {
  clear_error();
  if (!gbs || bytes < (1 << 20) || bytes > (int64_t(96) << 20) || passes < 1 || passes > 1000)
    return set_error(MBE_ERR_INVALID, "bytes must be 1-96 MiB and passes 1-1000");
  *gbs = 0;
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return set_error(MBE_ERR_CUDA, "cudaSetDevice: %s", cuda_error_text(e));
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const size_t n16 = (size_t)bytes / 16;
  uint4* buf = nullptr;
  unsigned* sink = nullptr;
  cudaStream_t st = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  float ms = 0;
  e = cudaMalloc((void**)&buf, n16 * 16);
  if (e == cudaSuccess) e = cudaMalloc((void**)&sink, sizeof(unsigned));
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&ev1);
  if (e == cudaSuccess) e = cudaMemsetAsync(buf, 0x5a, n16 * 16, st);
  const int blocks = std::max(sms, 1) * 4;
  if (e == cudaSuccess) {
    l2_read_kernel<<<blocks, 512, 0, st>>>(buf, n16, 2, sink);  // warm-up: brings it into L2
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaEventRecord(ev0, st);
  if (e == cudaSuccess) {
    l2_read_kernel<<<blocks, 512, 0, st>>>(buf, n16, passes, sink);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaEventRecord(ev1, st);
  if (e == cudaSuccess) e = cudaEventSynchronize(ev1);
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, ev0, ev1);
  if (ev0) cudaEventDestroy(ev0);
  if (ev1) cudaEventDestroy(ev1);
  if (st) cudaStreamDestroy(st);
  cudaFree(sink);
  cudaFree(buf);
  if (e != cudaSuccess) return set_error(MBE_ERR_CUDA, "L2 read measurement: %s", cuda_error_text(e));
  if (ms <= 0) return set_error(MBE_ERR_CUDA, "L2 read measurement: no elapsed time");
  *gbs = (double)n16 * 16.0 * passes / (ms / 1e3) / 1e9;
  return MBE_OK;
}
