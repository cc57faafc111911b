// How many SMs a stream's work may run on: all of the device's, or those of the green context
// (an SM partition) that the stream belongs to. A cooperative launch needs all its blocks resident at
// once and is refused where they are not.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

namespace lbm_b200 {

namespace stream_sms_detail {
struct Driver {
  CUresult (*stream_green)(CUstream, CUgreenCtx*) = nullptr;
  CUresult (*green_resource)(CUgreenCtx, CUdevResource*, CUdevResourceType) = nullptr;
  Driver() {
    auto find = [](const char* name) {
      cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
      void* p = nullptr;
      if (cudaGetDriverEntryPointByVersion(name, &p, 13000, cudaEnableDefault, &q) == cudaSuccess &&
          q == cudaDriverEntryPointSuccess)
        return p;
      cudaGetLastError();
      return static_cast<void*>(nullptr);
    };
    stream_green = reinterpret_cast<decltype(stream_green)>(find("cuStreamGetGreenCtx"));
    green_resource = reinterpret_cast<decltype(green_resource)>(find("cuGreenCtxGetDevResource"));
  }
};
}  // namespace stream_sms_detail

// device_sms where the stream is in no partition or that cannot be told. Asked for at each launch:
// the null stream's partition is that of the thread's current context.
inline int stream_sm_count(cudaStream_t stream, int device_sms) {
  static const stream_sms_detail::Driver driver;
  CUgreenCtx green = nullptr;
  CUdevResource r{};
  if (!driver.stream_green || !driver.green_resource || driver.stream_green(stream, &green) != CUDA_SUCCESS || !green ||
      driver.green_resource(green, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS)
    return device_sms;
  return std::min(device_sms, static_cast<int>(r.sm.smCount));
}

}  // namespace lbm_b200
