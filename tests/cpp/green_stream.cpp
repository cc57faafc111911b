// A stream on a partition of the GPU's SMs, for tests: the driver's documented green-context calls,
// reached through the driver library itself.
#include <cuda.h>
#include <dlfcn.h>

extern "C" int green_stream_create(unsigned sms, void** stream, void** ctx, unsigned* got) {
  void* lib = dlopen("libcuda.so.1", RTLD_NOW);
  if (!lib) return 1;
#define FN(name) auto p_##name = reinterpret_cast<decltype(&name)>(dlsym(lib, #name)); if (!p_##name) return 2
  FN(cuCtxGetDevice);
  FN(cuDeviceGetDevResource);
  FN(cuDevSmResourceSplitByCount);
  FN(cuDevResourceGenerateDesc);
  FN(cuGreenCtxCreate);
  FN(cuGreenCtxStreamCreate);
#undef FN
  CUdevice dev = 0;
  CUdevResource all{}, part{}, rest{};
  CUdevResourceDesc desc = nullptr;
  CUgreenCtx green = nullptr;
  CUstream s = nullptr;
  unsigned groups = 1;
  if (p_cuCtxGetDevice(&dev) != CUDA_SUCCESS || p_cuDeviceGetDevResource(dev, &all, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS ||
      p_cuDevSmResourceSplitByCount(&part, &groups, &all, &rest, 0, sms) != CUDA_SUCCESS || groups != 1 ||
      p_cuDevResourceGenerateDesc(&desc, &part, 1) != CUDA_SUCCESS ||
      p_cuGreenCtxCreate(&green, desc, dev, CU_GREEN_CTX_DEFAULT_STREAM) != CUDA_SUCCESS ||
      p_cuGreenCtxStreamCreate(&s, green, CU_STREAM_NON_BLOCKING, 0) != CUDA_SUCCESS)
    return 3;
  *stream = s;
  *ctx = green;
  *got = part.sm.smCount;
  return 0;
}

extern "C" int green_stream_destroy(void* stream, void* ctx) {
  void* lib = dlopen("libcuda.so.1", RTLD_NOW);
  auto sd = reinterpret_cast<CUresult (*)(CUstream)>(dlsym(lib, "cuStreamDestroy_v2"));
  auto gd = reinterpret_cast<CUresult (*)(CUgreenCtx)>(dlsym(lib, "cuGreenCtxDestroy"));
  return sd && gd && sd(static_cast<CUstream>(stream)) == CUDA_SUCCESS && gd(static_cast<CUgreenCtx>(ctx)) == CUDA_SUCCESS ? 0 : 1;
}
