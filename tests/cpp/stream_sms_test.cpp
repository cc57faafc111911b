// Host check of csrc/stream_sms.h with a stand-in for the driver: the SM count of a stream in no
// partition, in one, and where the driver cannot tell. No GPU and no CUDA library involved. Exit
// status 0 when every answer is the expected one.
#include <cstdio>
#include <cstring>
#include <string>

#include "stream_sms.h"

namespace {
bool known = true;
CUresult green_result = CUDA_SUCCESS, resource_result = CUDA_SUCCESS;
unsigned partition = 0;  // SMs of the streams' green context; 0: none

CUresult stream_green(CUstream, CUgreenCtx* g) {
  *g = partition ? reinterpret_cast<CUgreenCtx>(&partition) : nullptr;
  return green_result;
}
CUresult green_resource(CUgreenCtx g, CUdevResource* r, CUdevResourceType t) {
  if (t != CU_DEV_RESOURCE_TYPE_SM || !g) return CUDA_ERROR_INVALID_VALUE;
  r->type = t;
  r->sm.smCount = partition;
  return resource_result;
}
}  // namespace

extern "C" {
cudaError_t CUDARTAPI cudaGetDriverEntryPointByVersion(const char* name, void** fn, unsigned, unsigned long long,
                                                       cudaDriverEntryPointQueryResult* q) {
  const bool a = !std::strcmp(name, "cuStreamGetGreenCtx"), b = !std::strcmp(name, "cuGreenCtxGetDevResource");
  *q = known && (a || b) ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  *fn = a ? reinterpret_cast<void*>(&stream_green) : reinterpret_cast<void*>(&green_resource);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
}

int main(int argc, char** argv) {
  known = !(argc > 1 && std::string(argv[1]) == "unknown");
  int bad = 0;
  auto expect = [&](int want, const char* what) {
    const int got = lbm_b200::stream_sm_count(nullptr, 152);
    if (got != want) std::printf("%s: %d SMs, not %d\n", what, got, want), ++bad;
  };
  expect(152, "no partition");
  partition = 16;
  expect(known ? 16 : 152, "a partition of 16");
  partition = 400;
  expect(152, "never more than the device's");
  partition = 16;
  resource_result = CUDA_ERROR_INVALID_CONTEXT;
  expect(152, "a partition that cannot be asked");
  resource_result = CUDA_SUCCESS;
  green_result = CUDA_ERROR_INVALID_HANDLE;
  expect(152, "a stream that cannot be asked");
  return bad == 0 ? 0 : 1;
}
