// Host memory that kernels read and write in place.
//
// Pinned and registered buffers have a device address. On hosts whose page tables the GPU uses
// (Grace, over NVLink-C2C: cudaDevAttrPageableMemoryAccess) any other host address works too, but
// only pages that are there are fast: the GPU's first touch of a missing page is a fault of its
// own (77 MB into a fresh buffer: 16.7 ms by the GPU's faults, 3.7 ms by cudaMemcpy, whose single
// thread takes the faults, 2.1 ms with the pages made by four threads first). And a page that the
// kernel may not read or write at all is a fault that ends the CUDA context, where a copy would have
// met an ordinary error of the host. So the pages of a pageable buffer are populated, for reading or
// for writing, before it is used in place, also those that are there: that is what asks the host
// whether they may be (pages of 64 KB that are there: 28 us for 77 MB in a row of such calls; a read
// back of 4 MB takes 98 us with it, 93 us without).
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <exception>
#include <new>
#include <thread>
#include <vector>

namespace lbm_b200 {

// Can kernels on `device` use ordinary host memory, atomics included?
inline bool host_memory_direct(int device) {
  int pageable = 0, atomics = 0;
  return cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, device) == cudaSuccess &&
         cudaDeviceGetAttribute(&atomics, cudaDevAttrHostNativeAtomicSupported, device) == cudaSuccess &&
         pageable && atomics;
}

// Makes the pages of [p, p + bytes) present (contents kept) by up to four threads for large buffers.
// False where the range is not mapped as a whole, may not be read (write: written), or that cannot
// be told.
inline bool host_pages_ready(void* p, size_t bytes, bool write) {
#if defined(__linux__) && defined(MADV_POPULATE_WRITE)
  try {
    const uintptr_t page = static_cast<uintptr_t>(sysconf(_SC_PAGESIZE));
    const uintptr_t lo = reinterpret_cast<uintptr_t>(p) / page * page;
    const uintptr_t hi = (reinterpret_cast<uintptr_t>(p) + bytes + page - 1) / page * page;
    // A thread costs about 20 us to start, a page about 10 us to make (48 fresh buffers of 0.1 to
    // 19 MB: 9.8 ms with a thread for each 2 MB, 11.9 ms for each 8 MB) and 0.02 us to look at.
    int n = 1;
    if (hi - lo > (2u << 20)) {
      std::vector<unsigned char> in((hi - lo) / page);
      if (mincore(reinterpret_cast<void*>(lo), hi - lo, in.data()) != 0) return false;
      const size_t missing = static_cast<size_t>(std::count_if(in.begin(), in.end(), [](unsigned char c) { return !(c & 1); }));
      n = static_cast<int>(std::min<size_t>(4, 1 + missing * page / (2u << 20) + (hi - lo) / (256u << 20)));
    }
    const uintptr_t share = ((hi - lo) / page + n - 1) / n * page;
    bool ok[4] = {true, true, true, true};
    auto part = [&](int k) {
      const uintptr_t a = std::min(hi, lo + k * share), b = std::min(hi, a + share);
      ok[k] = a == b || madvise(reinterpret_cast<void*>(a), b - a, write ? MADV_POPULATE_WRITE : MADV_POPULATE_READ) == 0;
    };
    std::vector<std::thread> more;
    more.reserve(4);
    int started = 1;
    try {
      for (; started < n; ++started) more.emplace_back(part, started);
    } catch (const std::exception&) {  // no thread, or no memory for one: this one does the rest
    }
    part(0);
    for (int k = started; k < n; ++k) part(k);
    for (std::thread& t : more) t.join();
    return ok[0] && ok[1] && ok[2] && ok[3];
  } catch (const std::bad_alloc&) {
    return false;
  }
#else
  (void)p;
  (void)bytes;
  (void)write;
  return false;
#endif
}

// The address under which kernels may use the host buffer [p, p + bytes) of `elem`-byte values, or
// null: it is then copied through device memory, which takes any alignment and any registration.
// Kernels load and store whole values, so the address has to be a multiple of `elem`; pinned or
// registered memory has to be so from the first byte to the last, at one range of device
// addresses. direct: host_memory_direct; output: the buffer will be written.
inline void* host_view(const void* p, size_t bytes, size_t elem, bool direct, bool output) {
  if (bytes == 0 || reinterpret_cast<uintptr_t>(p) % elem != 0) return nullptr;
  cudaPointerAttributes a{}, end{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (a.type == cudaMemoryTypeHost) {
    if (cudaPointerGetAttributes(&end, static_cast<const char*>(p) + bytes - 1) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    const uintptr_t first = reinterpret_cast<uintptr_t>(a.devicePointer), last = reinterpret_cast<uintptr_t>(end.devicePointer);
    const bool whole = end.type == cudaMemoryTypeHost && first != 0 && last == first + (bytes - 1);
    return whole && first % elem == 0 ? a.devicePointer : nullptr;
  }
  if (a.type != cudaMemoryTypeUnregistered || !direct) return nullptr;
  void* q = const_cast<void*>(p);
  return host_pages_ready(q, bytes, output) ? q : nullptr;
}

}  // namespace lbm_b200
