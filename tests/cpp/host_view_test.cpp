// Host check of csrc/host_access.h with a stand-in for the CUDA runtime's pointer queries: which host
// buffers kernels are given in place, and which take a copy. No GPU and no CUDA library involved.
// Exit status 0 when every answer is the expected one.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <string>

#include "host_access.h"

namespace {
// Registered ranges: [lo, lo + bytes) with device address dev.
struct Range {
  uintptr_t lo;
  size_t bytes;
  uintptr_t dev;
};
Range ranges[2];
int range_count = 0;
// Allocations left before operator new fails (negative: no limit).
long allocations = -1;
}  // namespace

void* operator new(size_t n) {
  if (allocations == 0) throw std::bad_alloc();
  if (allocations > 0) --allocations;
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t CUDARTAPI cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  *a = cudaPointerAttributes{};
  a->type = cudaMemoryTypeUnregistered;
  const uintptr_t v = reinterpret_cast<uintptr_t>(p);
  for (int k = 0; k < range_count; ++k)
    if (v >= ranges[k].lo && v < ranges[k].lo + ranges[k].bytes) {
      a->type = cudaMemoryTypeHost;
      a->hostPointer = const_cast<void*>(p);
      a->devicePointer = reinterpret_cast<void*>(ranges[k].dev + (v - ranges[k].lo));
    }
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 1;
  return cudaSuccess;
}
}

namespace {
int bad = 0;
void expect(bool ok, const char* what) {
  if (ok) return;
  std::printf("wrong: %s\n", what);
  ++bad;
}

void pinned() {
  using lbm_b200::host_view;
  alignas(64) static unsigned char buf[4096];
  const uintptr_t base = reinterpret_cast<uintptr_t>(buf);
  const uintptr_t dev = uintptr_t(1) << 44;
  ranges[0] = {base, sizeof buf, dev};
  range_count = 1;
  for (bool direct : {false, true})
    for (bool output : {false, true}) {
      expect(host_view(buf, 1024, 4, direct, output) == reinterpret_cast<void*>(dev), "pinned: its device address");
      expect(host_view(buf + 8, 1024, 8, direct, output) == reinterpret_cast<void*>(dev + 8), "pinned at an aligned offset");
      expect(host_view(buf, sizeof buf, 4, direct, output) == reinterpret_cast<void*>(dev), "pinned: all of it");
      for (int off : {1, 2, 3, 5})
        expect(host_view(buf + off, 1024, 4, direct, output) == nullptr, "pinned, not aligned to 4-byte values");
      expect(host_view(buf + 4, 1024, 8, direct, output) == nullptr, "pinned, not aligned to 8-byte values");
      expect(host_view(buf + 8, 1024, 16, direct, output) == nullptr, "pinned, not aligned to 16-byte words");
      expect(host_view(buf, 0, 4, direct, output) == nullptr, "no bytes");
    }
  // A device address of another alignment than the host's.
  ranges[0] = {base, sizeof buf, dev + 2};
  expect(host_view(buf, 1024, 4, true, true) == nullptr, "device address not aligned");
  // A registration that ends inside the buffer, and one whose other half lies elsewhere.
  ranges[0] = {base, 1000, dev};
  expect(host_view(buf, 1024, 4, true, false) == nullptr, "registered in part");
  expect(host_view(buf, 1000, 4, true, false) == reinterpret_cast<void*>(dev), "registered to its end");
  ranges[0] = {base, 512, dev};
  ranges[1] = {base + 512, 512, dev + (1 << 20)};
  range_count = 2;
  expect(host_view(buf, 1024, 4, true, false) == nullptr, "two registrations, apart on the device");
  ranges[1].dev = dev + 512;
  expect(host_view(buf, 1024, 4, true, false) == reinterpret_cast<void*>(dev), "two registrations, one range");
  range_count = 0;
}

// Pageable memory that cannot be read or written: a copy reports that as an ordinary error of the
// host, so kernels do not get it.
void protection() {
  using lbm_b200::host_view;
  const size_t page = static_cast<size_t>(sysconf(_SC_PAGESIZE)), pages = 8, bytes = pages * page;
  auto map = [&](int fd = -1) {
    void* p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, fd < 0 ? MAP_PRIVATE | MAP_ANONYMOUS : MAP_SHARED, fd, 0);
    if (p == MAP_FAILED) std::exit(3);
    return static_cast<unsigned char*>(p);
  };
  unsigned char* p = map();
  expect(host_view(p, bytes, 4, true, true) == p, "fresh output: its pages are made");
  std::memset(p, 1, bytes);
  expect(host_view(p, bytes, 4, true, true) == p && host_view(p, bytes, 4, true, false) == p, "present pages");
  expect(host_view(p, bytes, 4, false, true) == nullptr, "pageable memory out of the device's reach");
  mprotect(p + 3 * page, page, PROT_READ);
  expect(host_view(p, bytes, 4, true, true) == nullptr, "output with a read-only page");
  expect(host_view(p, bytes, 4, true, false) == p, "input with a read-only page");
  expect(host_view(p, 3 * page, 4, true, true) == p, "output up to the read-only page");
  mprotect(p + 3 * page, page, PROT_NONE);
  expect(host_view(p, bytes, 4, true, false) == nullptr, "input with an inaccessible page");
  expect(host_view(p, bytes, 4, true, true) == nullptr, "output with an inaccessible page");
  for (size_t k = 0; k < bytes; k += page)
    if (k != 3 * page) expect(p[k] == 1, "contents kept");
  munmap(p, bytes);
  // A read-only mapping from the start, never touched.
  p = map();
  mprotect(p, bytes, PROT_READ);
  expect(host_view(p, bytes, 4, true, true) == nullptr, "fresh read-only output");
  munmap(p, bytes);
  // A hole.
  p = map();
  std::memset(p, 1, bytes);
  munmap(p + 2 * page, page);
  expect(host_view(p, bytes, 4, true, true) == nullptr && host_view(p, bytes, 4, true, false) == nullptr, "unmapped page");
  munmap(p, bytes);
  // A shared file that ends inside the mapping.
  std::FILE* f = std::tmpfile();
  if (!f || ftruncate(fileno(f), static_cast<off_t>(2 * page))) std::exit(3);
  p = map(fileno(f));
  std::memset(p, 1, 2 * page);
  expect(host_view(p, 2 * page, 4, true, true) == p, "file mapping up to its end");
  expect(host_view(p, bytes, 4, true, true) == nullptr, "output past the file's end");
  expect(host_view(p, bytes, 4, true, false) == nullptr, "input past the file's end");
  munmap(p, bytes);
  std::fclose(f);
}

// Memory that runs out at any of the allocations of a large buffer's preparation, also between the
// starts of its threads: an answer, no exception and no abort.
void allocation() {
  const size_t bytes = 32u << 20;
  int usable = 0;
  for (long limit = 0; limit < 12; ++limit) {
    void* p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED) std::exit(3);
    allocations = limit;
    void* v = nullptr;
    bool thrown = false;
    try {
      v = lbm_b200::host_view(p, bytes, 4, true, true);
    } catch (...) {
      thrown = true;
    }
    allocations = -1;
    expect(!thrown && (v == nullptr || v == p), "an answer without memory");
    usable += v == p;
    munmap(p, bytes);
  }
  expect(usable > 0 && usable < 12, "limits on both sides of what a preparation takes");
}
}  // namespace

int main(int argc, char** argv) {
  const std::string which = argc > 1 ? argv[1] : "";
  if (which == "pinned") pinned();
  else if (which == "protection") protection();
  else if (which == "allocation") allocation();
  else return 2;
  std::printf("%s: %d wrong\n", which.c_str(), bad);
  return bad == 0 ? 0 : 1;
}
