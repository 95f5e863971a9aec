// stage_check.cpp -- TEST INFRASTRUCTURE ONLY: stage_h2d (capi.cpp) on the host,
// with a stand-in for the copy and an allocator that gives out after a number of
// allocations of the calling thread.
#include <cstdlib>
#include <cstring>
#include <new>

#include "../../supergwas_b200/csrc/capi.cpp"

static thread_local int left = -1;  // allocations until the allocator throws; -1: never

void* operator new(std::size_t n) {
  if (left == 0) throw std::bad_alloc();
  if (left > 0) --left;
  void* p = std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}

// 0: copied and equal; 1: copied and not equal; 2: the call threw.
extern "C" int stage_call(uint64_t bytes, int allocations) {
  std::vector<char> src(bytes), stage(bytes), dst(bytes);
  for (size_t i = 0; i < bytes; ++i) src[i] = (char)(i * 31 >> 3);
  int rc = 0;
  left = allocations;
  try {
    kgctx::stage_h2d(dst.data(), stage.data(), src.data(), bytes, nullptr);
  } catch (const std::bad_alloc&) {
    rc = 2;
  }
  left = -1;
  return rc ? rc : std::memcmp(src.data(), dst.data(), bytes) != 0;
}
