// Host check of the grow-only device buffer (internal.cuh) with an allocator that
// fails on demand: a buffer whose growth failed is empty, not one that claims its
// former size without memory.
#include <cstdio>
#include <cstdlib>

#include "../../aran_gb300/csrc/internal.cuh"

static bool fail_next = false;
extern "C" cudaError_t cudaMalloc(void **p, size_t n) {
  *p = fail_next ? nullptr : std::malloc(n);
  return fail_next ? cudaErrorMemoryAllocation : cudaSuccess;
}
extern "C" cudaError_t cudaFree(void *p) {
  std::free(p);
  return cudaSuccess;
}

int main() {
  aran::DBuf<double> b;
  b.reserve(100);
  fail_next = true;
  bool thrown = false;
  try {
    b.reserve(100000);
  } catch (const aran::CudaError &e) {
    thrown = e.code == cudaErrorMemoryAllocation;
  }
  fail_next = false;
  const bool empty = b.ptr == nullptr && b.cap == 0;
  b.reserve(10);             // a later, smaller solve
  const bool usable = b.ptr != nullptr && b.cap >= 10;
  b.release();
  std::printf("%s\n", thrown && empty && usable ? "OK" : "FAIL");
  return thrown && empty && usable ? 0 : 1;
}
