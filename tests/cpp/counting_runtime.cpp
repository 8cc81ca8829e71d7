// A CUDA runtime for host-only checks: hands out addresses that nothing may touch, counts what is allocated,
// and accepts everything else that building a handle calls. Plain declarations (no CUDA headers).
#include <cstddef>
#include <cstdlib>

int mallocs = 0;
size_t malloc_bytes = 0, pool_bytes = 0;

static int give(void** p, size_t n) {
  static char* next = reinterpret_cast<char*>(size_t(1) << 40);
  *p = next;
  next += (n + 511) & ~size_t(511);
  return 0;
}

extern "C" {
int cudaMalloc(void** p, size_t n) {
  mallocs++;
  malloc_bytes += n;
  return give(p, n);
}
int cudaMallocFromPoolAsync(void** p, size_t n, void*, void*) {
  pool_bytes += n;
  return give(p, n);
}
int cudaMallocHost(void** p, size_t n) {
  *p = std::malloc(n);
  return 0;
}
int cudaFreeHost(void* p) {
  std::free(p);
  return 0;
}
int cudaOccupancyMaxActiveClusters(int* n, const void*, const void*) {
  *n = 1;
  return 0;
}
int cudaGetDevice(int* d) {
  *d = 0;
  return 0;
}
static int some(void** p) {
  *p = reinterpret_cast<void*>(size_t(16));
  return 0;
}
int cudaStreamCreateWithFlags(void** s, unsigned) { return some(s); }
int cudaEventCreateWithFlags(void** e, unsigned) { return some(e); }
int cudaFuncSetAttribute(const void*, int, int) { return 0; }
int cudaMemsetAsync(void*, int, size_t, void*) { return 0; }
int cudaMemcpyAsync(void*, const void*, size_t, int, void*) { return 0; }
int cudaStreamSynchronize(void*) { return 0; }
int cudaStreamDestroy(void*) { return 0; }
int cudaEventDestroy(void*) { return 0; }
int cudaFree(void*) { return 0; }
int cudaFreeAsync(void*, void*) { return 0; }
int cudaGetLastError() { return 0; }
const char* cudaGetErrorString(int) { return "error"; }
void** __cudaRegisterFatBinary(void*) {
  static void* handle = nullptr;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
