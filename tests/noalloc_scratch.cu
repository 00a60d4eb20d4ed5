// Host-side check of pcc_soft_forces_noalloc's scratch (pcc_noalloc.cu, built
// by nvcc with the CUDA calls replaced by host stand-ins): every call works in
// the array that the current CUDA context holds, also after the context was
// reset and the array lies elsewhere.  No kernel runs.  Prints "ok" or the failure.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>

static void* g_array;    // where the context's array is
static void* g_cleared;  // what the call cleared
static size_t g_cleared_bytes;

static cudaError_t stand_in_symbol(void** p, const void*) { return *p = g_array, cudaSuccess; }
static cudaError_t stand_in_set(void* p, int, size_t bytes, cudaStream_t) {
  g_cleared = p;
  g_cleared_bytes = bytes;
  return cudaSuccess;
}
static cudaError_t stand_in_copy(void* dst, const void*, size_t bytes, cudaMemcpyKind, cudaStream_t) {
  return memset(dst, 0, bytes), cudaSuccess;
}
static cudaError_t stand_in_sync(cudaStream_t) { return cudaSuccess; }
static cudaError_t stand_in_device(int* d) { return *d = 0, cudaSuccess; }
static cudaError_t no_error() { return cudaSuccess; }

#define cudaGetSymbolAddress(p, symbol) stand_in_symbol(p, nullptr)
#define cudaMemsetAsync stand_in_set
#define cudaMemcpyAsync stand_in_copy
#define cudaStreamSynchronize stand_in_sync
#define cudaGetDevice stand_in_device
#define cudaGetLastError no_error
#define cudaPeekAtLastError no_error
#include "pcc_noalloc.cu"

int main() {
  static unsigned char first[kScratchBytes], second[kScratchBytes];
  double d[64] = {}, out[6 * 64], st[64];
  int id[4] = {};
  for (unsigned char* array : {first, second, first}) {
    g_array = array;
    const size_t n = 64;
    if (pcc_soft_forces_noalloc(id, id, d, d, d, d, d, d, 4, d, n, 1.0, out, st, nullptr) != PCC_OK)
      return printf("the call failed\n"), 1;
    const unsigned char* at = static_cast<unsigned char*>(g_cleared);
    if (at < array || at + g_cleared_bytes > array + kScratchBytes)
      return printf("the call worked in an array that is gone\n"), 1;
  }
  printf("ok\n");
  return 0;
}
