// Host-side check of the general BBPGD solver's grid (bbpgd_solve in
// pcc_solver.cu): the library's own source, built by nvcc with the CUDA calls
// replaced by host stand-ins.  A cooperative launch may hold no more blocks
// than fit the device at once, and the plain and the traced kernel may fit
// differently, in whichever order one context runs them.  Prints "ok <cases>" or the
// first failure.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

static int g_fit_plain, g_fit_traced;  // blocks per SM
static const void* g_traced_kernel;
static const void* g_kernel;  // of the last cooperative launch
static int g_blocks;

template <class T>
static cudaError_t stand_in_malloc(T** p, size_t bytes, cudaStream_t) {
  *p = static_cast<T*>(calloc(bytes, 1));
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
static cudaError_t stand_in_free(void* p, cudaStream_t) { return free(p), cudaSuccess; }
static cudaError_t stand_in_copy(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
  return memcpy(dst, src, bytes), cudaSuccess;
}
static cudaError_t stand_in_copy_now(void* dst, const void* src, size_t bytes, cudaMemcpyKind) {
  return memcpy(dst, src, bytes), cudaSuccess;
}
static cudaError_t stand_in_set(void* p, int v, size_t bytes, cudaStream_t) { return memset(p, v, bytes), cudaSuccess; }
static cudaError_t stand_in_sync(cudaStream_t) { return cudaSuccess; }
static cudaError_t stand_in_last_error() { return cudaSuccess; }
static cudaError_t stand_in_occupancy(int* per_sm, const void* k, int, size_t) {
  *per_sm = k == g_traced_kernel ? g_fit_traced : g_fit_plain;
  return cudaSuccess;
}
static cudaError_t stand_in_cooperative(const void* k, dim3 grid, dim3, void**, size_t, cudaStream_t) {
  g_kernel = k;
  g_blocks = (int)grid.x;
  return cudaSuccess;
}

#define cudaMallocAsync stand_in_malloc
#define cudaFreeAsync stand_in_free
#define cudaMemcpyAsync stand_in_copy
#define cudaMemcpy stand_in_copy_now
#define cudaMemsetAsync stand_in_set
#define cudaStreamSynchronize stand_in_sync
#define cudaGetLastError stand_in_last_error
#define cudaOccupancyMaxActiveBlocksPerMultiprocessor stand_in_occupancy
#define cudaLaunchCooperativeKernel stand_in_cooperative
#include "pcc_solver.cu"

namespace pcc {
cudaError_t resident_bbpgd(pcc_ctx*, double, bool, bool, bool* taken, int*) { return *taken = false, cudaSuccess; }
cudaError_t order_incidence(pcc_ctx*) { return cudaSuccess; }
ConsView ConsBufs::view() { return {}; }
long long planar_chunks(size_t m) { return chunk_count((long long)m); }
}  // namespace pcc

int main() {
  g_traced_kernel = (const void*)pcc::k_bbpgd<1>;
  long long cases = 0;
  for (int plain = 1; plain <= 4; ++plain) {
    for (int traced = 1; traced <= 4; ++traced) {
      for (int first = 0; first < 2; ++first) {
        pcc_ctx* ctx = new pcc_ctx();
        ctx->num_sms = 148;
        ctx->n = 300000;
        ctx->ncons = 1000000;
        ctx->params.solver_variant = PCC_SOLVER_GENERAL;
        ctx->params.max_bbpgd_iterations = 10;
        ctx->status = new pcc::DevStatus();
        ctx->status_host = new pcc::DevStatus();
        g_fit_plain = plain;
        g_fit_traced = traced;
        for (int k = 0; k < 2; ++k, ++cases) {
          ctx->trace_active = k == first;
          ctx->params.log_bbpgd_trace = ctx->trace_active ? 2 : 0;
          long long it;
          double residual;
          int status;
          if (pcc::bbpgd_solve(ctx, 1e-3, &it, &residual, &status)) return printf("solve failed\n"), 1;
          const int fit = 148 * (ctx->trace_active ? traced : plain);
          if ((g_kernel == g_traced_kernel) != ctx->trace_active) return printf("the other kernel ran\n"), 1;
          if (g_blocks < 1 || g_blocks > fit)
            return printf("%s after the other: %d blocks where %d fit\n", ctx->trace_active ? "traced" : "plain",
                          g_blocks, fit),
                   1;
        }
      }
    }
  }
  printf("ok %lld\n", cases);
  return 0;
}
