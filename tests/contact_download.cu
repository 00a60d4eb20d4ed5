// Host-side check of the contact download (pcc_get_constraints in
// pcc_api.cu): the library's own source, built by nvcc with the CUDA calls it
// makes replaced by host stand-ins that copy at once, count what is still in
// flight and fail on request.  Whatever fails, the call must return an error
// with nothing in flight; if nothing fails, every array must arrive whole, also
// on a device too full for a scratch of its own, where the vectors go through
// several pieces.  Prints "ok <cases>" or the first failure.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

static int g_calls, g_fail_at, g_in_flight;  // g_fail_at: the call that fails, counted from 1 (0: none)
static bool g_full;  // no device memory is left
static bool fails() { return ++g_calls == g_fail_at; }

static cudaError_t stand_in_copy(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
  if (fails()) return cudaErrorUnknown;
  ++g_in_flight;
  memcpy(dst, src, bytes);
  return cudaSuccess;
}
static cudaError_t stand_in_sync(cudaStream_t) {
  g_in_flight = 0;
  return fails() ? cudaErrorUnknown : cudaSuccess;
}
template <class T>
static cudaError_t stand_in_malloc(T** p, size_t bytes, cudaStream_t) {
  if (g_full) return cudaErrorMemoryAllocation;
  *p = static_cast<T*>(malloc(bytes));  // kept: the program ends soon
  return cudaSuccess;
}

#define cudaMemcpyAsync stand_in_copy
#define cudaStreamSynchronize stand_in_sync
#define cudaMallocAsync stand_in_malloc
#include "pcc_api.cu"

namespace pcc {
cudaError_t interleave3(pcc_ctx*, const double* x, const double* y, const double* z, size_t n, double* out) {
  if (fails()) return cudaErrorUnknown;
  for (size_t k = 0; k < n; ++k) {
    out[3 * k] = x[k];
    out[3 * k + 1] = y[k];
    out[3 * k + 2] = z[k];
  }
  return cudaSuccess;
}
}  // namespace pcc

int main() {
  long long cases = 0;
  const size_t sizes[] = {1, 2, 63, 64, 65, 1000}, rooms[] = {0, 3, 64, 300, 3000, 5000};  // 0: the device has room
  for (size_t m : sizes) {
    for (size_t room : rooms) {
      pcc_ctx* ctx = new pcc_ctx();  // kept: its buffers are not device memory
      std::vector<std::vector<double>*> keep;
      auto column = [&](pcc::DevBuf<double>& b) {
        auto* v = new std::vector<double>(m + 1);
        for (size_t k = 0; k < m; ++k) (*v)[k] = 1000.0 * (double)keep.size() + (double)k;
        keep.push_back(v);
        b.p = v->data();
        b.cap = m + 1;
      };
      auto& c = ctx->cons;
      for (auto* b : {&c.sd, &c.gamma, &c.nx, &c.ny, &c.nz, &c.rix, &c.riy, &c.riz, &c.rjx, &c.rjy, &c.rjz, &c.cpx,
                      &c.cpy, &c.cpz, &c.si, &c.sj})
        column(*b);
      std::vector<int> ids[3];
      pcc::DevBuf<int>* ib[3] = {&c.gi, &c.gj, &c.phase};
      for (int q = 0; q < 3; ++q) {
        for (size_t k = 0; k < m; ++k) ids[q].push_back((int)(7 * k) + q);
        ib[q]->p = ids[q].data();
        ib[q]->cap = m;
      }
      g_full = room != 0;
      std::vector<double> scratch(room);
      ctx->pk.p = scratch.data();
      ctx->pk.cap = room;
      ctx->ncons = m;
      for (int at = 0;; ++at) {
        std::vector<int> gi(m), gj(m), ph(m);
        std::vector<double> sd(m), ga(m), si(m), sj(m), n(3 * m), ri(3 * m), rj(3 * m), cp(3 * m);
        pcc_contacts o;
        memset(&o, 0, sizeof o);
        o.gid_i = gi.data(), o.gid_j = gj.data(), o.phase = ph.data();
        o.sd = sd.data(), o.gamma = ga.data(), o.stress_i = si.data(), o.stress_j = sj.data();
        o.normal = n.data(), o.r_i = ri.data(), o.r_j = rj.data(), o.contact_point = cp.data();
        g_calls = g_in_flight = 0;
        g_fail_at = at;
        size_t got = 0;
        const pcc_status rc = pcc_get_constraints(ctx, &o, m, &got);
        ++cases;
        if (at && at > g_calls) break;  // past the last call: every one of them has failed once
        if (g_in_flight) return printf("m=%zu room=%zu, call %d fails: returned with copies in flight\n", m, room, at), 1;
        if (at && rc == PCC_OK) return printf("m=%zu room=%zu, call %d fails: no error\n", m, room, at), 1;
        if (at) continue;
        if (rc != PCC_OK || got != m) return printf("m=%zu room=%zu: status %d (%s)\n", m, room, rc, ctx->err.c_str()), 1;
        bool same = gi == ids[0] && gj == ids[1] && ph == ids[2];
        auto is = [&](const std::vector<double>& v, const pcc::DevBuf<double>& b) {
          for (size_t k = 0; k < m; ++k) same = same && v[k] == b.p[k];
        };
        auto are = [&](const std::vector<double>& v, const pcc::DevBuf<double>& x, const pcc::DevBuf<double>& y,
                       const pcc::DevBuf<double>& z) {
          for (size_t k = 0; k < m; ++k)
            same = same && v[3 * k] == x.p[k] && v[3 * k + 1] == y.p[k] && v[3 * k + 2] == z.p[k];
        };
        is(sd, c.sd), is(ga, c.gamma), is(si, c.si), is(sj, c.sj);
        are(n, c.nx, c.ny, c.nz), are(ri, c.rix, c.riy, c.riz), are(rj, c.rjx, c.rjy, c.rjz);
        are(cp, c.cpx, c.cpy, c.cpz);
        if (!same) return printf("m=%zu room=%zu: a value differs\n", m, room), 1;
      }
    }
  }
  printf("ok %lld\n", cases);
  return 0;
}
