// Soft-model force assembly that allocates no device memory.
//
// Who needs this: a host that hands this library only memory it already owns
// and forbids it from allocating -- for instance a serving loop that admits
// colonies against a fixed HBM budget and accounts every byte through its own
// pool, or a latency-critical stepping loop that shares the GPU with other
// colonies' streams, where a cudaMalloc/cudaFree (cudaFree waits for the whole
// device) would stall work that is not its own.  pcc_soft_forces_noalloc takes
// the contacts and cell diameters in device buffers the caller owns and writes
// force/torque and stress into caller-owned device buffers.  Its intermediates
// (Hertz magnitudes, per-cell incidence lists) live in one file-scope device
// array, g_noalloc_scratch, of fixed size; nothing here calls cudaMalloc,
// cudaFree or any allocating library routine.
//
// Limits and sharing: at most kNoallocMaxCells cells and kNoallocMaxContacts
// contacts per call (larger calls return PCC_ERR_CAPACITY before touching the
// GPU).  Every gid_i / gid_j must be a cell index in [0, n): a contact with an
// id outside that range is skipped on the device (no scratch or output entry
// is touched for it), a flag in the scratch records it, and the call returns
// PCC_ERR_BOUNDS.  To read that flag the call waits for its own work on
// `stream` before it returns.  Every call on a device uses the same scratch
// array, which keeps the previous call's contents; the counters and the flag
// that must start at zero are cleared on the caller's stream at the start of
// each call.  Calls that overlap on the
// GPU (two streams, or two host threads) race on the scratch and must not be
// issued concurrently on one device.
//
// Every call resolves the device address of the scratch array with
// cudaGetSymbolAddress while its device is current (the host-side name of a
// __device__ array is only a stand-in and must never be passed to a kernel).
// With lazy module loading (the CUDA 12 default) the first call on a device,
// and the first launch of each kernel here, may also make the driver load this
// file's device code, which takes device memory of the driver's own; warm calls
// allocate nothing.
#include <cstdio>

#include "pcc_common.cuh"

namespace {

constexpr long long kNoallocMaxCells = 65536;
constexpr long long kNoallocMaxContacts = 393216;

// Scratch layout (bytes, each part 256-byte aligned):
//   fel       kNoallocMaxContacts doubles     Hertz force magnitudes
//   flag      1 unsigned                       out-of-range contact seen (cleared per call)
//   cnt       kNoallocMaxCells + 1 ints        incidence counts  (cleared per call, with the flag)
//   cursor    kNoallocMaxCells + 1 ints        fill cursors
//   off       kNoallocMaxCells + 1 ints        incidence offsets
//   ent       2 kNoallocMaxContacts ints       incidence entries (2c + side)
constexpr size_t align256(size_t b) { return (b + 255) / 256 * 256; }
constexpr size_t kFelBytes = align256(sizeof(double) * kNoallocMaxContacts);
constexpr size_t kCellIntBytes = align256(sizeof(int) * (kNoallocMaxCells + 1));
constexpr size_t kEntBytes = align256(sizeof(int) * 2 * kNoallocMaxContacts);
constexpr size_t kFlagBytes = 256;
constexpr size_t kScratchBytes = kFelBytes + 3 * kCellIntBytes + kEntBytes + kFlagBytes;  // 6.75 MiB

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

__device__ __forceinline__ double pow15_na(double x) {
  const double s = __dsqrt_rn(x);
  const double r = fma(-s, s, x);
  const double ds = r / (2.0 * s);
  const double p = x * s;
  const double pe = fma(x, s, -p);
  return p + (pe + x * ds);
}

// A contact whose ids are not both cell indices in [0, n) is left out.
__device__ __forceinline__ bool na_ids_ok(int a, int b, long long n) {
  return (unsigned)a < (unsigned long long)n && (unsigned)b < (unsigned long long)n;
}

__global__ void k_na_fel(const int* __restrict__ gi, const int* __restrict__ gj, const double* __restrict__ sd,
                         long long m, long long n, const double* __restrict__ diam, double kcc,
                         double* __restrict__ fel, int* __restrict__ cnt, unsigned* __restrict__ flag) {
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m) return;
  const int a = gi[c], b = gj[c];
  if (!na_ids_ok(a, b, n)) {
    fel[c] = 0.0;
    atomicOr(flag, 1u);
    return;
  }
  atomicAdd(&cnt[a], 1);
  atomicAdd(&cnt[b], 1);
  const double overlap = -sd[c];
  if (overlap <= 0.00) {
    fel[c] = 0.0;
    return;
  }
  const double R1 = pcc::dvd(diam[a], 2.0), R2 = pcc::dvd(diam[b], 2.0);
  const double R_eff = __dsqrt_rn(pcc::dvd(pcc::mul(R1, R2), pcc::add(R1, R2)));
  fel[c] = pcc::mul(pcc::mul(R_eff, kcc), pow15_na(overlap));
}

// Sum of one value per thread over a 256-thread block, to every thread, and
// the exclusive prefix of each thread.
__device__ __forceinline__ int na_block_scan(int v, int* sm, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) sm[warp] = x;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    before += w < warp ? sm[w] : 0;
    all += sm[w];
  }
  *total = all;
  return before + x - v;
}

// Exclusive scan of n+1 counts into offsets and fill cursors, one launch: a
// block takes kNaScanTile counts and adds up all counts before them itself (at
// most 65,536, from L2): 9.6 us at 37,000 cells (cold).  One block over all
// counts, each thread walking its
// own stretch, took 33 us.
constexpr int kNaScanTile = 2048;
__global__ void __launch_bounds__(256) k_na_scan(const int* __restrict__ cnt, int n, int* __restrict__ off,
                                                 int* __restrict__ cursor) {
  __shared__ int sm[8];
  const int b0 = (int)blockIdx.x * kNaScanTile;
  int s = 0, before;
  for (int i = 4 * (int)threadIdx.x; i < b0; i += 4 * 256) {
    const int4 v = *reinterpret_cast<const int4*>(cnt + i);
    s += v.x + v.y + v.z + v.w;
  }
  na_block_scan(s, sm, &before);
  const int base = b0 + 8 * (int)threadIdx.x;
  int v[8], own = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    v[k] = base + k < n + 1 ? cnt[base + k] : 0;
    own += v[k];
  }
  int total, run = na_block_scan(own, sm, &total) + before;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (base + k < n + 1) {
      off[base + k] = run;
      cursor[base + k] = run;
    }
    run += v[k];
  }
}

__global__ void k_na_fill(const int* __restrict__ gi, const int* __restrict__ gj, long long m, long long n,
                          int* __restrict__ cursor, int* __restrict__ ent) {
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m) return;
  const int a = gi[c], b = gj[c];
  if (!na_ids_ok(a, b, n)) return;
  ent[atomicAdd(&cursor[a], 1)] = (int)(2 * c);
  ent[atomicAdd(&cursor[b], 1)] = (int)(2 * c + 1);
}

// Eight lanes per cell: order its incidence entries by rank, then add the
// force, torque and stress of each overlapping contact in that order (the
// order of the reference's VecSetValues ADD stream per cell): the lanes form
// eight contacts' terms at once, which seven of them add up from shared
// memory, one sum each.  One thread per cell was a chain of dependent loads:
// 20 us at 37,000 cells (cold), now 15.6; the whole call 95 -> 56.
constexpr int kNaLanes = 8;
constexpr int kNaRanked = 32;  // entries that the lanes rank in registers; a longer list is sorted by one lane
__global__ void __launch_bounds__(256) k_na_gather(int n, const int* __restrict__ off, int* __restrict__ ent,
                                                   const double* __restrict__ sd, const double* __restrict__ normal,
                                                   const double* __restrict__ r_i, const double* __restrict__ r_j,
                                                   const double* __restrict__ s_i, const double* __restrict__ s_j,
                                                   const double* __restrict__ fel, double* __restrict__ force,
                                                   double* __restrict__ stress) {
  __shared__ double term[256 / kNaLanes][kNaLanes][8];  // force, torque, stress, 1 if the contact overlaps
  const int i = ((int)blockIdx.x * 256 + (int)threadIdx.x) / kNaLanes;
  const int lane = threadIdx.x & 31, l = lane % kNaLanes;
  const unsigned group = 0xffu << (lane - l);
  if (i >= n) return;  // whole groups
  double(*mine)[8] = term[threadIdx.x / kNaLanes];
  const int b = off[i], d = off[i + 1] - b;
  if (d <= kNaRanked) {
    int e[kNaRanked / kNaLanes], at[kNaRanked / kNaLanes];
#pragma unroll
    for (int q = 0; q < kNaRanked / kNaLanes; ++q) {
      const int k = l + q * kNaLanes;
      at[q] = -1;
      if (k >= d) continue;
      e[q] = ent[b + k];
      at[q] = 0;
      for (int o = 0; o < d; ++o) at[q] += ent[b + o] < e[q] ? 1 : 0;
    }
    __syncwarp(group);
#pragma unroll
    for (int q = 0; q < kNaRanked / kNaLanes; ++q)
      if (at[q] >= 0) ent[b + at[q]] = e[q];
  } else if (l == 0) {
    for (int k = b + 1; k < b + d; ++k) {
      int x = ent[k], j = k - 1;
      while (j >= b && ent[j] > x) {
        ent[j + 1] = ent[j];
        --j;
      }
      ent[j + 1] = x;
    }
  }
  __syncwarp(group);
  double sum = 0.0;
  for (int k0 = 0; k0 < d; k0 += kNaLanes) {
    if (k0 + l < d) {
      const int en = ent[b + k0 + l];
      const long long q = en >> 1;
      const bool sj = en & 1, in = !(-sd[q] <= 0.00);
      mine[l][7] = in ? 1.0 : 0.0;
      if (in) {
        const double fe = fel[q];
        const double* rr = sj ? r_j + 3 * q : r_i + 3 * q;
        double f[3], r[3], t[3];
        for (int x = 0; x < 3; ++x) {
          const double v = pcc::mul(normal[3 * q + x], fe);
          f[x] = sj ? -v : v;
          r[x] = rr[x];
        }
        pcc::cross3(r, f, t);
        for (int x = 0; x < 3; ++x) {
          mine[l][x] = f[x];
          mine[l][3 + x] = t[x];
        }
        mine[l][6] = pcc::mul(sj ? s_j[q] : s_i[q], fe);
      }
    }
    __syncwarp(group);
    const int c = d - k0 < kNaLanes ? d - k0 : kNaLanes;
    for (int x = 0; x < c; ++x)
      if (l < 7 && mine[x][7] != 0.0) sum = pcc::add(sum, mine[x][l]);
    __syncwarp(group);
  }
  if (l < 6) force[6 * (long long)i + l] = sum;
  if (l == 6) stress[i] = sum;
}

}  // namespace

extern "C" pcc_status pcc_soft_forces_noalloc(const int* gid_i, const int* gid_j, const double* sd,
                                              const double* normal, const double* r_i, const double* r_j,
                                              const double* stress_i, const double* stress_j, size_t m,
                                              const double* diameter, size_t n, double kcc, double* force,
                                              double* stress, void* stream) {
  if ((long long)n > kNoallocMaxCells || (long long)m > kNoallocMaxContacts) {
    std::fprintf(stderr,
                 "pcc_soft_forces_noalloc: %zu cells / %zu contacts exceed the fixed scratch "
                 "(at most %lld cells and %lld contacts)\n",
                 n, m, kNoallocMaxCells, kNoallocMaxContacts);
    return PCC_ERR_CAPACITY;
  }
  if (n == 0) return PCC_OK;
  if (!diameter || !force || !stress || (m && (!gid_i || !gid_j || !sd || !normal || !r_i || !r_j || !stress_i ||
                                               !stress_j)))
    return PCC_ERR_INVALID;
  // an error left pending by earlier work in the process is not this call's:
  // report it without launching (and without clearing it)
  if (cudaPeekAtLastError() != cudaSuccess) return PCC_ERR_CUDA;
  // asked at every call: the array belongs to the current CUDA context, which
  // the program may reset between calls
  void* base = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&base, g_noalloc_scratch);
  if (e != cudaSuccess || !base) {
    std::fprintf(stderr, "pcc_soft_forces_noalloc: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(e));
    return PCC_ERR_CUDA;
  }
  unsigned char* b = static_cast<unsigned char*>(base);
  double* fel = reinterpret_cast<double*>(b);
  unsigned* flag = reinterpret_cast<unsigned*>(b + kFelBytes);
  int* cnt = reinterpret_cast<int*>(b + kFelBytes + kFlagBytes);
  int* cursor = reinterpret_cast<int*>(b + kFelBytes + kFlagBytes + kCellIntBytes);
  int* off = reinterpret_cast<int*>(b + kFelBytes + kFlagBytes + 2 * kCellIntBytes);
  int* ent = reinterpret_cast<int*>(b + kFelBytes + kFlagBytes + 3 * kCellIntBytes);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the bounds flag and, right after it, the counters of the previous call must start at zero
  if (cudaMemsetAsync(flag, 0, kFlagBytes + sizeof(int) * (n + 1), s) != cudaSuccess) return PCC_ERR_CUDA;
  const int T = pcc::kBlock;
  if (m) {
    k_na_fel<<<pcc::grid_for((long long)m, T), T, 0, s>>>(gid_i, gid_j, sd, (long long)m, (long long)n, diameter, kcc,
                                                          fel, cnt, flag);
    if (cudaGetLastError() != cudaSuccess) return PCC_ERR_CUDA;
  }
  k_na_scan<<<(unsigned)(n / kNaScanTile + 1), 256, 0, s>>>(cnt, (int)n, off, cursor);
  if (cudaGetLastError() != cudaSuccess) return PCC_ERR_CUDA;
  if (m) {
    k_na_fill<<<pcc::grid_for((long long)m, T), T, 0, s>>>(gid_i, gid_j, (long long)m, (long long)n, cursor, ent);
    if (cudaGetLastError() != cudaSuccess) return PCC_ERR_CUDA;
  }
  k_na_gather<<<pcc::grid_for((long long)n * kNaLanes, 256), 256, 0, s>>>((int)n, off, ent, sd, normal, r_i, r_j,
                                                                          stress_i, stress_j, fel, force, stress);
  if (cudaGetLastError() != cudaSuccess) return PCC_ERR_CUDA;
  unsigned host_flag = 0;
  if (cudaMemcpyAsync(&host_flag, flag, sizeof host_flag, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return PCC_ERR_CUDA;
  return host_flag ? PCC_ERR_BOUNDS : PCC_OK;
}
