// Per-step cell updates (sm_100a): growth, division with device-side append
// of daughters, the x-sort that renumbers cells, colony radius and the CFL
// time-step adaptation.
#include <cmath>
#include <cstring>

#include "pcc_kernels.hpp"

namespace pcc {

namespace {

// ---------------------------------------------------------------- division draw
__host__ __device__ inline unsigned division_seed(unsigned long long seed, unsigned long long k) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ULL * (k + 1ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  z = z ^ (z >> 31);
  return (unsigned)(z & 0xffffffffULL);
}

// First two outputs of MT19937 seeded with s (Matsumoto & Nishimura's
// init_genrand, one in-place twist of words 0 and 1, tempering).
__host__ __device__ inline void mt19937_first_two(unsigned s, unsigned out[2]) {
  unsigned m0 = s, m1 = 0, m2 = 0, m397 = 0, m398 = 0, prev = s;
  for (unsigned i = 1; i < 399; ++i) {
    unsigned v = 1812433253u * (prev ^ (prev >> 30)) + i;
    if (i == 1) m1 = v;
    if (i == 2) m2 = v;
    if (i == 397) m397 = v;
    if (i == 398) m398 = v;
    prev = v;
  }
  const unsigned a[2] = {m0, m1}, b[2] = {m1, m2}, c[2] = {m397, m398};
  for (int k = 0; k < 2; ++k) {
    unsigned y = (a[k] & 0x80000000u) | (b[k] & 0x7fffffffu);
    unsigned v = c[k] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
    v ^= v >> 11;
    v ^= (v << 7) & 0x9d2c5680u;
    v ^= (v << 15) & 0xefc60000u;
    v ^= v >> 18;
    out[k] = v;
  }
}

#ifdef __CUDA_ARCH__
#define PCC_ADD(a, b) __dadd_rn(a, b)
#define PCC_MUL(a, b) __dmul_rn(a, b)
#define PCC_DIV(a, b) __ddiv_rn(a, b)
#else
#define PCC_ADD(a, b) ((a) + (b))
#define PCC_MUL(a, b) ((a) * (b))
#define PCC_DIV(a, b) ((a) / (b))
#endif

// Left-daughter length of the k-th division (simulation/Particle.cpp:128-135):
// std::uniform_real_distribution over [0.98, 1.02] * len/2 fed by
// std::mt19937 seeded with division_seed(seed, k); the canonical double is
// (x0 + x1 * 2^32) / 2^64 kept below 1 (two 32-bit draws for 53 bits).
__host__ __device__ inline double division_length(unsigned long long seed, unsigned long long k, double len) {
  unsigned x[2];
  mt19937_first_two(division_seed(seed, k), x);
  double sum = 0.0;
  sum = PCC_ADD(sum, PCC_MUL((double)x[0], 1.0));
  sum = PCC_ADD(sum, PCC_MUL((double)x[1], 4294967296.0));
  double u = PCC_DIV(sum, 18446744073709551616.0);
  if (u >= 1.0) u = 0.99999999999999988898;  // nextafter(1, 0)
  const double half = PCC_DIV(len, 2.0);
  const double a = PCC_MUL(half, 0.98), b = PCC_MUL(half, 1.02);
  return PCC_ADD(PCC_MUL(u, b - a), a);
}

__global__ void k_div_flag(const double* __restrict__ len, const double* __restrict__ l0, long long n,
                           int* __restrict__ flag) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  flag[i] = len[i] >= mul(2.0, l0[i]) ? 1 : 0;
}

// Particle::divide (simulation/Particle.cpp:122-150): the parent becomes the
// left daughter in place, the right daughter is appended at n + rank, where
// rank counts dividing cells in id order (ParticleManager::divideParticles,
// ParticleManager.cpp:139-148, and Domain::commitNewParticles, Domain.cpp:55-67).
__global__ void k_divide(CellsView c, long long n, const int* __restrict__ flag, const int* __restrict__ off,
                         unsigned long long seed, unsigned long long base) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !flag[i]) return;
  const long long k = off[i];
  const double len = c.len[i];
  const double l1 = division_length(seed, base + (unsigned long long)k, len);
  const double l2 = sub(len, l1);
  double t[3];
  cell_axis(c.q0[i], c.q1[i], c.q2[i], c.q3[i], t);
  const double h1 = dvd(l1, 2.0), h2 = dvd(l2, 2.0);
  const double p[3] = {c.x[i], c.y[i], c.z[i]};
  const long long j = n + k;
  c.x[j] = add(p[0], mul(t[0], h2));
  c.y[j] = add(p[1], mul(t[1], h2));
  c.z[j] = add(p[2], mul(t[2], h2));
  c.x[i] = sub(p[0], mul(t[0], h1));
  c.y[i] = sub(p[1], mul(t[1], h1));
  c.z[i] = sub(p[2], mul(t[2], h1));
  c.q0[j] = c.q0[i];
  c.q1[j] = c.q1[i];
  c.q2[j] = c.q2[i];
  c.q3[j] = c.q3[i];
  c.len[i] = l1;
  c.len[j] = l2;
  c.l0[j] = c.l0[i];
  c.diam[j] = c.diam[i];
  const int age = c.age[i] + 1;
  c.age[i] = age;
  c.age[j] = age;
  c.ncons[j] = 0;
  c.ldot[j] = 0.0;
  c.imp[j] = 0.0;
  c.stress[j] = 0.0;
  for (int d = 0; d < 6; ++d) {
    c.force[6 * j + d] = 0.0;
    c.vel[6 * j + d] = 0.0;
  }
}

__device__ __forceinline__ void move_cell(const CellsView& src, const CellsView& dst, long long i, long long j) {
  dst.x[j] = src.x[i];
  dst.y[j] = src.y[i];
  dst.z[j] = src.z[i];
  dst.q0[j] = src.q0[i];
  dst.q1[j] = src.q1[i];
  dst.q2[j] = src.q2[i];
  dst.q3[j] = src.q3[i];
  dst.len[j] = src.len[i];
  dst.l0[j] = src.l0[i];
  dst.diam[j] = src.diam[i];
  dst.ldot[j] = src.ldot[i];
  dst.imp[j] = src.imp[i];
  dst.stress[j] = src.stress[i];
  dst.age[j] = src.age[i];
  dst.ncons[j] = src.ncons[i];
  for (int d = 0; d < 6; ++d) {
    dst.force[6 * j + d] = src.force[6 * i + d];
    dst.vel[6 * j + d] = src.vel[6 * i + d];
  }
}

// Ranks by counting, for colonies of up to kRankMost cells: a block takes 32
// elements, its eight warps an eighth of every tile of keys each, and counts
// the keys below its own (below or equal among earlier elements: a stable
// order).  n^2 comparisons, but one launch; an LSD radix sort of the 64-bit
// keys is 8 x 3 launches whose latency is what a small colony pays for.
// Measured per x-sort: 225 us in 42 launches (2,474 cells) before.
constexpr int kRankMost = 16384;
constexpr int kRankRows = 32;
constexpr int kRankTile = 2048;

// Rank of element blockIdx.x * 32 + lane among n keys; all threads call, every
// warp returns it.  key(j) gives the key of element j.
template <class Key>
__device__ __forceinline__ int block_rank(int n, Key key, unsigned long long* tile, int* part,
                                          unsigned long long* own) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int base = (int)blockIdx.x * kRankRows, i = base + lane;
  const unsigned long long mine = i < n ? key(i) : 0ULL;
  *own = mine;
  int count = 0;
  for (int t0 = 0; t0 < n; t0 += kRankTile) {
    const int len = n - t0 < kRankTile ? n - t0 : kRankTile;
    __syncthreads();
    for (int j = threadIdx.x; j < len; j += kBlock) tile[j] = key(t0 + j);
    __syncthreads();
    const int per = (len + 7) / 8, lo = warp * per, hi = lo + per < len ? lo + per : len;
    // elements before this block's 32, the 32 themselves, elements after
    const int cut = base - t0 < lo ? lo : base - t0 > hi ? hi : base - t0;
    const int cut2 = base + kRankRows - t0 < cut ? cut : base + kRankRows - t0 > hi ? hi : base + kRankRows - t0;
#pragma unroll 8
    for (int j = lo; j < cut; ++j) count += tile[j] <= mine ? 1 : 0;
    for (int j = cut; j < cut2; ++j) count += (tile[j] < mine || (tile[j] == mine && t0 + j < i)) ? 1 : 0;
#pragma unroll 8
    for (int j = cut2; j < hi; ++j) count += tile[j] < mine ? 1 : 0;
  }
  part[warp * 32 + lane] = count;
  __syncthreads();
  int rank = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) rank += part[w * 32 + lane];
  return rank;
}

// The x-sort of a small colony: ranks, then every warp moves an eighth of the fields.
__global__ void __launch_bounds__(kBlock) k_rank_sort(CellsView src, CellsView dst, int n) {
  __shared__ unsigned long long tile[kRankTile];
  __shared__ int part[kBlock];
  unsigned long long own;
  const int j = block_rank(n, [&](int k) { return double_key(src.x[k]); }, tile, part, &own);
  const int i = (int)blockIdx.x * kRankRows + (int)(threadIdx.x & 31), warp = threadIdx.x >> 5;
  if (i >= n) return;
  const double* from[13] = {src.x, src.y, src.z, src.q0, src.q1, src.q2, src.q3,
                            src.len, src.l0, src.diam, src.ldot, src.imp, src.stress};
  double* to[13] = {dst.x, dst.y, dst.z, dst.q0, dst.q1, dst.q2, dst.q3,
                    dst.len, dst.l0, dst.diam, dst.ldot, dst.imp, dst.stress};
#pragma unroll
  for (int f = 0; f < 13; ++f)
    if ((f & 7) == warp) to[f][j] = from[f][i];
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    if (d == warp) {
      dst.force[6 * (long long)j + d] = src.force[6 * (long long)i + d];
      dst.vel[6 * (long long)j + d] = src.vel[6 * (long long)i + d];
    }
  }
  if (warp == 6) dst.age[j] = src.age[i];
  if (warp == 7) dst.ncons[j] = src.ncons[i];
}

// The x-sort of a larger colony: two buckets per cell over [-r, r] in x (r the
// colony radius; cells beyond it fall in the end buckets), then each cell's
// rank among its bucket's cells by (key, index).  Buckets hold about half a
// cell each; five launches where a radix sort of the 64-bit keys takes 24.  A
// bucket of k cells costs k comparisons for each of them, so a colony with
// more than kBucketMost cells in one (a tall one whose cells share few x, one
// stretched by a far outlier) takes the radix sort, whose cost does not depend
// on the keys.  Steps of separate cells, buckets / radix, ms, by the cells in
// each bucket: 17,000 cells, 4,000 0.46 / 0.28, 1,000 0.26 / 0.27; 300,000
// cells, 300,000 69.0 / 0.50, 9,000 2.44 / 0.51, 1,000 0.60 / 0.52, 700
// 0.53 / 0.52, 400 0.45 / 0.52; 1,000,000 cells, 2,000 2.23 / 1.07, 700
// 1.31 / 1.06, 400 1.09 / 1.06.
constexpr int kBucketMost = 256;
struct Buckets {
  double lo, scale;
  int count;
  __device__ __forceinline__ int of(double x) const {
    const double b = (x - lo) * scale;
    if (!(b == b)) return (double_key(x) >> 63) ? count - 1 : 0;  // not a number: first or last, as its key sorts
    return b <= 0.0 ? 0 : b >= (double)(count - 1) ? count - 1 : (int)b;
  }
};

__global__ void k_bucket_count(const double* __restrict__ x, long long n, Buckets bk, int* __restrict__ cnt,
                               int* __restrict__ arrival, int* __restrict__ crowded) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int at = atomicAdd(&cnt[bk.of(x[i])], 1);
  arrival[i] = at;
  if (at == kBucketMost) *crowded = 1;
}

__global__ void k_bucket_place(const double* __restrict__ x, long long n, Buckets bk, const int* __restrict__ off,
                               const int* __restrict__ arrival, const int* __restrict__ crowded,
                               int* __restrict__ cells, DevStatus* st) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) st->crowded = *crowded;
  if (i < n) cells[off[bk.of(x[i])] + arrival[i]] = (int)i;
}

// skip: leave dst alone if the buckets are crowded (the host then sorts by radix); null: sort them all the same.
__global__ void k_bucket_gather(CellsView src, CellsView dst, long long n, Buckets bk, const int* __restrict__ off,
                                const int* __restrict__ cells, const int* __restrict__ skip) {
  const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n || (skip && *skip)) return;
  const int i = cells[s];
  const double x = src.x[i];
  const unsigned long long mine = double_key(x);
  const int b = bk.of(x), lo = off[b], hi = off[b + 1];
  int j = lo;
  for (int k = lo; k < hi; ++k) {
    const int o = cells[k];
    const unsigned long long key = double_key(src.x[o]);
    j += (key < mine || (key == mine && o < i)) ? 1 : 0;
  }
  move_cell(src, dst, i, j);
}

__global__ void k_x_keys(const double* __restrict__ x, long long n, unsigned long long* __restrict__ keys,
                         int* __restrict__ perm) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = double_key(x[i]);
  perm[i] = (int)i;
}

__global__ void k_gather_cells(CellsView src, CellsView dst, const int* __restrict__ perm, long long n) {
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) move_cell(src, dst, perm[j], j);
}

// Distance of a cell's far end from the origin (spatial/Domain.cpp:148-153).
__device__ __forceinline__ double end_distance(const CellsView& c, long long i, double len) {
  double t[3];
  cell_axis(c.q0[i], c.q1[i], c.q2[i], c.q3[i], t);
  const double half = sub(dvd(len, 2.0), dvd(c.diam[i], 2.0));
  const double e[3] = {add(c.x[i], mul(t[0], half)), add(c.y[i], mul(t[1], half)), add(c.z[i], mul(t[2], half))};
  return __dsqrt_rn(dot3(e, e));
}

__device__ __forceinline__ void warp_max_into(unsigned long long* dst, double m) {
  for (int o = 16; o > 0; o >>= 1) {
    double w = __shfl_down_sync(0xffffffffu, m, o);
    m = m < w ? w : m;
  }
  if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(dst, (unsigned long long)__double_as_longlong(m));
}

// Growth; at the end of a step (kEnd) also the colony radius and the division
// flags, which need the grown lengths: one pass over the cells instead of three.
template <bool kEnd>
__global__ void k_grow(CellsView c, long long n, double dt, int* __restrict__ flag, DevStatus* st) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double m = 0.0;
  if (i < n) {
    double l = add(c.len[i], mul(dt, c.ldot[i]));
    const double cap = mul(2.0, c.l0[i]);
    if (l > cap) l = cap;
    c.len[i] = l;
    if constexpr (kEnd) {
      flag[i] = l >= cap ? 1 : 0;
      m = end_distance(c, i, l);
    }
  }
  if constexpr (kEnd) warp_max_into(&st->radius_bits, m);
}

__global__ void k_radius(CellsView c, long long n, DevStatus* st) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  warp_max_into(&st->max_bits, i < n ? end_distance(c, i, c.len[i]) : 0.0);
}

// |v| + ldot per cell as an ordered key (Domain::adaptDt, spatial/Domain.cpp:73-77)
__device__ __forceinline__ unsigned long long speed_key(const CellsView& c, long long i) {
  const double* v = c.vel + 6 * i;
  const double vv[3] = {v[0], v[1], v[2]};
  return double_key(add(__dsqrt_rn(dot3(vv, vv)), c.ldot[i]));
}

__global__ void k_speed_keys(CellsView c, long long n, unsigned long long* __restrict__ keys, int* __restrict__ vals) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = speed_key(c, i);
  vals[i] = (int)i;
}

// The keys of ranks lo and lo + 1 of a small colony's speeds.
__global__ void __launch_bounds__(kBlock) k_rank_median(CellsView c, int n, int lo, DevStatus* st) {
  __shared__ unsigned long long tile[kRankTile];
  __shared__ int part[kBlock];
  unsigned long long own;
  const int r = block_rank(n, [&](int k) { return speed_key(c, k); }, tile, part, &own);
  const int i = (int)blockIdx.x * kRankRows + (int)(threadIdx.x & 31);
  if (threadIdx.x < 32 && i < n && (r == lo || r == lo + 1)) st->median[r - lo] = own;
}

double key_to_double(unsigned long long k) {
  unsigned long long b = (k & 0x8000000000000000ULL) ? (k & 0x7fffffffffffffffULL) : ~k;
  double d;
  std::memcpy(&d, &b, sizeof d);
  return d;
}

}  // namespace

cudaError_t reset_ldot(pcc_ctx* ctx) {
  if (!ctx->n) return cudaSuccess;
  return cudaMemsetAsync(ctx->cells.ldot.p, 0, ctx->n * sizeof(double), ctx->stream);
}

cudaError_t grow_cells(pcc_ctx* ctx, double dt, bool step_end) {
  cudaStream_t s = ctx->stream;
  const size_t n = ctx->n;
  if (step_end) cudaMemsetAsync(&ctx->status->radius_bits, 0, sizeof(unsigned long long), s);
  if (!n) return cudaSuccess;
  if (step_end) {
    cudaError_t e;
    if ((e = ctx->div_flag.reserve(n + 1, 0, s))) return e;
    k_grow<true><<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), (long long)n, dt, ctx->div_flag.p, ctx->status);
  } else {
    k_grow<false><<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), (long long)n, dt, nullptr, ctx->status);
  }
  ctx->launches++;
  return cudaGetLastError();
}

cudaError_t divide_cells(pcc_ctx* ctx, size_t* added) {
  cudaStream_t s = ctx->stream;
  const size_t n = ctx->n;
  cudaError_t e;
  *added = 0;
  if (!n) return cudaSuccess;
  size_t k;
  if (ctx->div_known) {  // counted at the end of the previous step, on these very cells
    k = ctx->div_next;
  } else {
    if ((e = ctx->div_flag.reserve(n + 1, 0, s)) || (e = ctx->div_off.reserve(n + 1, 0, s))) return e;
    k_div_flag<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.len.p, ctx->cells.l0.p, (long long)n, ctx->div_flag.p);
    ctx->launches++;
    if ((e = exclusive_scan(ctx, ctx->div_flag.p, ctx->div_off.p, n))) return e;
    if ((e = cudaMemcpyAsync(ctx->pinned_ll + kSlotDivs, ctx->div_off.p + n, sizeof(int), cudaMemcpyDeviceToHost, s)))
      return e;
    if ((e = cudaStreamSynchronize(s))) return e;
    k = (size_t) * reinterpret_cast<int*>(ctx->pinned_ll + kSlotDivs);
  }
  ctx->div_known = false;
  if (!k) return cudaSuccess;
  if ((e = ctx->cells.reserve(n + k, n, s))) return e;
  k_divide<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), (long long)n, ctx->div_flag.p, ctx->div_off.p,
                                          ctx->params.seed, ctx->div_index);
  ctx->launches++;
  ctx->div_index += k;
  ctx->n = n + k;
  *added = k;
  return cudaGetLastError();
}

cudaError_t sort_cells_by_x(pcc_ctx* ctx) {
  cudaStream_t s = ctx->stream;
  const size_t n = ctx->n;
  cudaError_t e;
  if (n <= 1) return cudaSuccess;
  if ((e = ctx->cells_alt.reserve(n, 0, s))) return e;
  if (n <= (size_t)kRankMost) {
    k_rank_sort<<<grid_for((long long)n, kRankRows), kBlock, 0, s>>>(ctx->cells.view(), ctx->cells_alt.view(), (int)n);
    ctx->launches++;
  } else {
    const double r = ctx->radius > 0 && std::isfinite(ctx->radius) ? ctx->radius : 1.0;
    Buckets bk;
    bk.count = (int)(2 * n);
    bk.lo = -r;
    bk.scale = bk.count / (2.0 * r);
    if ((e = ctx->perm.reserve(n, 0, s)) || (e = ctx->perm_alt.reserve(n, 0, s)) ||
        (e = ctx->sort_hist.reserve(2 * (size_t)bk.count + 2, 0, s)))
      return e;
    int *cnt = ctx->sort_hist.p, *crowded = cnt + bk.count, *off = crowded + 1;
    // the first such sort since the upload asks whether the buckets are crowded
    // (the answer comes while the sort runs), a later one goes by the step before
    const bool ask = ctx->x_crowded < 0;
    int* flag = reinterpret_cast<int*>(ctx->pinned_ll + kSlotCrowded);
    if (ctx->x_crowded <= 0) {
      cudaMemsetAsync(cnt, 0, (bk.count + 1) * sizeof(int), s);
      k_bucket_count<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.x.p, (long long)n, bk, cnt, ctx->perm_alt.p, crowded);
      if (ask) {
        if (!ctx->x_ev && (e = cudaEventCreateWithFlags(&ctx->x_ev, cudaEventDisableTiming))) return e;
        if ((e = cudaMemcpyAsync(flag, crowded, sizeof(int), cudaMemcpyDeviceToHost, s)) ||
            (e = cudaEventRecord(ctx->x_ev, s)))
          return e;
      }
      if ((e = exclusive_scan(ctx, cnt, off, bk.count))) return e;
      k_bucket_place<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.x.p, (long long)n, bk, off, ctx->perm_alt.p, crowded,
                                                    ctx->perm.p, ctx->status);
      k_bucket_gather<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), ctx->cells_alt.view(), (long long)n, bk, off,
                                                    ctx->perm.p, ask ? crowded : nullptr);
      ctx->launches += 3;
    }
    if (ask) {
      if ((e = cudaEventSynchronize(ctx->x_ev))) return e;
      ctx->x_crowded = *flag;
    }
    if (ctx->x_crowded > 0) {
      if ((e = ctx->keys.reserve(n, 0, s))) return e;
      k_x_keys<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.x.p, (long long)n, ctx->keys.p, ctx->perm.p);
      if ((e = radix_sort_pairs(ctx, ctx->keys.p, ctx->perm.p, n, 64))) return e;
      k_gather_cells<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), ctx->cells_alt.view(), ctx->perm.p,
                                                    (long long)n);
      ctx->launches += 2;
    }
  }
  ctx->cells.swap(ctx->cells_alt);
  return cudaGetLastError();
}

cudaError_t colony_radius(pcc_ctx* ctx, double* out) {
  cudaStream_t s = ctx->stream;
  cudaMemsetAsync(&ctx->status->max_bits, 0, sizeof(unsigned long long), s);
  if (ctx->n) {
    k_radius<<<grid_for(ctx->n), kBlock, 0, s>>>(ctx->cells.view(), (long long)ctx->n, ctx->status);
    ctx->launches++;
  }
  cudaError_t e = cudaMemcpyAsync(ctx->pinned_ll + kSlotRadius, &ctx->status->max_bits, sizeof(unsigned long long),
                                  cudaMemcpyDeviceToHost, s);
  if (!e) e = cudaStreamSynchronize(s);
  if (e) return e;
  std::memcpy(out, ctx->pinned_ll + kSlotRadius, sizeof *out);
  return cudaSuccess;
}

cudaError_t step_end_enqueue(pcc_ctx* ctx) {
  cudaStream_t s = ctx->stream;
  const size_t n = ctx->n;
  cudaError_t e;
  if ((e = ctx->div_flag.reserve(n + 1, 0, s)) || (e = ctx->div_off.reserve(n + 1, 0, s))) return e;
  if ((e = exclusive_scan(ctx, ctx->div_flag.p, ctx->div_off.p, n, &ctx->status->divisions))) return e;
  if (!ctx->params.fixed_dt && n) {
    const size_t lo = n % 2 == 0 ? n / 2 - 1 : n / 2;
    if (n <= (size_t)kRankMost) {
      k_rank_median<<<grid_for((long long)n, kRankRows), kBlock, 0, s>>>(ctx->cells.view(), (int)n, (int)lo,
                                                                        ctx->status);
      ctx->launches++;
    } else {
      if ((e = ctx->keys.reserve(n, 0, s)) || (e = ctx->perm.reserve(n, 0, s))) return e;
      k_speed_keys<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), (long long)n, ctx->keys.p, ctx->perm.p);
      ctx->launches++;
      if ((e = radix_sort_pairs(ctx, ctx->keys.p, ctx->perm.p, n, 64))) return e;
      if ((e = cudaMemcpyAsync(ctx->status->median, ctx->keys.p + lo, 2 * sizeof(unsigned long long),
                               cudaMemcpyDeviceToDevice, s)))
        return e;
    }
  }
  return cudaMemcpyAsync(ctx->status_host, ctx->status, kStatusBytes, cudaMemcpyDeviceToHost, s);
}

// Domain::adaptDt (spatial/Domain.cpp:69-118): median of |v| + ldot (for an
// even count, the mean of the two middle values), dt* = cfl*tol/median,
// dt <- clamp(0.99 dt + 0.01 dt*, 0.9 dt, 1.1 dt).
static void adapt_dt(pcc_ctx* ctx) {
  const size_t n = ctx->n;
  if (!n) return;
  const unsigned long long* pk = ctx->status_host->median;
  double med;
  if (n % 2 == 0) {
    const double lower = key_to_double(pk[0]), upper = key_to_double(pk[1]);
    med = 0.5 * (lower + upper);
  } else {
    med = key_to_double(pk[0]);
  }
  const double gmed = med / 1;
  if (gmed == 0.0) return;
  const double cfl = ctx->params.cfl_factor * ctx->params.tolerance;
  const double cap_dt = cfl / gmed;
  const double dt = ctx->params.dt;
  volatile double t1 = dt * (1.0 - 0.01);
  volatile double t2 = 0.01 * cap_dt;
  double nd = t1 + t2;
  const double lo_dt = 0.9 * dt, hi_dt = 1.1 * dt;
  nd = nd < lo_dt ? lo_dt : (hi_dt < nd ? hi_dt : nd);
  ctx->params.dt = nd;
}

void step_end_collect(pcc_ctx* ctx) {
  const DevStatus& st = *ctx->status_host;
  if (!ctx->params.fixed_dt) adapt_dt(ctx);
  std::memcpy(&ctx->radius, &st.radius_bits, sizeof ctx->radius);
  ctx->box_known = true;
  if (ctx->x_crowded == 0) ctx->x_crowded = st.crowded;
  ctx->div_next = (size_t)st.divisions;
  ctx->div_known = true;
}

}  // namespace pcc

extern "C" unsigned int pcc_division_seed(unsigned long long seed, unsigned long long k) {
  return pcc::division_seed(seed, k);
}

extern "C" double pcc_division_length_host(unsigned long long seed, unsigned long long k, double len) {
  return pcc::division_length(seed, k, len);
}
