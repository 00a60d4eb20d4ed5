// On-chip BBPGD solver (sm_100a) for constraint sets whose operands fit the
// shared memory of a cluster or of the whole GPU.
//
// The method, the chunks, the per-cell sums and every reduction tree are those
// of the streaming kernels (pcc_planar.cu, pcc_solver.cu), so the results are
// theirs bit for bit; what differs is where the operands live and how the
// blocks meet.  A small constraint set is bound by latency: each iteration is
// two dependent gathers and two barriers, and the streaming kernel walks a
// cell's entries one dependent load at a time.  Here a block owns a contiguous
// range of cells (balanced by incidence entries) and some warps' worth of
// constraints, and keeps their rows, (gamma, g) pairs and Phi in shared memory
// for the whole solve.
//   * Entries are laid out by warp: the cells of a block in order of falling
//     entry count, 16 to a warp (two lanes each), step j of the warp's 32
//     lanes consecutive in memory, so the cell pass is a conflict-free stream
//     and its padding is small.
//   * Cluster form (kCluster): random reads of another block's shared memory
//     cost about 3 cycles each per SM (measured: 512 16-byte reads take 1,570
//     cycles; from L2 866), so nothing is read remotely: a constraint's owner
//     pushes its new pair into the slots of its two entries, and a cell's owner
//     pushes its velocity to the blocks that have a constraint on the cell.
//     Constraints are dealt to blocks in order of their first cell, so most
//     pushes stay in the block.  Blocks meet at the hardware cluster barrier
//     (about 500 cycles; a grid barrier through L2 takes 2,200), and every warp
//     pushes its dot products to every block.
//   * Grid form: pairs, velocities and chunk partials pass through L2; the
//     block first copies its entries' pairs to their slots, one thread per
//     entry, so an iteration pays one gather latency.
// A group of cells that does not fit the block's room (an unusually crowded
// range) is read from the constraints themselves at every use; the host sizes
// the room so that this does not happen in ordinary colonies.  What bounds such
// a group is the chain of its longest cell's entries, each a load of the entry
// and then of its constraint: with the next entry's load in flight, 800 knotted
// cells of up to 183 entries beside 28,000 sparse ones (59 groups without room,
// FP64) take 68.6 -> 54.0 us per iteration (the streaming kernel's form of one
// entry at a time took 57.6), 300 beside 2,000 (six, mixed, 16 blocks) 31.8 ->
// 25.5 (29.4).
//
// Measured, us per iteration before (streaming kernels) and now, B200 at 1965
// MHz: 447 cells / 3,000 constraints FP64 18.7 -> 4.3; 1,788 / 12,000 FP64 15.5
// -> 6.2; 9,172 / 70,000 mixed 17.9 -> 7.3; 1,005 / 6,500 in 3D 35.2 -> 6.4.
//
// k3D: six D components (colonies out of the plane, FP64 only); otherwise
// the planar form's three, in FP64 or with FP32 operands (Real = float).
#include <cfloat>
#include <cmath>

#include "pcc_bbpgd.cuh"
#include "pcc_kernels.hpp"

namespace pcc {

namespace {

template <bool k3D>
struct Form;
template <>
struct Form<false> {
  static constexpr int kD = 3;    // D components per side: n_x, n_y, z torque arm
  static constexpr int kRow = 4;  // entry row: D, stress weight
  static constexpr int kU = 4;    // velocity row: u_x, u_y, w_z, dldot
  static constexpr int kCon = 6;  // constraint row: n_x, n_y, t_iz, t_jz, s_i, s_j
};
template <>
struct Form<true> {
  static constexpr int kD = 6;
  static constexpr int kRow = 8;   // D, stress weight, unused
  static constexpr int kU = 8;     // 6 velocities, dldot, unused
  static constexpr int kCon = 11;  // n, t_i, t_j, s_i, s_j
};
constexpr int kMaxCluster = 16;
constexpr int kClusterThreads = 512;
constexpr int kGridThreads = 1024;
constexpr int kClusterShare = 512;  // constraints per block from which the cluster is doubled
constexpr long long kClusterChunks = 256;  // chunk partials that one warp sums in eight groups
constexpr int kGroup = 32 / kLanes;        // cells per warp of the cell pass
constexpr int kAhead = 3;                  // gathers that a thread of the grid form has in flight
constexpr int kDegrees = 256;              // bins of the sort by entry count

// The constraints of one warp of a chunk's 256-thread unit: 32 consecutive
// ones and, past the chunk's first 256, the 32 that are 256, 512, ... further.
struct Vwarp {
  int c0, hi;       // first constraint, end of the chunk
  int base, base2;  // first slot of the first 32, of the next
  int id;           // 8 * chunk + warp
  int pad[3];
};

struct ResArgs {
  long long m, n;
  ConsView cs;
  const int *inc_off, *inc_ent;
  const double *len, *ldot_prev;
  const double* uext;       // rotational U_ext, 3 per cell; null: zero
  double2* gg;              // grid form: (gamma, g) of the last iteration
  double* gprev;            // gamma_{k-1} of the last residual iteration
  void* u;                  // grid form: velocity rows
  double *U, *F, *sig, *ldot, *imp;
  double dt, lambda, tau, xi, tol;
  long long max_it;
  double* partials;         // grid form: value-major, one per chunk
  long long nchunks;
  int nvw;                  // warps' worths of constraints in all (8 per chunk)
  int lvw;                  // ... of one block at most
  int cstride;              // grid form: slots per chunk
  int extra;                // cluster form: rounds of 32 slots for constraints past a chunk's first 256
  int slots;                // constraint slots per block
  int cells_max;            // cells per block at most
  int cap;                  // entry slots per block
  int kappa;                // weight of a cell beside its entries in the split over blocks
  SolverScalars* sc;
  DevStatus* st;
};

// Shared-memory layout (bytes from the start), the same on host and device.
template <class Real, bool k3D, bool kCluster>
struct Layout {
  using F = Form<k3D>;
  size_t gg, phi, crow, ccode, pcode, vw, clo, vtab, vkey, u, umask, cell, off, perm, gbase, wres, pair, egold, erow, ecode, end;
  __host__ __device__ Layout(int slots, int lvw, int nvw, int cells_max, int cap, long long n, long long nchunks) {
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o += (bytes + 15) / 16 * 16;
      return at;
    };
    gg = take(16 * (size_t)slots);
    phi = take(8 * (size_t)slots);
    crow = take(sizeof(Real) * F::kCon * (size_t)slots);
    ccode = take(8 * (size_t)slots);
    pcode = take(kCluster ? 8 * (size_t)slots : 0);
    vw = take(sizeof(Vwarp) * (size_t)lvw);
    clo = take(4 * ((size_t)nchunks + 1));
    vtab = take(kCluster ? 4 * (size_t)nvw : 0);
    vkey = take(kCluster ? 4 * (size_t)nvw : 0);
    u = take(kCluster ? sizeof(Real) * F::kU * (size_t)n : 0);
    umask = take(kCluster ? 4 * (size_t)cells_max : 0);
    cell = take(sizeof(Real) * 4 * (size_t)cells_max);
    off = take(4 * ((size_t)cells_max + 1));
    perm = take(8 * (size_t)cells_max);
    gbase = take(4 * ((size_t)(cells_max + kGroup - 1) / kGroup + 1));
    wres = take(kCluster ? 256 * (size_t)nchunks : 32 * (size_t)(kGridThreads / 32));
    pair = take(16 * (size_t)cap);
    egold = take(8 * (size_t)cap);
    erow = take(sizeof(Real) * F::kRow * (size_t)cap);
    ecode = take(kCluster ? 0 : 4 * (size_t)cap);
    end = o;
  }
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned mapa(unsigned addr, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ double2 ld_cluster(unsigned addr) {
  double2 v;
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned addr, unsigned v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned addr, double2 v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
__device__ __forceinline__ void or_cluster(unsigned addr, unsigned v) {
  asm volatile("red.shared::cluster.or.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// The four values (sum, sum, sum, max) of a warp by the xor tree of
// warp_reduce4, splitting the values over the lanes as the tree narrows: lane
// l returns value l / 8 with the bits that warp_reduce4 leaves in lane 0 (6
// double exchanges instead of 20).
// With check == false the fourth value is taken as zero.
template <bool kCheck>
__device__ __forceinline__ double warp_reduce_split(const double v[4]) {
  const int lane = threadIdx.x & 31;
  const bool h16 = lane & 16, h8 = lane & 8, is_max = kCheck && h16 && h8;
  // lane 0 of warp_reduce4 keeps its own maximum unless it is smaller
  auto op = [](bool mx, double lo, double hi) { return kCheck && mx ? (lo < hi ? hi : lo) : add(lo, hi); };
  const double v3 = kCheck ? v[3] : 0.0;
  double a = h16 ? v[2] : v[0], b = h16 ? v3 : v[1];
  a = add(a, __shfl_xor_sync(kFull, h16 ? v[0] : v[2], 16));
  b = op(h16, __shfl_xor_sync(kFull, h16 ? v[1] : v3, 16), b);
  double r = h8 ? b : a;
  r = op(is_max, __shfl_xor_sync(kFull, h8 ? a : b, 8), r);
#pragma unroll
  for (int w = 4; w > 0; w >>= 1) {
    const double x = __shfl_xor_sync(kFull, r, w);
    if constexpr (kCheck) r = op(is_max, (lane & w) ? x : r, (lane & w) ? r : x);
    else r = add(r, x);
  }
  return r;
}

// Eight values by the xor tree of unit_reduce4's second half.
__device__ __forceinline__ double tree8(const double w[8], bool is_max) {
  auto op = [is_max](double lo, double hi) { return is_max ? (lo < hi ? hi : lo) : add(lo, hi); };
  return op(op(op(w[0], w[4]), op(w[2], w[6])), op(op(w[1], w[5]), op(w[3], w[7])));
}

// First cell whose weight (its offset in the incidence list + kappa per cell
// before it) reaches block b's share.
__host__ __device__ __forceinline__ int first_cell(const int* __restrict__ off, long long n, long long kappa, long long b,
                                          long long nb) {
  if (b >= nb) return (int)n;
  const long long total = (long long)off[n] + kappa * n, want = (b * total + nb - 1) / nb;
  long long lo = 0, hi = n;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if ((long long)off[mid] + kappa * mid < want) lo = mid + 1;
    else hi = mid;
  }
  return (int)lo;
}

template <class Real, bool k3D, bool kCluster>
__global__ void __launch_bounds__(kCluster ? kClusterThreads : kGridThreads, 1) k_bbpgd_res(const ResArgs a) {
  using F = Form<k3D>;
  constexpr int T = kCluster ? kClusterThreads : kGridThreads;
  constexpr int kWarps = T / 32;
  constexpr bool kF64 = sizeof(Real) == 8;
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_bnd[kMaxCluster + 1];
  __shared__ int s_hist[kDegrees + 1];
  __shared__ double s_alpha, s_v[4], s_grp[32];
  __shared__ int s_conv, s_nlv, s_end;  // s_end: end of the used entry slots
  const Layout<Real, k3D, kCluster> L(a.slots, a.lvw, a.nvw, a.cells_max, a.cap, a.n, a.nchunks);
  double2* const gg = reinterpret_cast<double2*>(sm + L.gg);
  double* const phi = reinterpret_cast<double*>(sm + L.phi);
  Real* const crow = reinterpret_cast<Real*>(sm + L.crow);  // component-major: crow[q * slots + slot]
  int2* const ccode = reinterpret_cast<int2*>(sm + L.ccode);
  uint2* const pcode = reinterpret_cast<uint2*>(sm + L.pcode);
  Vwarp* const vw = reinterpret_cast<Vwarp*>(sm + L.vw);
  int* const clo = reinterpret_cast<int*>(sm + L.clo);      // chunk_lo
  unsigned* const vtab = reinterpret_cast<unsigned*>(sm + L.vtab);  // of every warp's worth: block, place there
  int* const vkey = reinterpret_cast<int*>(sm + L.vkey);
  Real* const us = reinterpret_cast<Real*>(sm + L.u);
  unsigned* const umask = reinterpret_cast<unsigned*>(sm + L.umask);
  Real* const cellc = reinterpret_cast<Real*>(sm + L.cell);
  int* const soff = reinterpret_cast<int*>(sm + L.off);
  int* const perm = reinterpret_cast<int*>(sm + L.perm);  // cells in order, then each cell's place
  int* const gbase = reinterpret_cast<int*>(sm + L.gbase);
  double* const wres = reinterpret_cast<double*>(sm + L.wres);
  double2* const pair = reinterpret_cast<double2*>(sm + L.pair);
  double* const egold = reinterpret_cast<double*>(sm + L.egold);
  Real* const erow = reinterpret_cast<Real*>(sm + L.erow);  // 16-byte pieces, piece-major: piece * cap + slot
  int* const ecode = reinterpret_cast<int*>(sm + L.ecode);
  constexpr int kPiece = 16 / sizeof(Real);  // Reals per 16-byte piece of an entry row
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const unsigned nb = gridDim.x, rank = blockIdx.x;  // one cluster is the whole grid
  const int m = (int)a.m, nch = (int)a.nchunks;
  SolverScalars* const sc = a.sc;
  GridBarrier bar{sc, a.st, nb};
  auto meet = [&]() -> bool {
    if constexpr (kCluster) {
      if (nb == 1) {
        __syncthreads();
      } else {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      }
      return true;
    } else {
      return bar.sync();
    }
  };

  // ---------------------------------------------------------------- layout
  if constexpr (kCluster) {
    if (t <= (int)nb) s_bnd[t] = first_cell(a.inc_off, a.n, a.kappa, t, nb);
  } else {
    if (t < 2) s_bnd[t] = first_cell(a.inc_off, a.n, a.kappa, (long long)rank + t, nb);
  }
  for (int i = t; i <= kDegrees; i += T) s_hist[i] = 0;
  for (int i = t; i <= nch; i += T) clo[i] = (int)chunk_lo(i, m, nch);
  if constexpr (!kCluster) {
    for (int s = t; s < a.cap; s += T) ecode[s] = -1;  // padding
  }
  __syncthreads();
  const int cb = s_bnd[kCluster ? rank : 0];
  int ncell = s_bnd[kCluster ? rank + 1 : 1] - cb;
  if (ncell > a.cells_max) {  // cannot happen: the weights bound it
    if (t == 0) raise_error(a.st, kDevErrBounds, 23);
    ncell = a.cells_max;
  }
  const int eb = a.inc_off[cb];
  const int ngroups = (ncell + kGroup - 1) / kGroup;
  for (int i = t; i <= ncell; i += T) soff[i] = a.inc_off[cb + i] - eb;
  for (int i = t; i < ncell; i += T) {
    const double l = a.len[cb + i];
    cellc[4 * i] = (Real)dvd(1.0, mul(l, a.xi));  // mobilities (Physics.cpp:192-218)
    cellc[4 * i + 1] = (Real)dvd(12.0, mul(mul(mul(l, l), l), a.xi));
    cellc[4 * i + 2] = (Real)l;
    cellc[4 * i + 3] = (Real)a.ldot_prev[cb + i];
    if constexpr (kCluster) umask[i] = 0;
  }
  __syncthreads();
  // the block's cells by falling entry count (the order within a count is
  // arbitrary: which lanes sum a cell changes nothing in its sums)
  auto degree_bin = [&](int i) {
    const int d = soff[i + 1] - soff[i];
    return kDegrees - 1 - (d < kDegrees ? d : kDegrees - 1);
  };
  for (int i = t; i < ncell; i += T) atomicAdd(&s_hist[degree_bin(i)], 1);
  __syncthreads();
  if (warp == 0) {
    int run = 0;
    for (int b = 0; b < kDegrees; b += 32) {
      const int v = s_hist[b + lane];
      int x = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
      }
      s_hist[b + lane] = run + x - v;
      run += __shfl_sync(kFull, x, 31);
    }
  }
  __syncthreads();
  for (int i = t; i < ncell; i += T) {
    const int at = atomicAdd(&s_hist[degree_bin(i)], 1);
    perm[at] = i;
    perm[a.cells_max + i] = at;
  }
  __syncthreads();
  if (warp == 0) {
    int run = 0;
    for (int g0 = 0; g0 < ngroups; g0 += 32) {
      const int g = g0 + lane;
      int steps = 0;
      if (g < ngroups) {
        for (int j = g * kGroup; j < ncell && j < (g + 1) * kGroup; ++j) {
          const int d = (soff[perm[j] + 1] - soff[perm[j]] + kLanes - 1) / kLanes;
          steps = steps < d ? d : steps;
        }
      }
      int x = steps;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
      }
      if (g < ngroups) gbase[g] = (run + x) * 32 <= a.cap ? (run + x - steps) * 32 : -1;  // -1: no room
      run += __shfl_sync(kFull, x, 31);
    }
    if (lane == 0) s_end = run * 32 < a.cap ? run * 32 : a.cap;
  }

  // the block's constraints, in warps' worths
  const float per_m = (float)nch / (float)m;
  auto chunk_of = [&](int c) {
    int ch = (int)((float)c * per_m);
    if (ch >= nch) ch = nch - 1;
    while (clo[ch + 1] <= c) ++ch;
    while (clo[ch] > c) --ch;
    return ch;
  };
  if constexpr (kCluster) {
    // dealt to the blocks in order of their first constraint's smaller cell:
    // block r takes positions [start(r), start(r + 1)) of that order
    auto start = [&](int r) { return (int)((long long)r * a.nvw / nb); };
    for (int id = t; id < a.nvw; id += T) {
      const int c = clo[id >> 3] + 32 * (id & 7), hi = clo[(id >> 3) + 1];
      vkey[id] = c < hi ? a.cs.gi[c] : 0x7fffffff;
    }
    __syncthreads();
    for (int id = t; id < a.nvw; id += T) {
      const int key = vkey[id];
      int pos = 0;
      for (int o = 0; o < a.nvw; ++o) {
        const int k = vkey[o];
        pos += (k < key || (k == key && o < id)) ? 1 : 0;
      }
      vtab[id] = (unsigned)pos;
    }
    __syncthreads();
    for (int id = t; id < a.nvw; id += T) {
      const int pos = (int)vtab[id];
      int r = (int)((long long)pos * nb / a.nvw);
      while (start(r + 1) <= pos) ++r;
      while (start(r) > pos) --r;
      int extra = 0;  // chunks whose first warp is in the block before this one
      if ((id & 7) == 0) {
        for (int o = 0; o < nch; ++o) {
          const int p = (int)vtab[8 * o];
          extra += (p >= start(r) && p < pos) ? 1 : 0;
        }
        if (extra >= a.extra) {  // cannot happen: the constraints of a phase are in order of their smaller cell
          raise_error(a.st, kDevErrBounds, 24);
          extra = a.extra - 1;
        }
      }
      vkey[id] = (r << 24) | ((pos - start(r)) << 12) | extra;
    }
    __syncthreads();
    for (int id = t; id < a.nvw; id += T) {
      const unsigned w = (unsigned)vkey[id];
      vtab[id] = w;
      if ((w >> 24) != rank) continue;
      const int local = (w >> 12) & 0xfff;
      vw[local] = Vwarp{clo[id >> 3] + 32 * (id & 7), clo[(id >> 3) + 1], 32 * local,
                        32 * (a.lvw + (int)(w & 0xfff)), id, {0, 0, 0}};
    }
    if (t == 0) s_nlv = start(rank + 1) - start(rank);
  } else {
    // whole chunks rank, rank + nb, ...: eight consecutive warps each
    const int nlc = nch > (int)rank ? (nch - (int)rank + (int)nb - 1) / (int)nb : 0;
    for (int v = t; v < 8 * nlc; v += T) {
      const int ch = (int)rank + (int)nb * (v >> 3), base = a.cstride * (v >> 3) + 32 * (v & 7);
      vw[v] = Vwarp{clo[ch] + 32 * (v & 7), clo[ch + 1], base, base + kBlock, 8 * ch + (v & 7), {0, 0, 0}};
    }
    if (t == 0) s_nlv = 8 * nlc;
  }
  __syncthreads();
  const int nlv = s_nlv;
  // block and slot of constraint c (cluster form)
  auto owner = [&](int c, unsigned* slot) -> unsigned {
    const int ch = chunk_of(c), j = c - clo[ch];
    const unsigned w = vtab[8 * ch + (j < kBlock ? j >> 5 : 0)];
    *slot = j < kBlock ? 32 * ((w >> 12) & 0xfff) + (j & 31) : 32 * (a.lvw + (w & 0xfff)) + (j - kBlock);
    return w >> 24;
  };
  auto block_of_cell = [&](int p) -> unsigned {
    unsigned lo = 0, hi = nb - 1;
    while (lo < hi) {
      const unsigned mid = (lo + hi + 1) >> 1;
      if (s_bnd[mid] <= p) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  };
  // f(c, slot) for this thread's constraints of the warp's worth w
  auto each_constraint = [&](const Vwarp& w, auto&& f) {
    int s = w.base + lane, next = w.base2 + lane;
#pragma unroll 1
    for (int c = w.c0 + lane; c < w.hi; c += kBlock) {
      f(c, s);
      s = next;
      next += kBlock;
    }
  };
  for (int v = warp; v < nlv; v += kWarps) {
    each_constraint(vw[v], [&](int c, int s) {
      gg[s] = make_double2(a.cs.gamma[c], 0.0);
      phi[s] = a.cs.sd[c];
      ccode[s] = make_int2(a.cs.gi[c], a.cs.gj[c]);
      if constexpr (kCluster) pcode[s] = make_uint2(0u, 0u);
      auto put = [&](int q, double x) { crow[q * a.slots + s] = (Real)x; };
      if constexpr (k3D) {
        put(0, a.cs.nx[c]);
        put(1, a.cs.ny[c]);
        put(2, a.cs.nz[c]);
        put(3, a.cs.tix[c]);
        put(4, a.cs.tiy[c]);
        put(5, a.cs.tiz[c]);
        put(6, a.cs.tjx[c]);
        put(7, a.cs.tjy[c]);
        put(8, a.cs.tjz[c]);
        put(9, a.cs.si[c]);
        put(10, a.cs.sj[c]);
      } else {
        put(0, a.cs.nx[c]);
        put(1, a.cs.ny[c]);
        put(2, a.cs.tiz[c]);
        put(3, a.cs.tjz[c]);
        put(4, a.cs.si[c]);
        put(5, a.cs.sj[c]);
      }
    });
  }
  if constexpr (kCluster) meet();  // every block's tables are clear before others write to them
  // row of incidence entry `ent` from its constraint
  auto load_row = [&](int ent, Real r[F::kRow]) {
    const int c = ent >> 1;
    const bool sj = ent & 1;
    r[0] = (Real)(sj ? -a.cs.nx[c] : a.cs.nx[c]);
    r[1] = (Real)(sj ? -a.cs.ny[c] : a.cs.ny[c]);
    if constexpr (k3D) {
      r[2] = sj ? -a.cs.nz[c] : a.cs.nz[c];
      r[3] = sj ? a.cs.tjx[c] : a.cs.tix[c];
      r[4] = sj ? a.cs.tjy[c] : a.cs.tiy[c];
      r[5] = sj ? a.cs.tjz[c] : a.cs.tiz[c];
      r[6] = sj ? a.cs.sj[c] : a.cs.si[c];
      r[7] = 0;
    } else {
      r[2] = (Real)(sj ? a.cs.tjz[c] : a.cs.tiz[c]);
      r[3] = (Real)(sj ? a.cs.sj[c] : a.cs.si[c]);
    }
  };
  // entry slots
  const int ne = soff[ncell];
#pragma unroll 1
  for (int k = t; k < ne; k += T) {
    const int ent = a.inc_ent[eb + k], c = ent >> 1, i = (ent & 1 ? a.cs.gj[c] : a.cs.gi[c]) - cb;
    const int at = perm[a.cells_max + i], g0 = gbase[at / kGroup], x = k - soff[i];
    if (g0 < 0) continue;
    const int s = g0 + 32 * (x / kLanes) + kLanes * (at % kGroup) + x % kLanes;
    Real r[F::kRow];
    load_row(ent, r);
#pragma unroll
    for (int q = 0; q < F::kRow; ++q) erow[(q / kPiece * a.cap + s) * kPiece + q % kPiece] = r[q];
    egold[s] = a.cs.gamma[c];
    if constexpr (kCluster) {
      unsigned slot;
      const unsigned to = owner(c, &slot);
      st_cluster(mapa(smem_addr(pcode + slot) + 4 * (ent & 1), to), mapa(smem_addr(pair + s), rank));
    } else {
      ecode[s] = c;
    }
  }
  if constexpr (kCluster) {
    // blocks that need a cell's velocity
    for (int v = warp; v < nlv; v += kWarps) {
      each_constraint(vw[v], [&](int, int s) {
        const int2 ij = ccode[s];
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          const int p = side ? ij.y : ij.x;
          const unsigned r = block_of_cell(p);
          or_cluster(mapa(smem_addr(umask + (p - s_bnd[r])), r), 1u << rank);
        }
      });
    }
  }

  // ---------------------------------------------------------------- passes
  const double itau = dvd(1.0, a.tau);
  // mode 0 at gamma_0, mode 1 at gamma_k = max(gamma - alpha g, 0); final also
  // writes the per-cell outputs
  auto cell_pass = [&](int mode, double alpha, bool final) {
    // gamma_k of every entry and its change since gamma_0, one thread per
    // entry (in the grid form after the gather of its constraint's pair)
    auto stage = [&](int s, double2 p) {
      const double gc = project(p.x, p.y, alpha);
      pair[s] = make_double2(gc, sub(gc, egold[s]));
    };
    const int end = s_end;
    if (mode == 0) {
#pragma unroll 1
      for (int s = t; s < end; s += T) pair[s] = make_double2(egold[s], sub(egold[s], egold[s]));
    } else if constexpr (kCluster) {
#pragma unroll 2
      for (int s = t; s < end; s += T) stage(s, pair[s]);
    } else {
#pragma unroll 1
      for (int s0 = t; s0 < end; s0 += kAhead * T) {
        int c[kAhead];
        double2 x[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) c[q] = s0 + q * T < end ? ecode[s0 + q * T] : -1;
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
          if (c[q] >= 0) x[q] = ldcg(a.gg + c[q]);
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
          if (c[q] >= 0) stage(s0 + q * T, x[q]);
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int w = t; w < 32 * ngroups; w += T) {
      const int i = w >> 5 << 4 | lane / kLanes, l = lane % kLanes;
      const bool live = i < ncell;
      const int pl = live ? perm[i] : 0, g0 = gbase[w >> 5];
      const int d = live ? soff[pl + 1] - soff[pl] : 0;
      Real f[F::kD];
      double sg = 0.0;
#pragma unroll
      for (int q = 0; q < F::kD; ++q) f[q] = 0;
      auto take = [&](const Real r[F::kRow], double gc, double diff) {
        if constexpr (kF64) {
#pragma unroll
          for (int q = 0; q < F::kD; ++q) f[q] = add(f[q], mul(r[q], diff));
          sg = add(sg, mul((double)r[F::kD], gc));
        } else {
          const float df = (float)diff;
#pragma unroll
          for (int q = 0; q < F::kD; ++q) f[q] = fmaf(r[q], df, f[q]);
          sg = fma((double)r[F::kD], gc, sg);
        }
      };
      if (g0 >= 0) {
        const int steps = (d - l + kLanes - 1) / kLanes;
        int s = g0 + lane;
#pragma unroll(k3D ? 2 : 4)
        for (int j = 0; j < steps; ++j, s += 32) {
          Real r[F::kRow];
#pragma unroll
          for (int q = 0; q < F::kRow; q += kPiece)
            *reinterpret_cast<int4*>(r + q) = *reinterpret_cast<const int4*>(erow + (q / kPiece * a.cap + s) * kPiece);
          const double2 p = pair[s];
          take(r, p.x, p.y);
        }
      } else {  // no room in shared memory
        const int* list = a.inc_ent + eb + soff[pl];
        int next = l < d ? list[l] : 0;
#pragma unroll 1
        for (int k = l; k < d; k += kLanes) {
          const int ent = next;
          if (k + kLanes < d) next = list[k + kLanes];  // in flight beside this entry's loads
          Real r[F::kRow];
          load_row(ent, r);
          const double go = a.cs.gamma[ent >> 1];
          double gc = go;
          if (mode != 0) {
            double2 p;
            if constexpr (kCluster) {
              unsigned slot;
              const unsigned o = owner(ent >> 1, &slot);
              p = ld_cluster(mapa(smem_addr(gg + slot), o));
            } else {
              p = ldcg(a.gg + (ent >> 1));
            }
            gc = project(p.x, p.y, alpha);
          }
          take(r, gc, sub(gc, go));
        }
      }
#pragma unroll
      for (int q = 0; q < F::kD; ++q) {
        if constexpr (kF64) f[q] = add(f[q], __shfl_xor_sync(kFull, f[q], 1));
        else f[q] = __fadd_rn(f[q], __shfl_xor_sync(kFull, f[q], 1));
      }
      sg = add(sg, __shfl_xor_sync(kFull, sg, 1));
      if (!live || l != 0) continue;
      const Real ml = cellc[4 * pl], mr = cellc[4 * pl + 1];
      const int p = cb + pl;
      double v[F::kD];
#pragma unroll
      for (int q = 0; q < F::kD; ++q) {
        const bool rot = q >= (k3D ? 3 : 2);
        const double ue = (rot && a.uext) ? a.uext[3 * (size_t)p + (k3D ? q - 3 : 2)] : 0.0;
        if constexpr (kF64) {
          v[q] = add(add(0.0, mul(rot ? mr : ml, f[q])), ue);  // U = U_ext + M F (HardModelGradient.cpp:21)
        } else {
          const float x = (rot ? mr : ml) * f[q];
          v[q] = rot ? (double)x + ue : (double)x;
        }
      }
      const double im = exp(vscale(-a.lambda, sg));
      const double ld = vscale(itau, mul((double)cellc[4 * pl + 2], im));
      const double dl = sub(ld, (double)cellc[4 * pl + 3]);
      if constexpr (kCluster) {
        const unsigned at = smem_addr(us + (size_t)F::kU * p);
        for (unsigned need = umask[pl]; need; need &= need - 1) {
          const unsigned to = mapa(at, __ffs(need) - 1);
          if constexpr (k3D) {
            st_cluster(to, make_double2(v[0], v[1]));
            st_cluster(to + 16, make_double2(v[2], v[3]));
            st_cluster(to + 32, make_double2(v[4], v[5]));
            st_cluster(to + 48, dl);
          } else if constexpr (kF64) {
            st_cluster(to, make_double2(v[0], v[1]));
            st_cluster(to + 16, make_double2(v[2], dl));
          } else {
            st_cluster(to, make_float4((float)v[0], (float)v[1], (float)v[2], (float)dl));
          }
        }
      } else {
        Real* ur = reinterpret_cast<Real*>(a.u) + (size_t)F::kU * p;
        if constexpr (k3D) {
          *reinterpret_cast<double2*>(ur) = make_double2(v[0], v[1]);
          *reinterpret_cast<double2*>(ur + 2) = make_double2(v[2], v[3]);
          *reinterpret_cast<double2*>(ur + 4) = make_double2(v[4], v[5]);
          ur[6] = dl;
        } else if constexpr (kF64) {
          *reinterpret_cast<double2*>(ur) = make_double2(v[0], v[1]);
          *reinterpret_cast<double2*>(ur + 2) = make_double2(v[2], dl);
        } else {
          *reinterpret_cast<float4*>(ur) = make_float4((float)v[0], (float)v[1], (float)v[2], (float)dl);
        }
      }
      if (final) {
        double* Up = a.U + 6 * (size_t)p;
        double* Fp = a.F + 6 * (size_t)p;
        if constexpr (k3D) {
#pragma unroll
          for (int q = 0; q < 6; ++q) {
            Up[q] = v[q];
            Fp[q] = f[q];
          }
        } else {
          Up[0] = v[0];
          Up[1] = v[1];
          Up[2] = Up[3] = Up[4] = 0.0;
          Up[5] = v[2];
          Fp[0] = f[0];
          Fp[1] = f[1];
          Fp[2] = Fp[3] = Fp[4] = 0.0;
          Fp[5] = f[2];
        }
        a.sig[p] = sg;
        a.ldot[p] = ld;
        a.imp[p] = im;
      }
    }
  };

  auto load_u = [&](int p, Real u[F::kU]) {
    constexpr int kStep = kCluster || !kF64 ? kPiece : 4;
#pragma unroll
    for (int q = 0; q < F::kU; q += kStep) {
      if constexpr (kCluster) {
        *reinterpret_cast<int4*>(u + q) = *reinterpret_cast<const int4*>(us + (size_t)F::kU * p + q);
      } else if constexpr (kF64) {
        const double4 w = ld256w(reinterpret_cast<const double4*>(a.u) + ((size_t)F::kU * p + q) / 4);
        u[q] = w.x;
        u[q + 1] = w.y;
        u[q + 2] = w.z;
        u[q + 3] = w.w;
      } else {
        *reinterpret_cast<int4*>(u + q) =
            *(reinterpret_cast<const int4*>(reinterpret_cast<const Real*>(a.u) + (size_t)F::kU * p + q));
      }
    }
  };
  // phi_next of the constraint at slot s (MatMult row in ascending columns:
  // gi < gj for every emitted constraint; VecMAXPY(phi_next, {dt, -dt}, ...))
  auto grad = [&](int s) -> double {
    const int2 ij = ccode[s];
    Real ui[F::kU], uj[F::kU], r[F::kCon];
    load_u(ij.x, ui);
    load_u(ij.y, uj);
#pragma unroll
    for (int q = 0; q < F::kCon; ++q) r[q] = crow[q * a.slots + s];
    if constexpr (k3D) {
      double pd = 0.0;
#pragma unroll
      for (int q = 0; q < 6; ++q) pd = add(pd, mul(r[q], ui[q]));
#pragma unroll
      for (int q = 0; q < 6; ++q) pd = add(pd, mul(q < 3 ? -r[q] : r[3 + q], uj[q]));
      double gr = 0.0;
      gr = add(gr, mul(r[9], ui[6]));
      gr = add(gr, mul(r[10], uj[6]));
      return add(phi[s], add(mul(a.dt, pd), mul(-a.dt, gr)));
    } else if constexpr (kF64) {
      double pd = 0.0;
      pd = add(pd, mul(r[0], ui[0]));
      pd = add(pd, mul(r[1], ui[1]));
      pd = add(pd, mul(r[2], ui[2]));
      pd = add(pd, mul(-r[0], uj[0]));
      pd = add(pd, mul(-r[1], uj[1]));
      pd = add(pd, mul(r[3], uj[2]));
      double gr = 0.0;
      gr = add(gr, mul(r[4], ui[3]));
      gr = add(gr, mul(r[5], uj[3]));
      return add(phi[s], add(mul(a.dt, pd), mul(-a.dt, gr)));
    } else {
      float pd = r[0] * ui[0];
      pd = fmaf(r[1], ui[1], pd);
      pd = fmaf(r[2], ui[2], pd);
      pd = fmaf(-r[0], uj[0], pd);
      pd = fmaf(-r[1], uj[1], pd);
      pd = fmaf(r[3], uj[2], pd);
      const float gr = fmaf(r[5], uj[3], r[4] * ui[3]);
      return phi[s] + a.dt * ((double)pd - (double)gr);
    }
  };

  // new (gamma, g), dot products and residual per chunk; mode 0 evaluates g at
  // gamma_0 (residual only)
  auto constraint_pass = [&](int mode, double alpha, bool check) {
#pragma unroll 1
    for (int x = warp; x < nlv; x += kWarps) {
      const Vwarp w = vw[x];
      double v[4] = {0, 0, 0, 0};
      each_constraint(w, [&](int c, int s) {
        const double g = grad(s);
        const double2 o = gg[s];
        const double gam = mode == 0 ? o.x : project(o.x, o.y, alpha);
        const double2 now = make_double2(gam, g);
        gg[s] = now;
        if constexpr (kCluster) {
          const uint2 to = pcode[s];
          if (to.x) st_cluster(to.x, now);
          if (to.y) st_cluster(to.y, now);
        } else {
          a.gg[c] = now;
        }
        if (mode != 0) {
          const double dgm = sub(gam, o.x), dg = sub(g, o.y);
          v[0] = add(v[0], mul(dgm, dgm));
          v[1] = add(v[1], mul(dgm, dg));
          v[2] = add(v[2], mul(dg, dg));
          if (check) a.gprev[c] = o.x;  // what the solve returns if it ends here (Hard.cpp:170, BBPGD.cpp:124)
        }
        if (mode == 0 || check) {
          const double rr = proj_grad_abs(g, gam);
          v[3] = v[3] < rr ? rr : v[3];
        }
      });
      const double r = check ? warp_reduce_split<true>(v) : warp_reduce_split<false>(v);
      const int ch = w.id >> 3, w8 = w.id & 7, q = lane >> 3;
      if constexpr (kCluster) {
        const unsigned at = smem_addr(wres + ((q * 8 + w8) * nch + ch));
        for (unsigned d = lane & 7; d < nb; d += 8) st_cluster(mapa(at, d), r);
      } else {
        // the eight warps of a chunk are one 256-thread group of the block
        const int unit = warp >> 3;
        if ((lane & 7) == 0) wres[(unit * 4 + q) * 8 + w8] = r;
        asm volatile("bar.sync %0, %1;" ::"r"(unit + 1), "r"(kBlock) : "memory");
        if (w8 == 0 && lane < 4) {
          double y[8];
#pragma unroll
          for (int z = 0; z < 8; ++z) y[z] = wres[(unit * 4 + lane) * 8 + z];
          a.partials[(size_t)lane * nch + ch] = tree8(y, lane == 3);
        }
        if (x + kWarps < nlv) asm volatile("bar.sync %0, %1;" ::"r"(unit + 1), "r"(kBlock) : "memory");
      }
    }
  };

  // Sums of the chunk partials in the order of reduce_partials, by every block
  // alike.  In the cluster form every thread returns them, in the grid form
  // warp 0.
  auto tree32 = [&](double r, bool mx) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double y = __shfl_xor_sync(kFull, r, o);
      r = mx ? (r < y ? y : r) : add(r, y);
    }
    return r;
  };
  auto reduce = [&](double v[4], bool check) {
    const int values = check ? 4 : 3;
    if constexpr (kCluster) {
      // warp q: value q; lane = chunk within a group of 32, groups as the warps of the 256-thread unit
      if (warp < values) {
        const bool mx = warp == 3;
        const double* w = wres + warp * 8 * nch;
        double r = 0.0;
#pragma unroll 1
        for (int x = 0; 32 * x < nch; ++x) {
          const int ch = 32 * x + lane;
          r = 0.0;
          if (ch < nch) {
            double y[8];
#pragma unroll
            for (int z = 0; z < 8; ++z) y[z] = w[z * nch + ch];
            r = tree8(y, mx);
            r = mx ? (0.0 < r ? r : 0.0) : add(0.0, r);
          }
          r = tree32(r, mx);
          if (nch > 32 && lane == 0) s_grp[warp * 8 + x] = r;
        }
        if (nch > 32) {
          __syncwarp();
          double y[8];
#pragma unroll
          for (int z = 0; z < 8; ++z) y[z] = 32 * z < nch ? s_grp[warp * 8 + z] : 0.0;
          r = tree8(y, mx);
        } else if (!mx) {
          r = add(r, 0.0);  // the other seven warps' sums
        }
        if (lane == 0) s_v[warp] = r;
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = s_v[q];
    } else {
      // warp (q, x): value q of the chunks of warp x of the 256-thread unit
      const int q = warp >> 3;
      if (q < values) {
        const double* part = a.partials + (size_t)q * nch;
        double r = 0.0;
        constexpr int kAtOnce = 3;
#pragma unroll 1
        for (int ch = 32 * (warp & 7) + lane; ch < nch; ch += kAtOnce * kBlock) {
          double y[kAtOnce];
#pragma unroll
          for (int z = 0; z < kAtOnce; ++z) y[z] = ch + z * kBlock < nch ? ldcg(part + ch + z * kBlock) : 0.0;
#pragma unroll
          for (int z = 0; z < kAtOnce; ++z) {
            if (ch + z * kBlock < nch) r = q == 3 ? (r < y[z] ? y[z] : r) : add(r, y[z]);
          }
        }
        r = tree32(r, q == 3);
        if (lane == 0) s_grp[warp] = r;
      }
      __syncthreads();
      if (warp != 0) return;
      double r = s_grp[lane];
      const bool mx = lane >= 24;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(kFull, r, o);
        r = mx ? (r < y ? y : r) : add(r, y);
      }
#pragma unroll
      for (int z = 0; z < 4; ++z) v[z] = __shfl_sync(kFull, r, 8 * z);
    }
  };

  // ---------------------------------------------------------------- solve
  const bool recorder = rank == 0 && t == 0;
  if (recorder) sc->overlap_bits = 0;  // the barriers of an iteration order it before the sums at the end
  double v[4] = {0, 0, 0, 0};
  if constexpr (kCluster) meet();
  else __syncthreads();
  long long it = 0;
  double alpha = 0.0;
  bool conv = false;
#pragma unroll 1
  while (it < a.max_it || it == 0) {
    // it = 0: the gradient at gamma_0 and the initial residual (BBPGD.cpp:40-44)
    const int mode = it == 0 ? 0 : 1;
    const bool check = it % 10 == 0;
    cell_pass(mode, alpha, mode != 0 && check);
    if (!meet()) return;
    constraint_pass(mode, alpha, check);
    if (!meet()) return;
    reduce(v, check);
    auto decide = [&]() {
      conv = mode != 0 && check && v[3] <= a.tol;
      if (!conv) alpha = mode == 0 ? dvd(1.0, v[3]) : bb_step(v, it);
      if (recorder && check) {
        sc->residual = v[3];
        if (mode == 0) sc->res0 = v[3];
      }
    };
    if constexpr (kCluster) {
      decide();
    } else {
      if (warp == 0) {
        decide();
        if (lane == 0) {
          s_alpha = alpha;
          s_conv = conv ? 1 : 0;
        }
      }
      __syncthreads();
      alpha = s_alpha;
      conv = s_conv;
    }
    if (conv) break;
    ++it;
  }
  if (recorder) {
    sc->iterations = it;
    sc->converged = conv ? 1 : 0;
    sc->alpha = alpha;
  }
  // the returned iterate (Hard.cpp:170 with BBPGD.cpp:124): gamma_{k-1} and
  // phi of gamma_k; a planar solve that ran out of iterations leaves the
  // gamma_{k-1} of its last residual iteration, as the streaming kernel does
  if (conv || (!k3D && it > 10)) {
    double most = 0.0;
    for (int x = warp; x < nlv; x += kWarps) {
      each_constraint(vw[x], [&](int c, int s) {
        a.cs.gamma[c] = a.gprev[c];
        if (!conv) return;
        const double g = gg[s].y;
        a.cs.sd[c] = g;
        most = overlap_of(most, g);
      });
    }
    __syncwarp();
    fold_overlap(sc, most);
  }
}

// Shape of a launch: blocks, room per block, shared memory.
struct Shape {
  int nb = 0, nvw = 0, lvw = 0, cstride = 0, extra = 0, slots = 0, cells_max = 0, cap = 0, kappa = 0;
  size_t smem = 0;
};

constexpr size_t kSmemMost = 227 * 1024 - 2048;  // dynamic part; the kernel's own variables need the rest

template <class Real, bool k3D, bool kCluster>
bool shape_for(long long m, long long n, long long nchunks, int phases, int nb, Shape* o) {
  const long long e = 2 * m;
  o->nb = nb;
  o->kappa = (int)(e / (n ? n : 1)) + 4;
  const long long total = e + o->kappa * n, share = total / nb + 1;
  o->cells_max = (int)(share / o->kappa + 2);
  if (o->cells_max > n) o->cells_max = (int)n;
  o->nvw = (int)(8 * nchunks);
  if (kCluster) {
    o->lvw = (o->nvw + nb - 1) / nb;
    // at most one chunk's first warp in eight of a phase's run of warps
    o->extra = o->lvw / 8 + phases + 2;
    if (o->extra > nchunks) o->extra = (int)nchunks;
    o->slots = 32 * (o->lvw + o->extra);
  } else {
    o->cstride = (int)(((m + nchunks - 1) / nchunks + 32 + 31) / 32 * 32);  // chunk starts are multiples of 32
    if (o->cstride < kBlock) o->cstride = kBlock;
    const int nlc = (int)((nchunks + nb - 1) / nb);
    o->lvw = 8 * nlc;
    o->slots = nlc * o->cstride;
  }
  auto bytes = [&](int cap) {
    return Layout<Real, k3D, kCluster>(o->slots, o->lvw, o->nvw, o->cells_max, cap, n, nchunks).end;
  };
  if (bytes(0) > kSmemMost) return false;
  const long long per = 16 + 8 + sizeof(Real) * Form<k3D>::kRow + (kCluster ? 0 : 4);
  const long long room = ((long long)(kSmemMost - bytes(0)) / per) & ~31LL;
  // a block's entries, a tenth for the padding of the cells' order (their
  // counts fall slowly within a warp's group) and a few groups' worth
  const long long entries = e / nb, want = (entries + entries / 10 + 32 * 24) & ~31LL;
  if (room < want) return false;
  const long long most = (2 * want) & ~31LL;
  o->cap = (int)(room < most ? room : most);
  o->smem = bytes(o->cap);
  return o->smem <= kSmemMost;
}

// The form and shape for m constraints, found in `phases` detections, on n
// cells: the smallest cluster that leaves a block at most kClusterShare
// constraints (or the largest, if its shared memory holds them), else the grid
// form; false: neither holds them.
template <class Real, bool k3D>
bool pick_shape(long long m, long long n, int phases, int num_sms, int cluster_max, Shape* sh, bool* cluster) {
  const long long nchunks = chunk_count(m);
  *cluster = false;
  if (nchunks <= kClusterChunks) {
    for (int nb = 1; nb <= cluster_max && !*cluster; nb *= 2) {
      if (nb < cluster_max && m > (long long)nb * kClusterShare) continue;
      *cluster = shape_for<Real, k3D, true>(m, n, nchunks, phases, nb, sh);
    }
  }
  return *cluster || shape_for<Real, k3D, false>(m, n, nchunks, 1, (int)(nchunks < num_sms ? nchunks : num_sms), sh);
}

// Opts both forms into their shared memory and asks for the largest cluster
// that the device can hold (0: none), once per context and kernel: the opt-in
// belongs to the CUDA context, which a program may reset between colonies.
template <class Real, bool k3D>
cudaError_t largest_cluster(int* known) {
  if (*known >= 0) return cudaSuccess;
  const void* kc = (const void*)k_bbpgd_res<Real, k3D, true>;
  const void* kg = (const void*)k_bbpgd_res<Real, k3D, false>;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(kc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost)) ||
      (e = cudaFuncSetAttribute(kg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost)) ||
      (e = cudaFuncSetAttribute(kc, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)))
    return e;
  int most = kMaxCluster;
  for (; most > 0; most /= 2) {
    cudaLaunchConfig_t q = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)most, 1, 1};
    q.gridDim = dim3((unsigned)most);
    q.blockDim = dim3(kClusterThreads);
    q.dynamicSmemBytes = kSmemMost;
    q.attrs = at;
    q.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, kc, &q) == cudaSuccess && fit > 0) break;
    cudaGetLastError();
  }
  *known = most;
  return cudaSuccess;
}

template <class Real, bool k3D>
cudaError_t try_resident(pcc_ctx* ctx, double dt, bool* taken, int* kind) {
  cudaStream_t s = ctx->stream;
  const long long n = (long long)ctx->n, m = (long long)ctx->ncons;
  const long long nchunks = chunk_count(m);
  const void* kc = (const void*)k_bbpgd_res<Real, k3D, true>;
  const void* kg = (const void*)k_bbpgd_res<Real, k3D, false>;
  cudaError_t e;
  *taken = false;
  int& cluster_max = ctx->cluster_most[k3D ? 2 : sizeof(Real) == 8];
  if ((e = largest_cluster<Real, k3D>(&cluster_max))) return e;
  Shape sh;
  bool cluster = false;
  if (!pick_shape<Real, k3D>(m, n, ctx->trace_phase + 1, ctx->num_sms, cluster_max, &sh, &cluster)) return cudaSuccess;
  if ((e = ctx->p_gg.reserve(m + 1, 0, s)) || (e = ctx->p_phin.reserve(m + 1, 0, s)) ||
      (e = ctx->partials.reserve(4 * (nchunks + 1), 0, s)) || (e = ctx->p_u.reserve(2 * (n + 1), 0, s)))
    return e;
  ResArgs a;
  a.m = m;
  a.n = n;
  a.cs = ctx->cons.view();
  a.inc_off = ctx->inc_off.p;
  a.inc_ent = ctx->inc_ent.p;
  a.len = ctx->cells.len.p;
  a.ldot_prev = ctx->cells.ldot.p;
  a.uext = ctx->uext_active ? ctx->uext.p : nullptr;
  a.gg = ctx->p_gg.p;
  a.gprev = ctx->p_phin.p;
  a.u = ctx->p_u.p;
  a.U = ctx->U.p;
  a.F = ctx->F.p;
  a.sig = ctx->sig.p;
  a.ldot = ctx->ldot_new.p;
  a.imp = ctx->imp_new.p;
  a.dt = dt;
  a.lambda = ctx->params.lambda;
  a.tau = ctx->params.tau;
  a.xi = ctx->params.xi;
  a.tol = ctx->params.tolerance;
  a.max_it = ctx->params.max_bbpgd_iterations;
  a.partials = ctx->partials.p;
  a.nchunks = nchunks;
  a.nvw = sh.nvw;
  a.lvw = sh.lvw;
  a.cstride = sh.cstride;
  a.extra = sh.extra;
  a.slots = sh.slots;
  a.cells_max = sh.cells_max;
  a.cap = sh.cap;
  a.kappa = sh.kappa;
  a.sc = &ctx->status->solver;
  a.st = ctx->status;
  if ((e = order_incidence(ctx))) return e;
  // the grid form's barrier counts from zero; a cluster clears what it adds to
  if (!cluster) cudaMemsetAsync(a.sc, 0, sizeof(SolverScalars), s);
  void* args[] = {&a};
  if (ctx->profiling) cudaEventRecord(ctx->ev[0], s);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  if (cluster) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)sh.nb, 1, 1};
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cfg.gridDim = dim3((unsigned)sh.nb);
  cfg.blockDim = dim3(cluster ? kClusterThreads : kGridThreads);
  cfg.dynamicSmemBytes = sh.smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  *taken = true;
  *kind = sh.nb > 1 ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, cluster ? kc : kg, args);
}

}  // namespace

cudaError_t resident_bbpgd(pcc_ctx* ctx, double dt, bool full, bool mixed, bool* taken, int* kind) {
  if (full) return try_resident<double, true>(ctx, dt, taken, kind);
  return mixed ? try_resident<float, false>(ctx, dt, taken, kind) : try_resident<double, false>(ctx, dt, taken, kind);
}

}  // namespace pcc
