// Broadphase + narrowphase contact detection (sm_100a).
//
// Replaces SpatialGrid::findPotentialCollisions (spatial/SpatialGrid.cpp:58-121)
// and CollisionDetector::tryCreateConstraint (spatial/CollisionDetector.cpp:201-311)
// of the reference.  Cells are binned on their centres exactly like the
// reference grid (origin -1, edge linked_cell_size, floor), so the candidate
// pairs -- every unordered pair in the same or an adjacent bin of the
// 27-stencil -- are the same set.  Binning is a counting sort: atomic counts,
// an exclusive scan, an atomic scatter and each cell's rank by id within its
// bin, which makes the bin contents (and everything downstream)
// deterministic.  Each cell's geometry is packed once per phase in bin order
// so the neighbour scans read contiguous 32-byte groups.  The full pass scans
// the stencil once, counts the constraints and records each cell's partners
// within a wider reach in a candidate list; the emit pass and the later ReLCP
// phases of the same step walk those lists (with the reference's bin-adjacency
// test on the current bins and a displacement bound that proves no other pair
// can qualify).  Counts are scanned into offsets, so constraints come out
// grouped by the smaller id in a fixed order, without atomics on the output.
//
// The pair passes are chains of dependent loads and of double-precision
// geometry, so they are bound by latency unless the GPU is full: kPairLanes
// lanes share a cell's candidates.  Measured (stencil scan / list count / list
// emit, us, ncu, cold caches): one thread per cell 56 / 23 / 27 at 447 cells
// and 84 / 35 / 45 at 44,700; eight lanes 13 / 8 / 8 and 57 / 37 / 35; four
// lanes 62 / 31 / 35 at 44,700.  At 302,180 cells, where memory bounds them,
// 295 / 128 / 195 with one thread, 319 / 150 / 185 with four lanes and 337 /
// 245 / 207 with eight.
//
// At the end of a pass the host needs the number of contacts and a few flags:
// they are collected in the device status, cleared by one memset and read by
// one copy per pass.
#include <cmath>
#include <cstring>

#include "pcc_kernels.hpp"

namespace pcc {

namespace {

constexpr int kPack = 16;  // doubles per packed cell record
// record layout: [x y z len | sx sy sz diam | ex ey ez gid | tx ty tz ghost]
constexpr int kList = 32;  // candidate partners kept per cell
constexpr double kListReach = 0.25;  // list reach beyond contact: the first ReLCP phase's tolerance
constexpr int kFewCells = 20000;  // below: 8 lanes per cell in the pair passes, from there on 4
enum : unsigned { kListOverflow = 1u, kListStale = 2u, kOutOfBox = 4u };

// Warp-wide max of a non-negative double folded into *dst (all lanes call).
__device__ __forceinline__ void warp_max_into(unsigned long long* dst, double v) {
  for (int o = 16; o > 0; o >>= 1) {
    const double u = __shfl_xor_sync(0xffffffffu, v, o);
    v = v < u ? u : v;
  }
  if ((threadIdx.x & 31) == 0 && v > 0.0) atomicMax(dst, (unsigned long long)__double_as_longlong(v));
}

// Bounding-box keys: a maximum that starts from 0 serves for both ends.
__host__ __device__ inline unsigned box_key_hi(int b) { return (unsigned)b ^ 0x80000000u; }
__host__ __device__ inline unsigned box_key_lo(int b) { return ~box_key_hi(b); }

struct Grid {
  int mx, my, mz, nx, ny, nz;
};

struct Binned {
  int bx, by, bz, ghost;
};

// Bin of a cell (origin -1, edge h, floor: the reference grid) and its
// self-ghost; folds the planarity flag, the longest cell and (when xref is
// given) the largest squared displacement since xref into the status, one
// atomic per warp (all lanes call; live: the lane has a cell).
__device__ __forceinline__ Binned bin_cell(const CellsView& c, size_t i, bool live, double h, int ghost_mode,
                                           const double* __restrict__ xref, DevStatus* st) {
  Binned o = {0, 0, 0, 0};
  int nonplanar = 0;
  double len = 0.0, drift2 = 0.0;
  if (live) {
    const double x = c.x[i], y = c.y[i], z = c.z[i];
    o.bx = (int)floor(dvd(sub(x, -1.0), h));
    o.by = (int)floor(dvd(sub(y, -1.0), h));
    o.bz = (int)floor(dvd(sub(z, -1.0), h));
    len = c.len[i];
    if (xref) {
      const double dx = x - xref[3 * i], dy = y - xref[3 * i + 1], dz = z - xref[3 * i + 2];
      drift2 = dx * dx + dy * dy + dz * dz;
    }
    // planar colony (z = 0, rotation about z only): the solver may use its 2D form
    nonplanar = (z != 0.0 || c.q1[i] != 0.0 || c.q2[i] != 0.0) ? 1 : 0;
    if (ghost_mode == PCC_GHOSTS_SINGLE_RANK) {
      // Domain::exchangeGhostParticles at world size 1 (spatial/Domain.cpp:339-403)
      // with calculateDistanceToAngularBoundary (263-290) for the sector [0, 360).
      // The distance is |y| up to rounding (radius * sin of the angle to the x
      // axis), so a cell well beyond 2.5 in y needs no angle.
      const double radius = __dsqrt_rn(add(mul(x, x), mul(y, y)));
      if (radius >= 8.0 && !(fabs(y) > 3.0 && radius < 1e9)) {
        double ang = dvd(mul(atan2(y, x), 180.0), M_PI);
        if (ang < 0) ang += 360.0;
        double dmin = ang - 0.0, dmax = 360.0 - ang;
        while (dmin > 180.0) dmin -= 360.0;
        while (dmin < -180.0) dmin += 360.0;
        while (dmax > 180.0) dmax -= 360.0;
        while (dmax < -180.0) dmax += 360.0;
        double dist = 0.0;
        if (!(dmin >= 0 && dmax >= 0)) {
          double m = fabs(dmin) < fabs(dmax) ? fabs(dmin) : fabs(dmax);
          dist = mul(radius, sin(dvd(mul(m, M_PI), 180.0)));
        }
        o.ghost = dist < 2.5 ? 1 : 0;
      }
    }
  }
  const unsigned np = __reduce_or_sync(0xffffffffu, (unsigned)nonplanar);
  if ((threadIdx.x & 31) == 0 && np) atomicOr(&st->nonplanar, 1u);
  warp_max_into(&st->lmax_bits, len);
  if (xref) warp_max_into(&st->drift_bits, drift2);
  return o;
}

__device__ __forceinline__ int bin_key(const Grid& g, int bx, int by, int bz) {
  return ((bz - g.mz) * g.ny + (by - g.my)) * g.nx + (bx - g.mx);
}

// Bin counts with warp-aggregated atomics: the lanes of a warp that fall in
// the same bin (cells are in x-sorted order, so neighbours often do) find
// each other with __match_any_sync and one of them adds the group's size.
__device__ __forceinline__ void count_bin(int k, bool live, int* __restrict__ cnt) {
  const unsigned peers = __match_any_sync(0xffffffffu, live ? k : -1);
  if (live && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&cnt[k], __popc(peers));
}

// Bins every cell.  With kCount the grid is known (a box around the colony's
// radius) and the bins are counted too; a cell outside the box raises
// kOutOfBox, on which the passes that follow return at once (300,000 cells off
// the plane would else be ordered as one bin: 15.5 ms for a step that takes
// 0.6, 1,000,000 cells 150 ms for 1.6) and the caller starts again without the
// box.  Otherwise the bounding box of the bins is folded into the status for
// the caller to read.
template <bool kCount>
__global__ void k_bin(CellsView c, size_t n, double h, int ghost_mode, Grid g, int* __restrict__ binxyz,
                      int* __restrict__ ghost, int* __restrict__ key, int* __restrict__ cnt, DevStatus* st) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < n;
  const Binned b = bin_cell(c, i, live, h, ghost_mode, nullptr, st);
  if (live) {
    binxyz[3 * i] = b.bx;
    binxyz[3 * i + 1] = b.by;
    binxyz[3 * i + 2] = b.bz;
    ghost[i] = b.ghost;
  }
  if constexpr (kCount) {
    const bool in = b.bx >= g.mx && b.bx < g.mx + g.nx && b.by >= g.my && b.by < g.my + g.ny && b.bz >= g.mz &&
                    b.bz < g.mz + g.nz;
    if (live && !in) atomicOr(&st->list_flags, kOutOfBox);
    const int k = in ? bin_key(g, b.bx, b.by, b.bz) : 0;
    if (live) key[i] = k;
    count_bin(k, live && in, cnt);
  } else {
    const int v[3] = {b.bx, b.by, b.bz};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const unsigned lo = __reduce_max_sync(0xffffffffu, live ? box_key_lo(v[d]) : 0u);
      const unsigned hi = __reduce_max_sync(0xffffffffu, live ? box_key_hi(v[d]) : 0u);
      if ((threadIdx.x & 31) == 0) {
        if (lo) atomicMax(&st->box_lo[d], lo);
        if (hi) atomicMax(&st->box_hi[d], hi);
      }
    }
  }
}

__global__ void k_bin_count(const int* __restrict__ binxyz, size_t n, Grid g, int* __restrict__ key,
                            int* __restrict__ cnt) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < n;
  int k = 0;
  if (live) key[i] = k = bin_key(g, binxyz[3 * i], binxyz[3 * i + 1], binxyz[3 * i + 2]);
  count_bin(k, live, cnt);
}

// Scatter into the bins from their ends (the counts run down to zero): one
// atomic per group of same-bin lanes takes the group's slots, each lane the
// slot of its rank in the group (k_pack orders each bin).
__global__ void k_bin_scatter(const int* __restrict__ key, size_t n, const int* __restrict__ off,
                              int* __restrict__ cnt, int* __restrict__ cells, const DevStatus* st) {
  if (__ldcg(&st->list_flags) & kOutOfBox) return;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < n;
  const int k = live ? key[i] : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, k);
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  int base = 0;
  if (live && lane == leader) base = atomicSub(&cnt[k], __popc(peers)) - __popc(peers);
  base = __shfl_sync(peers, base, leader);
  if (live) cells[off[k] + base + __popc(peers & ((1u << lane) - 1u))] = (int)i;
}

// Packs cell i's record at slot s.
__device__ __forceinline__ void pack_cell(const CellsView& c, int i, int ghost, size_t s, double* __restrict__ pk) {
  double t[3];
  cell_axis(c.q0[i], c.q1[i], c.q2[i], c.q3[i], t);
  const double len = c.len[i], diam = c.diam[i];
  // CollisionDetector::getParticleEndpoints (spatial/CollisionDetector.cpp:61-75)
  const double half = sub(dvd(len, 2.0), dvd(diam, 2.0));
  const double p[3] = {c.x[i], c.y[i], c.z[i]};
  double r[kPack];
  r[0] = p[0];
  r[1] = p[1];
  r[2] = p[2];
  r[3] = len;
  for (int d = 0; d < 3; ++d) {
    const double hv = mul(t[d], half);
    r[4 + d] = sub(p[d], hv);
    r[8 + d] = add(p[d], hv);
    r[12 + d] = t[d];
  }
  r[7] = diam;
  r[11] = (double)i;
  r[15] = (double)ghost;
  double2* o = reinterpret_cast<double2*>(pk + s * kPack);
#pragma unroll
  for (int q = 0; q < kPack / 2; ++q) o[q] = make_double2(r[2 * q], r[2 * q + 1]);
}

// Orders each bin by id and packs the records in that order: thread per
// scattered cell, whose rank among its bin's cells is its slot there.
__global__ void k_pack(CellsView c, const int* __restrict__ raw, const int* __restrict__ key,
                       const int* __restrict__ off, const int* __restrict__ ghost, size_t n, int* __restrict__ slot_cell,
                       int* __restrict__ slot_of, double* __restrict__ pk, const DevStatus* st) {
  if (__ldcg(&st->list_flags) & kOutOfBox) return;
  const size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int i = raw[r], k = key[i], e = off[k + 1];
  int s = off[k];
  for (int q = s; q < e; ++q) s += raw[q] < i ? 1 : 0;
  slot_cell[s] = i;
  slot_of[i] = s;
  pack_cell(c, i, ghost[i], (size_t)s, pk);
}

// Later ReLCP phase on the slots of the pass that built the lists: current
// bins, ghosts and records in one pass.
__global__ void k_repack(CellsView c, const int* __restrict__ slot_cell, size_t n, double h, int ghost_mode,
                         const double* __restrict__ xref, int* __restrict__ binxyz, double* __restrict__ pk,
                         DevStatus* st) {
  const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = s < n;
  const size_t i = live ? (size_t)slot_cell[s] : 0;
  const Binned b = bin_cell(c, i, live, h, ghost_mode, xref, st);
  if (!live) return;
  binxyz[3 * i] = b.bx;
  binxyz[3 * i + 1] = b.by;
  binxyz[3 * i + 2] = b.bz;
  pack_cell(c, (int)i, b.ghost, s, pk);
}

// Closest points of two segments: Eberly's branch scheme for segment-segment
// distance (the variant the reference uses, util/SpherocylinderCell.h:64-261),
// restated with non-contracting IEEE operations.
__device__ void segment_closest(const double P0[3], const double P1[3], const double Q0[3], const double Q1[3],
                                double c0[3], double c1[3], double* dist) {
  double Pd[3], Qd[3], PQ[3];
  for (int k = 0; k < 3; ++k) {
    Pd[k] = sub(P1[k], P0[k]);
    Qd[k] = sub(Q1[k], Q0[k]);
    PQ[k] = sub(P0[k], Q0[k]);
  }
  const double a = dot3(Pd, Pd), b = dot3(Pd, Qd), c = dot3(Qd, Qd);
  const double d = dot3(Pd, PQ), e = dot3(Qd, PQ);
  const double det = sub(mul(a, c), mul(b, b));
  double s = 0.0, t = 0.0;
  if (det > 0.0) {
    const double bte = mul(b, e), ctd = mul(c, d);
    if (bte <= ctd) {
      s = 0.0;
      if (e <= 0.0) {
        t = 0.0;
        double nd = -d;
        if (nd >= a) s = 1.0;
        else if (nd > 0.0) s = dvd(nd, a);
      } else if (e < c) {
        t = dvd(e, c);
      } else {
        t = 1.0;
        double bmd = sub(b, d);
        if (bmd >= a) s = 1.0;
        else if (bmd > 0.0) s = dvd(bmd, a);
      }
    } else {
      s = sub(bte, ctd);
      if (s >= det) {
        s = 1.0;
        double bpe = add(b, e);
        if (bpe <= 0.0) {
          t = 0.0;
          double nd = -d;
          if (nd <= 0.0) s = 0.0;
          else if (nd < a) s = dvd(nd, a);
        } else if (bpe < c) {
          t = dvd(bpe, c);
        } else {
          t = 1.0;
          double bmd = sub(b, d);
          if (bmd <= 0.0) s = 0.0;
          else if (bmd < a) s = dvd(bmd, a);
        }
      } else {
        const double ate = mul(a, e), btd = mul(b, d);
        if (ate <= btd) {
          t = 0.0;
          double nd = -d;
          if (nd <= 0.0) s = 0.0;
          else if (nd >= a) s = 1.0;
          else s = dvd(nd, a);
        } else {
          t = sub(ate, btd);
          if (t >= det) {
            t = 1.0;
            double bmd = sub(b, d);
            if (bmd <= 0.0) s = 0.0;
            else if (bmd >= a) s = 1.0;
            else s = dvd(bmd, a);
          } else {
            s = dvd(s, det);
            t = dvd(t, det);
          }
        }
      }
    }
  } else {
    if (e <= 0.0) {
      t = 0.0;
      double nd = -d;
      if (nd <= 0.0) s = 0.0;
      else if (nd >= a) s = 1.0;
      else s = dvd(nd, a);
    } else if (e >= c) {
      t = 1.0;
      double bmd = sub(b, d);
      if (bmd <= 0.0) s = 0.0;
      else if (bmd >= a) s = 1.0;
      else s = dvd(bmd, a);
    } else {
      s = 0.0;
      t = dvd(e, c);
    }
  }
  double diff[3];
  for (int k = 0; k < 3; ++k) {
    c0[k] = add(P0[k], mul(Pd[k], s));
    c1[k] = add(Q0[k], mul(Qd[k], t));
    diff[k] = sub(c0[k], c1[k]);
  }
  *dist = __dsqrt_rn(dot3(diff, diff));
}


struct PairGeom {
  double sd, n[3], cp[3], ri[3], rj[3], si, sj;
};

// The centre-distance prefilter of tryCreateConstraint
// (spatial/CollisionDetector.cpp:210-213): the pair is dropped when
// sqrt(|x_a - x_b|^2) > (l_a + l_b)/2 + tol.  sqrt is correctly rounded and
// monotone, so away from the boundary the squared distance decides; within a
// relative 1e-9 of it the exact test runs.  (l_a + l_b) * 0.5 equals
// (l_a + l_b) / 2 exactly.
__device__ __forceinline__ bool rough_pass(const double4& a0, const double4& b0, double tol) {
  const double dv[3] = {sub(a0.x, b0.x), sub(a0.y, b0.y), sub(a0.z, b0.z)};
  const double d2 = dot3(dv, dv);
  const double reach = add(mul(add(a0.w, b0.w), 0.5), tol);
  const double r2 = reach * reach;
  if (d2 > r2 * (1.0 + 1e-9)) return false;
  if (d2 < r2 * (1.0 - 1e-9)) return true;
  return !(__dsqrt_rn(d2) > reach);
}

// The rest of tryCreateConstraint for a pair (I, J) = (A, B) that passed the
// prefilter.  With full == false only the separation is computed.
__device__ __forceinline__ bool pair_geom(const double* __restrict__ A, const double* __restrict__ B, double tol,
                                          bool full, PairGeom* o) {
  const double4 a1 = ld256(reinterpret_cast<const double4*>(A + 4));
  const double4 a2 = ld256(reinterpret_cast<const double4*>(A + 8));
  const double4 b1 = ld256(reinterpret_cast<const double4*>(B + 4));
  const double4 b2 = ld256(reinterpret_cast<const double4*>(B + 8));
  const double P0[3] = {a1.x, a1.y, a1.z}, P1[3] = {a2.x, a2.y, a2.z};
  const double Q0[3] = {b1.x, b1.y, b1.z}, Q1[3] = {b2.x, b2.y, b2.z};
  double c0[3], c1[3], dist;
  segment_closest(P0, P1, Q0, Q1, c0, c1, &dist);
  const double sd = sub(dist, dvd(add(a1.w, b1.w), 2.0));
  if (sd > tol) return false;
  o->sd = sd;
  if (!full) return true;
  double diff[3];
  for (int k = 0; k < 3; ++k) {
    o->cp[k] = mul(add(c0[k], c1[k]), 0.5);
    diff[k] = sub(c0[k], c1[k]);
  }
  // ArrayMath::normalize (util/ArrayMath.h:219-231)
  const double mag = __dsqrt_rn(dot3(diff, diff));
  if (mag > 2.220446049250313e-16) {
    const double inv = dvd(1.0, mag);
    for (int k = 0; k < 3; ++k) o->n[k] = mul(diff[k], inv);
  } else {
    o->n[0] = 1.0;
    o->n[1] = 0.0;
    o->n[2] = 0.0;
  }
  const double4 a0 = ld256(reinterpret_cast<const double4*>(A));
  const double4 b0 = ld256(reinterpret_cast<const double4*>(B));
  const double4 a3 = ld256(reinterpret_cast<const double4*>(A + 12));
  const double4 b3 = ld256(reinterpret_cast<const double4*>(B + 12));
  const double ta[3] = {a3.x, a3.y, a3.z}, tb[3] = {b3.x, b3.y, b3.z};
  const double nn[3] = {-o->n[0], -o->n[1], -o->n[2]};
  o->si = mul(0.5, fabs(dot3(o->n, ta)));
  o->sj = mul(0.5, fabs(dot3(nn, tb)));
  const double pa[3] = {a0.x, a0.y, a0.z}, pb[3] = {b0.x, b0.y, b0.z};
  for (int k = 0; k < 3; ++k) {
    o->ri[k] = sub(o->cp[k], pa[k]);
    o->rj[k] = sub(o->cp[k], pb[k]);
  }
  return true;
}

// Writes `copies` identical constraint rows for the pair (a, b) from row w on
// (a second copy stands for the partner's self-ghost).  Returns false when the
// rows would pass `cap`.
__device__ __forceinline__ bool emit_rows(ConsView cs, size_t& w, size_t cap, int a, int b, int phase, int copies,
                                          const PairGeom& pg, DevStatus* st) {
  double ti[3], tj[3];
  const double nj[3] = {-pg.n[0], -pg.n[1], -pg.n[2]};
  cross3(pg.ri, pg.n, ti);
  cross3(pg.rj, nj, tj);
  for (int k = 0; k < copies; ++k, ++w) {
    if (w >= cap) {
      raise_error(st, kDevErrCapacity, 10);
      return false;
    }
    cs.gi[w] = a;
    cs.gj[w] = b;
    cs.phase[w] = phase;
    cs.sd[w] = pg.sd;
    cs.gamma[w] = pg.sd >= 0.0 ? 0.0 : mul(-pg.sd, 5e2);
    cs.nx[w] = pg.n[0];
    cs.ny[w] = pg.n[1];
    cs.nz[w] = pg.n[2];
    cs.tix[w] = ti[0];
    cs.tiy[w] = ti[1];
    cs.tiz[w] = ti[2];
    cs.tjx[w] = tj[0];
    cs.tjy[w] = tj[1];
    cs.tjz[w] = tj[2];
    cs.rix[w] = pg.ri[0];
    cs.riy[w] = pg.ri[1];
    cs.riz[w] = pg.ri[2];
    cs.rjx[w] = pg.rj[0];
    cs.rjy[w] = pg.rj[1];
    cs.rjz[w] = pg.rj[2];
    cs.cpx[w] = pg.cp[0];
    cs.cpy[w] = pg.cp[1];
    cs.cpz[w] = pg.cp[2];
    cs.si[w] = pg.si;
    cs.sj[w] = pg.sj;
  }
  return true;
}

// Slots [lo, hi) of the up to three bins of stencil row (dy, dz) of a cell at
// bin (bx, by, bz) (grid coordinates): they hold consecutive slots.
__device__ __forceinline__ bool stencil_row(const Grid& g, const int* __restrict__ bin_off, int bx, int y, int z,
                                            int* lo, int* hi) {
  if (z < 0 || z >= g.nz || y < 0 || y >= g.ny) return false;
  const int x0 = bx > 0 ? bx - 1 : 0, x1 = bx + 1 < g.nx ? bx + 1 : g.nx - 1;
  const int row = (z * g.ny + y) * g.nx;
  *lo = bin_off[row + x0];
  *hi = bin_off[row + x1 + 1];
  return true;
}

// Full neighbourhood pass of a phase: kPairLanes lanes per cell in bin order
// scan the 27-stencil for partners with a larger id (the candidate pairs of
// SpatialGrid::findPotentialCollisions, spatial/SpatialGrid.cpp:58-121) and
// append every partner within the wider reach tol_list to the cell's candidate
// list (slots of the packed records) in stencil order, so the emit pass and
// the later ReLCP phases of the step need no stencil scan.  The lanes then
// share the listed pairs, so that the geometry runs with all lanes in use:
// for each pair that passes tryCreateConstraint they count the constraints
// the smaller id emits (a second copy when the partner has a self-ghost),
// track the largest overlap, and add to Particle::num_constraints of both
// cells (CollisionDetector.cpp:243-244, ghost copies included; the count of a
// cell that has a self-ghost lands on the copy and is lost, as in the
// reference).  The cell's position at list time is kept in xref.
//
// What bounds it is latency (candidate loads, then the geometry's FP64 chain):
// the rows of a layer are one sequence with kScanAhead candidates of a lane in
// flight, a cell with more than kList partners is scanned again for the rest
// instead of testing them within the scan (the geometry's registers are then
// live once, and three blocks fit an SM, with 80 registers and 92 bytes of them
// spilled).  Detection of 89,090 soft cells per
// step: 297 us row by row, 277 with one candidate ahead and two blocks, 263
// with two and three (three ahead 271).
constexpr int kScanAhead = 2;
template <int kPairLanes>
__global__ void __launch_bounds__(kBlock, 3) k_scan_count(const double* __restrict__ pk, const int* __restrict__ bin_off,
                                                       Grid g, const int* __restrict__ binxyz, size_t n, double tol,
                                                       double tol_list, int* __restrict__ cnt,
                                                       int* __restrict__ ncontacts, int* __restrict__ plist,
                                                       int* __restrict__ plist_n, double* __restrict__ xref,
                                                       DevStatus* st) {
  static_assert(kPairLanes >= 3, "three lanes write the position");
  __shared__ int s_list[kBlock / kPairLanes][kList];
  const size_t s = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / kPairLanes;
  const int lane = threadIdx.x & 31, l = lane % kPairLanes, shift = lane - l;
  constexpr unsigned kOnes = kPairLanes == 32 ? ~0u : (1u << kPairLanes) - 1u;
  const unsigned group = kOnes << shift;
  int* list = s_list[threadIdx.x / kPairLanes];
  if (__ldcg(&st->list_flags) & kOutOfBox) return;  // the binning failed: count nothing
  double maxov = 0.0;
  if (s < n) {
    const double* A = pk + s * kPack;
    const int a = (int)A[11];
    const double4 a0 = ld256(reinterpret_cast<const double4*>(A));
    if (l < 3) xref[3 * (size_t)a + l] = A[l];
    const int bx = binxyz[3 * (size_t)a] - g.mx, by = binxyz[3 * (size_t)a + 1] - g.my,
              bz = binxyz[3 * (size_t)a + 2] - g.mz;
    const int ga = A[15] != 0.0;
    int count = 0, nl, skip = 0;
    do {  // again only for a cell with more than kList partners
      nl = 0;
      for (int dz = -1; dz <= 1; ++dz) {
        // the layer's three rows as one sequence of candidates, in row order
        int first[3], end[3], total = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          int lo = 0, hi = 0;
          if (!stencil_row(g, bin_off, bx, by + q - 1, bz + dz, &lo, &hi)) lo = hi = 0;
          first[q] = lo - total;  // slot of candidate k of this row: first + k
          total += hi - lo;
          end[q] = total;
        }
        for (int k0 = 0; k0 < total; k0 += kScanAhead * kPairLanes) {
          int s2[kScanAhead], b[kScanAhead];
          double4 b0[kScanAhead];
#pragma unroll
          for (int q = 0; q < kScanAhead; ++q) {
            const int k = k0 + q * kPairLanes + l;
            s2[q] = k < end[0] ? first[0] + k : k < end[1] ? first[1] + k : first[2] + k;
            b[q] = -1;
            if (k >= total) continue;
            const double* B = pk + (size_t)s2[q] * kPack;
            b[q] = (int)B[11];
            b0[q] = ld256(reinterpret_cast<const double4*>(B));
          }
#pragma unroll
          for (int q = 0; q < kScanAhead; ++q) {
            const bool in = b[q] > a && rough_pass(a0, b0[q], tol_list);
            const unsigned hits = __ballot_sync(group, in) >> shift & kOnes;
            const int at = nl + __popc(hits & ((1u << l) - 1u)) - skip;
            nl += __popc(hits);
            if (!in || at < 0 || at >= kList) continue;
            list[at] = s2[q];
            if (skip == 0) plist[(size_t)a * kList + at] = s2[q];
          }
        }
      }
      __syncwarp(group);
      const int listed = nl - skip < kList ? nl - skip : kList;
      for (int k = l; k < listed; k += kPairLanes) {
        const double* B = pk + (size_t)list[k] * kPack;
        if (tol < tol_list && !rough_pass(a0, ld256(reinterpret_cast<const double4*>(B)), tol)) continue;
        PairGeom pg;
        if (!pair_geom(A, B, tol, false, &pg)) continue;
        const int gb = B[15] != 0.0;
        count += 1 + gb;
        const double ov = pg.sd < 0 ? -pg.sd : 0.0;
        maxov = maxov < ov ? ov : maxov;
        if (!gb) atomicAdd(&ncontacts[(int)B[11]], 1 + ga);
      }
      __syncwarp(group);  // the list is filled again
      skip += kList;
    } while (skip < nl);
#pragma unroll
    for (int o = kPairLanes / 2; o > 0; o >>= 1) count += __shfl_xor_sync(group, count, o);
    if (l == 0) {
      cnt[a] = count;
      if (!ga && count) atomicAdd(&ncontacts[a], count);
      plist_n[a] = nl;
      if (nl > kList) atomicOr(&st->list_flags, kListOverflow);
    }
  }
  warp_max_into(&st->max_bits, maxov);
}

// Count (kEmit = false) or emit pass over the candidate lists, kPairLanes
// lanes per cell in id order; the emit order per cell is the list order,
// which is the stencil order of the full pass.  The emit pass also adds to
// the cells' incidence counts.
//
// In a later ReLCP phase of the step (adjacent = true) the lists are reused
// without rebinning the colony.  A listed pair is a candidate only if the two
// cells' current bins are neighbours, which is the reference's test.  A pair
// that is not listed cannot be a candidate that passes: with D the largest
// displacement of any cell since the lists were built and L the longest cell,
// a pair within (l_a + l_b)/2 + tol now was within (l_a + l_b)/2 + tol + 2D
// then, which is inside the list reach when tol + 2D < tol_list, and closer
// than one bin edge h (so in neighbouring bins) when L + tol + 2D < h.  If
// either bound fails the pass does nothing and flags the lists stale; the
// caller then runs the full pass.
template <bool kEmit, int kPairLanes>
__global__ void __launch_bounds__(kBlock) k_list_pass(
    const double* __restrict__ pk, const int* __restrict__ slot_of, size_t n, double tol, int phase, bool adjacent,
    double tol_list, double h, const int* __restrict__ binxyz, const int* __restrict__ plist,
    const int* __restrict__ plist_n, int* __restrict__ cnt, int* __restrict__ ncontacts, const int* __restrict__ off,
    ConsView cs, size_t base, size_t cap, int* __restrict__ inc_cnt, DevStatus* st) {
  const size_t a = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / kPairLanes;
  if (!kEmit && adjacent) {
    const double d2 = __longlong_as_double((long long)__ldcg(&st->drift_bits));
    const double lmax = __longlong_as_double((long long)__ldcg(&st->lmax_bits));
    const double reach = tol + 2.0 * sqrt(d2);
    if (!(reach < tol_list - 1e-6 && lmax + reach < h - 1e-6)) {
      if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&st->list_flags, kListStale);
      return;
    }
  }
  const int lane = threadIdx.x & 31, l = lane % kPairLanes, shift = lane - l;
  constexpr unsigned kOnes = kPairLanes == 32 ? ~0u : (1u << kPairLanes) - 1u;
  const unsigned group = kOnes << shift;
  double maxov = 0.0;
  if (a < n) {
    const double* A = pk + (size_t)slot_of[a] * kPack;
    const double4 a0 = ld256(reinterpret_cast<const double4*>(A));
    const int ga = A[15] != 0.0;
    const int nl = min(plist_n[a], kList);  // lists in use never overflowed
    int bxa = 0, bya = 0, bza = 0;
    if (adjacent) {
      bxa = binxyz[3 * a];
      bya = binxyz[3 * a + 1];
      bza = binxyz[3 * a + 2];
    }
    int count = 0;
    size_t w = kEmit ? base + (size_t)off[a] : 0;
    for (int k0 = 0; k0 < nl; k0 += kPairLanes) {
      const int k = k0 + l;
      int b = 0, gb = 0;
      bool pass = false;
      PairGeom pg;
      if (k < nl) {
        const double* B = pk + (size_t)plist[a * kList + k] * kPack;
        b = (int)B[11];
        pass = true;
        if (adjacent) {
          const int ex = binxyz[3 * (size_t)b] - bxa, ey = binxyz[3 * (size_t)b + 1] - bya,
                    ez = binxyz[3 * (size_t)b + 2] - bza;
          pass = ex >= -1 && ex <= 1 && ey >= -1 && ey <= 1 && ez >= -1 && ez <= 1;
        }
        pass = pass && rough_pass(a0, ld256(reinterpret_cast<const double4*>(B)), tol);
        pass = pass && pair_geom(A, B, tol, kEmit, &pg);
        gb = pass && B[15] != 0.0;
      }
      if (kEmit) {
        const unsigned low = (1u << l) - 1u;
        const unsigned p = __ballot_sync(group, pass) >> shift, g2 = __ballot_sync(group, gb) >> shift;
        size_t at = w + __popc(p & low) + __popc(g2 & low);
        if (pass && emit_rows(cs, at, cap, (int)a, b, phase, 1 + gb, pg, st)) {
          count += 1 + gb;
          atomicAdd(&inc_cnt[b], 1 + gb);
        }
        w += __popc(p & kOnes) + __popc(g2 & kOnes);
      } else if (pass) {
        count += 1 + gb;
        const double ov = pg.sd < 0 ? -pg.sd : 0.0;
        maxov = maxov < ov ? ov : maxov;
        if (!gb) atomicAdd(&ncontacts[b], 1 + ga);
      }
    }
#pragma unroll
    for (int o = kPairLanes / 2; o > 0; o >>= 1) count += __shfl_xor_sync(group, count, o);
    if (l == 0) {
      if (kEmit) {
        if (count) atomicAdd(&inc_cnt[a], count);
      } else {
        cnt[a] = count;
        if (!ga && count) atomicAdd(&ncontacts[a], count);
      }
    }
  }
  if (!kEmit) warp_max_into(&st->max_bits, maxov);
}

// Emit pass over the 27-stencil, for a phase whose candidate lists overflowed.
__global__ void k_stencil_emit(const double* __restrict__ pk, const int* __restrict__ bin_off, Grid g,
                               const int* __restrict__ binxyz, size_t n, double tol, int phase,
                               const int* __restrict__ off, ConsView cs, size_t base, size_t cap,
                               int* __restrict__ inc_cnt, DevStatus* st) {
  const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const double* A = pk + s * kPack;
  const int a = (int)A[11];
  const double4 a0 = ld256(reinterpret_cast<const double4*>(A));
  const int bx = binxyz[3 * (size_t)a] - g.mx, by = binxyz[3 * (size_t)a + 1] - g.my,
            bz = binxyz[3 * (size_t)a + 2] - g.mz;
  size_t w = base + (size_t)off[a];
  for (int dz = -1; dz <= 1; ++dz) {
    for (int dy = -1; dy <= 1; ++dy) {
      int lo, hi;
      if (!stencil_row(g, bin_off, bx, by + dy, bz + dz, &lo, &hi)) continue;
      for (int s2 = lo; s2 < hi; ++s2) {
        const double* B = pk + (size_t)s2 * kPack;
        const int b = (int)B[11];
        if (b <= a) continue;
        const double4 b0 = ld256(reinterpret_cast<const double4*>(B));
        if (!rough_pass(a0, b0, tol)) continue;
        PairGeom pg;
        if (!pair_geom(A, B, tol, true, &pg)) continue;
        const int copies = 1 + (B[15] != 0.0 ? 1 : 0);
        if (!emit_rows(cs, w, cap, a, b, phase, copies, pg, st)) return;
        atomicAdd(&inc_cnt[a], copies);
        atomicAdd(&inc_cnt[b], copies);
      }
    }
  }
}

__global__ void k_inc_fill(const int* __restrict__ gi, const int* __restrict__ gj, size_t m, int* __restrict__ cursor,
                           int* __restrict__ raw) {
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m) return;
  raw[atomicAdd(&cursor[gi[c]], 1)] = (int)(2 * c);
  raw[atomicAdd(&cursor[gj[c]], 1)] = (int)(2 * c + 1);
}

// Orders each cell's entries, one thread per entry (its rank among the cell's
// entries): 4.4 us at 447 cells where an insertion sort per cell took 31, its
// longest list one chain of dependent loads.
__global__ void k_inc_order(const int* __restrict__ gi, const int* __restrict__ gj, const int* __restrict__ off,
                            const int* __restrict__ raw, size_t ne, int* __restrict__ ent) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ne) return;
  int at;
  const int e = entry_place(gi, gj, off, raw, k, &at);
  ent[at] = e;
}

__global__ void k_interleave3(const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
                              size_t n, double* __restrict__ out) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;  // one value: the writes are consecutive
  if (t >= 3 * n) return;
  const size_t k = t / 3;
  const int d = (int)(t - 3 * k);
  out[t] = d == 0 ? x[k] : d == 1 ? y[k] : z[k];
}

}  // namespace

cudaError_t interleave3(pcc_ctx* ctx, const double* x, const double* y, const double* z, size_t n, double* out) {
  k_interleave3<<<grid_for((long long)(3 * n)), kBlock, 0, ctx->stream>>>(x, y, z, n, out);
  ctx->launches++;
  return cudaGetLastError();
}

// Grid of the bins of every centre within `r` of the origin, if it is not too
// large for the colony (a long chain's box would be mostly empty); at z the
// one bin of the plane z = 0.
static bool box_of_radius(double r, double h, size_t n, Grid* g) {
  if (!(r >= 0) || !(r < 1e8 * h)) return false;
  const int lo = (int)std::floor((-r + 1.0) / h) - 1, hi = (int)std::floor((r + 1.0) / h) + 1;
  const long long w = (long long)hi - lo + 1;
  if (w * w > 8 * (long long)n + 16384) return false;
  g->mx = g->my = lo;
  g->nx = g->ny = (int)w;
  g->mz = (int)std::floor(1.0 / h);
  g->nz = 1;
  return true;
}

cudaError_t detect_contacts(pcc_ctx* ctx, double tol, int phase, bool reuse, size_t* added,
                            double* max_overlap_new) {
  cudaStream_t s = ctx->stream;
  const size_t n = ctx->n;
  cudaError_t e;
  *added = 0;
  *max_overlap_new = 0.0;
  if (!reuse) ctx->list_valid = false;
  if (n == 0) return cudaSuccess;
  const double h = ctx->params.linked_cell_size;
  const double tol_list = tol > kListReach ? tol : kListReach;
  const int ghosts = ctx->params.ghost_mode;
  const int lanes = n < (size_t)kFewCells ? 8 : 4;
  const unsigned pair_grid = grid_for((long long)n * lanes);
  bool use_list = reuse && ctx->list_valid && ctx->list_n == n;
  // the radius of the last step (or upload) bounds the centres at the start
  // of a step -- it is the largest distance of a cell's leading end, so a
  // centre is at most half a cell further out and a new daughter's a quarter
  // more -- which saves the round trip for the bins' bounding box; a colony
  // that left the plane z = 0 once does not try again
  Grid g{};
  bool boxed = !reuse && ctx->box_known && ctx->flat && box_of_radius(ctx->radius + 2 * ctx->params.l0, h, n, &g);
  if ((e = ctx->bin_of.reserve(3 * n, 0, s))) return e;
  if ((e = ctx->ghost.reserve(n, 0, s))) return e;
  if ((e = ctx->cand_cnt.reserve(n + 1, 0, s))) return e;
  if ((e = ctx->cand_off.reserve(n + 1, 0, s))) return e;
  if ((e = ctx->pk.reserve(n * kPack, 0, s))) return e;
  if ((e = ctx->plist.reserve(n * kList, 0, s))) return e;
  if ((e = ctx->plist_n.reserve(n + 1, 0, s))) return e;
  if ((e = ctx->slot_of.reserve(n + 1, 0, s))) return e;
  if ((e = ctx->xref.reserve(3 * n, 0, s))) return e;
  if ((e = ctx->bin_cells.reserve(n, 0, s))) return e;
  if ((e = ctx->bin_raw.reserve(n, 0, s))) return e;
  if ((e = ctx->inc_cnt.reserve(n + 1, ctx->ncons ? n : 0, s))) return e;
  if (ctx->ncons == 0) cudaMemsetAsync(ctx->inc_cnt.p, 0, n * sizeof(int), s);  // the emit passes add to them
  for (;;) {
    cudaMemsetAsync(reinterpret_cast<char*>(ctx->status) + kDetectBegin, 0, kDetectBytes, s);
    if (use_list) {
      // the slots of the pass that built the lists: bin_cells still maps slot -> cell
      k_repack<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), ctx->bin_cells.p, n, h, ghosts, ctx->xref.p,
                                              ctx->bin_of.p, ctx->pk.p, ctx->status);
      (lanes == 8 ? k_list_pass<false, 8> : k_list_pass<false, 4>)<<<pair_grid, kBlock, 0, s>>>(
          ctx->pk.p, ctx->slot_of.p, n, tol, phase, true, ctx->list_tol, h, ctx->bin_of.p, ctx->plist.p,
          ctx->plist_n.p, ctx->cand_cnt.p, ctx->cells.ncons.p, nullptr, ConsView{}, 0, 0, nullptr, ctx->status);
      ctx->launches += 2;
    } else {
      int* key = ctx->cand_cnt.p;  // per-cell bin key until the pair pass
      if (!boxed) {
        k_bin<false><<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), n, h, ghosts, g, ctx->bin_of.p, ctx->ghost.p,
                                                    nullptr, nullptr, ctx->status);
        ctx->launches++;
        cudaMemcpyAsync(ctx->status_host, ctx->status, kStatusBytes, cudaMemcpyDeviceToHost, s);
        if ((e = cudaStreamSynchronize(s))) return e;
        const DevStatus& st = *ctx->status_host;
        auto lo = [&](int d) { return (long long)(int)(~st.box_lo[d] ^ 0x80000000u); };
        auto hi = [&](int d) { return (long long)(int)(st.box_hi[d] ^ 0x80000000u); };
        const long long nx = hi(0) - lo(0) + 1, ny = hi(1) - lo(1) + 1, nz = hi(2) - lo(2) + 1;
        const long long most = 1LL << 30;
        if (nx <= 0 || ny <= 0 || nz <= 0 || nx > most || ny > most || nz > most || nx * ny > most ||
            nx * ny * nz > most) {
          ctx->err = "broadphase grid too large (cells spread over more than 2^30 bins)";
          return cudaErrorInvalidValue;
        }
        g = Grid{(int)lo(0), (int)lo(1), (int)lo(2), (int)nx, (int)ny, (int)nz};
      }
      const size_t nbins = (size_t)g.nx * g.ny * g.nz;
      if ((e = ctx->bin_cnt.reserve(nbins + 1, 0, s))) return e;
      if ((e = ctx->bin_off.reserve(nbins + 1, 0, s))) return e;
      cudaMemsetAsync(ctx->bin_cnt.p, 0, nbins * sizeof(int), s);
      if (boxed)
        k_bin<true><<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), n, h, ghosts, g, ctx->bin_of.p, ctx->ghost.p,
                                                   key, ctx->bin_cnt.p, ctx->status);
      else
        k_bin_count<<<grid_for(n), kBlock, 0, s>>>(ctx->bin_of.p, n, g, key, ctx->bin_cnt.p);
      if ((e = exclusive_scan(ctx, ctx->bin_cnt.p, ctx->bin_off.p, nbins))) return e;
      k_bin_scatter<<<grid_for(n), kBlock, 0, s>>>(key, n, ctx->bin_off.p, ctx->bin_cnt.p, ctx->bin_raw.p,
                                                ctx->status);
      k_pack<<<grid_for(n), kBlock, 0, s>>>(ctx->cells.view(), ctx->bin_raw.p, key, ctx->bin_off.p, ctx->ghost.p, n,
                                            ctx->bin_cells.p, ctx->slot_of.p, ctx->pk.p, ctx->status);
      (lanes == 8 ? k_scan_count<8> : k_scan_count<4>)<<<pair_grid, kBlock, 0, s>>>(ctx->pk.p, ctx->bin_off.p, g, ctx->bin_of.p, n, tol, tol_list,
                                                ctx->cand_cnt.p, ctx->cells.ncons.p, ctx->plist.p, ctx->plist_n.p,
                                                ctx->xref.p, ctx->status);
      ctx->launches += 4;
    }
    if ((e = exclusive_scan(ctx, ctx->cand_cnt.p, ctx->cand_off.p, n, &ctx->status->count))) return e;
    cudaMemcpyAsync(ctx->status_host, ctx->status, kStatusBytes, cudaMemcpyDeviceToHost, s);
    if ((e = cudaStreamSynchronize(s))) return e;
    const DevStatus& st = *ctx->status_host;
    const unsigned flags = st.list_flags;
    if (!use_list && boxed && (flags & kOutOfBox)) {
      // a cell outside the assumed box: nothing was counted, start again
      boxed = false;
      if (st.nonplanar) ctx->flat = false;
      continue;
    }
    // cells that left the plane since the last full pass (out-of-plane
    // Brownian kicks) must take the general solver
    ctx->planar = st.nonplanar == 0;
    if (use_list && (flags & kListStale)) {
      // cells moved too far since the lists were built: rebin this phase
      use_list = false;
      ctx->list_valid = false;
      continue;
    }
    const bool listed = use_list || (flags & kListOverflow) == 0;
    if (use_list) ctx->prof.detect_list_passes++;
    else ctx->prof.detect_full_passes++;
    if (!use_list) {
      ctx->list_valid = listed;
      ctx->list_n = n;
      ctx->list_tol = tol_list;
    }
    const size_t m = (size_t)st.count;
    memcpy(max_overlap_new, &st.max_bits, sizeof *max_overlap_new);
    *added = m;
    if (m == 0) return cudaSuccess;
    if ((e = ctx->cons.reserve(ctx->ncons + m, ctx->ncons, s))) return e;
    if (listed) {
      (lanes == 8 ? k_list_pass<true, 8> : k_list_pass<true, 4>)<<<pair_grid, kBlock, 0, s>>>(
          ctx->pk.p, ctx->slot_of.p, n, tol, phase, use_list, tol_list, h, ctx->bin_of.p, ctx->plist.p,
          ctx->plist_n.p, nullptr, nullptr, ctx->cand_off.p, ctx->cons.view(), ctx->ncons, ctx->ncons + m,
          ctx->inc_cnt.p, ctx->status);
    } else {
      k_stencil_emit<<<grid_for(n), kBlock, 0, s>>>(ctx->pk.p, ctx->bin_off.p, g, ctx->bin_of.p, n, tol, phase,
                                                    ctx->cand_off.p, ctx->cons.view(), ctx->ncons, ctx->ncons + m,
                                                    ctx->inc_cnt.p, ctx->status);
    }
    ctx->launches++;
    ctx->ncons += m;
    return cudaGetLastError();
  }
}

cudaError_t build_incidence(pcc_ctx* ctx, bool order) {
  cudaStream_t s = ctx->stream;
  const size_t n = ctx->n, m = ctx->ncons;
  cudaError_t e;
  if ((e = ctx->inc_cnt.reserve(n + 1, n, s))) return e;
  if ((e = ctx->inc_off.reserve(n + 1, 0, s))) return e;
  if ((e = ctx->inc_cur.reserve(n + 1, 0, s))) return e;
  if ((e = ctx->inc_raw.reserve(2 * m + 1, 0, s))) return e;
  if ((e = ctx->inc_ent.reserve(2 * m + 1, 0, s))) return e;
  if ((e = exclusive_scan(ctx, ctx->inc_cnt.p, ctx->inc_off.p, n, nullptr, ctx->inc_cur.p))) return e;
  if (m) {
    k_inc_fill<<<grid_for(m), kBlock, 0, s>>>(ctx->cons.gi.p, ctx->cons.gj.p, m, ctx->inc_cur.p, ctx->inc_raw.p);
    ctx->launches++;
  }
  if (order && (e = order_incidence(ctx))) return e;
  return cudaGetLastError();
}

cudaError_t order_incidence(pcc_ctx* ctx) {
  const size_t ne = 2 * ctx->ncons;
  if (!ne) return cudaSuccess;
  k_inc_order<<<grid_for((long long)ne), kBlock, 0, ctx->stream>>>(ctx->cons.gi.p, ctx->cons.gj.p, ctx->inc_off.p,
                                                                  ctx->inc_raw.p, ne, ctx->inc_ent.p);
  ctx->launches++;
  return cudaGetLastError();
}

}  // namespace pcc
