// Shared device-side definitions of the collision hot path (sm_100a).
//
// Cells live in structure-of-arrays form in global-id order (ids are ranks of
// the x-sort, spatial/Domain.cpp:492-508 of the reference).  Constraints live
// in structure-of-arrays form, appended phase by phase within a step.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "pcc_gpu.h"

namespace pcc {

constexpr int kBlock = 256;

// Error codes raised on the device (bitmask in DevStatus::flags).
enum : unsigned {
  kDevErrBounds = 1u << 0,     // an index fell outside its buffer
  kDevErrTimeout = 1u << 1,    // a bounded spin-wait gave up
  kDevErrCapacity = 1u << 2,   // a per-call capacity was exceeded
  kDevErrNan = 1u << 3,        // non-finite values appeared
};

// Grid barrier + reduction scratch of the persistent solver kernel.
// The arrival counter sits on a cache line of its own: every block adds to
// it at every grid barrier, while the release word and the scalars that the
// blocks read after a release share the next line.
constexpr int kTakeGroups = 8;
struct SolverScalars {
  unsigned long long arrive;     // block arrivals at grid barriers, monotonic within a launch
  unsigned long long pad0[15];
  unsigned long long released;   // ordinal of the last barrier whose reduction was published
  int converged;                 // 1 once the residual test passed
  int pad;
  long long iterations;          // BBPGD iteration count at exit
  double alpha;                  // current step size
  double residual;               // last evaluated residual
  double res0;                   // initial residual
  unsigned long long overlap_bits;  // largest overlap of the constraints after a converged solve
  // cell-unit counters of the multi-block planar cell pass, two sets used by
  // alternate iterations, one counter per 128-byte line
  alignas(128) unsigned long long take[2][kTakeGroups][16];
};
static_assert(offsetof(SolverScalars, take) == 256, "counters start on their own line");

struct DevStatus {
  unsigned flags;
  int where;
  // contact detection: cleared as one block at the start of a pass
  unsigned long long max_bits;    // running max of a non-negative double (bit pattern)
  unsigned long long drift_bits;  // largest squared displacement since the lists were built
  unsigned long long lmax_bits;   // longest cell
  unsigned list_flags;            // candidate lists overflowed / stale, cells outside the assumed box
  unsigned nonplanar;             // a cell is out of the plane
  unsigned box_lo[3], box_hi[3];  // bounding box of the bins, as keys whose maximum is taken (box_key)
  int count;                      // contacts found
  int pad;
  // end of a step
  unsigned long long radius_bits;  // colony radius
  unsigned long long median[2];    // the two middle adaptDt speeds, as ordered keys
  int divisions;                   // of the next step
  int crowded;                     // the last x-sort by buckets met a crowded one
  SolverScalars solver;  // of the last BBPGD launch
};
// What the host reads, in one copy: everything but the cell-unit counters.
constexpr size_t kStatusBytes = offsetof(DevStatus, solver) + offsetof(SolverScalars, take);
constexpr size_t kDetectBegin = offsetof(DevStatus, max_bits), kDetectBytes = offsetof(DevStatus, radius_bits) - kDetectBegin;

// Cell arrays (device pointers).
struct CellsView {
  double *x, *y, *z, *q0, *q1, *q2, *q3;
  double *len, *l0, *diam, *ldot, *imp, *stress;
  int* age;
  double* force;  // 6 per cell
  double* vel;    // 6 per cell
  int* ncons;     // contacts counted during the last solve (Particle::getNumConstraints)
};

// Constraint arrays (device pointers).  D row of constraint c
// (dynamics/Physics.cpp:118-154): [n, ti] at cell gi and [-n, tj] at cell gj
// with ti = ri x n and tj = rj x (-n).
struct ConsView {
  int *gi, *gj, *phase;
  double *sd, *gamma;
  double *nx, *ny, *nz;
  double *tix, *tiy, *tiz, *tjx, *tjy, *tjz;
  double *rix, *riy, *riz, *rjx, *rjy, *rjz;
  double *cpx, *cpy, *cpz;
  double *si, *sj;
};

// IEEE round-to-nearest arithmetic without contraction, so the geometry and
// the state update round exactly like the reference's strict build.
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }

// Unit axis of a cell: the quaternion applied to (1,0,0)
// (util/Quaternion.cpp:7-38, evaluated in the same order).
__device__ __forceinline__ void cell_axis(double w, double x, double y, double z, double t[3]) {
  const double vx = 1.0, vy = 0.0, vz = 0.0;
  const double c1x = sub(mul(y, vz), mul(z, vy));
  const double c1y = sub(mul(z, vx), mul(x, vz));
  const double c1z = sub(mul(x, vy), mul(y, vx));
  const double c2x = sub(mul(y, c1z), mul(z, c1y));
  const double c2y = sub(mul(z, c1x), mul(x, c1z));
  const double c2z = sub(mul(x, c1y), mul(y, c1x));
  const double w2 = mul(2.0, w);
  t[0] = add(add(vx, mul(w2, c1x)), mul(2.0, c2x));
  t[1] = add(add(vy, mul(w2, c1y)), mul(2.0, c2y));
  t[2] = add(add(vz, mul(w2, c1z)), mul(2.0, c2z));
}

__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  double r = 0.0;
  r = add(r, mul(a[0], b[0]));
  r = add(r, mul(a[1], b[1]));
  r = add(r, mul(a[2], b[2]));
  return r;
}

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double r[3]) {
  r[0] = sub(mul(a[1], b[2]), mul(a[2], b[1]));
  r[1] = sub(mul(a[2], b[0]), mul(a[0], b[2]));
  r[2] = sub(mul(a[0], b[1]), mul(a[1], b[0]));
}

// Incidence entry k of the unordered lists (2 c + side) and its place in
// ascending order among its cell's entries.
__device__ __forceinline__ int entry_place(const int* __restrict__ gi, const int* __restrict__ gj,
                                           const int* __restrict__ off, const int* __restrict__ raw, size_t k,
                                           int* at) {
  const int e = raw[k], p = (e & 1) ? gj[e >> 1] : gi[e >> 1], hi = off[p + 1];
  int s = off[p];
  for (int q = s; q < hi; ++q) s += raw[q] < e ? 1 : 0;
  *at = s;
  return e;
}

// Loads that bypass L1: data produced by other blocks of the same
// persistent kernel after a grid barrier.
template <typename T>
__device__ __forceinline__ T ldcg(const T* p) {
  return __ldcg(p);
}
template <>
__device__ __forceinline__ double4 ldcg<double4>(const double4* p) {
  const double2 lo = __ldcg(reinterpret_cast<const double2*>(p));
  const double2 hi = __ldcg(reinterpret_cast<const double2*>(p) + 1);
  return make_double4(lo.x, lo.y, hi.x, hi.y);
}

// One 32-byte load of a row of four, 32-byte aligned (rows of a buffer of the
// context): lanes that read scattered or strided rows cost L1 one lookup per
// row, not two.  ld256 is for rows that the kernel does not write, ld256w for
// rows that other blocks of it wrote before a grid barrier (not moved across
// it).  Streaming FP64 BBPGD, per iteration: 362,000 constraints (in L2) 22.8
// -> 20.4 us, 2.4 M (from DRAM) 114.4 -> 110.5; on-chip grid form, FP64,
// 76,000: 9.65 -> 9.05.
//
// ld256w and the solvers' other reads of (gamma, g) and velocity rows may stay
// in L1: a grid barrier is a release by every block and an acquire by every
// block, which drops the L1 lines of the SM, and the compiler keeps loads on
// their side of it.  Neighbouring constraints share cells, so a row is read
// again by the same SM: 20.4 -> 19.9 us per iteration (mixed 17.5 -> 16.5) and
// 109.5 -> 105.3 (91.0 -> 86.9) against loads that bypass L1.
__device__ __forceinline__ double4 ld256(const double4* p) {
  double4 r;
  asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
  return r;
}
__device__ __forceinline__ float4 ld256(const float4* p) { return *p; }  // 16 bytes: one load as it is
__device__ __forceinline__ double4 ld256w(const double4* p) {
  double4 r;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w)
               : "l"(p)
               : "memory");
  return r;
}
__device__ __forceinline__ float4 ld256w(const float4* p) { return *p; }

__device__ __forceinline__ void raise_error(DevStatus* st, unsigned flag, int where) {
  atomicOr(&st->flags, flag);
  atomicExch(&st->where, where);
}

// Monotone map of a double to an unsigned 64-bit key (ascending order
// preserved, -0 before +0).
__device__ __forceinline__ unsigned long long double_key(double v) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b & 0x8000000000000000ULL) ? ~b : (b | 0x8000000000000000ULL);
}

inline unsigned grid_for(long long n, int block = kBlock) {
  long long g = (n + block - 1) / block;
  if (g < 1) g = 1;
  if (g > 2147483647LL) g = 2147483647LL;
  return (unsigned)g;
}

}  // namespace pcc
