// Planar BBPGD solver (sm_100a): the hard model's Barzilai-Borwein projected
// gradient (solver/BBPGD.cpp:32-127, gradient of
// dynamics/models/hard/HardModelGradient.cpp:89-158) for a colony whose cells
// all lie in z = 0 and rotate about z only.  Then a D row has three non-zero
// entries per side (n_x, n_y and the z torque arm) and U three per cell
// (u_x, u_y, w_z); every other term of the general kernel is an exact zero,
// and a running sum that starts at +0 is unchanged by adding a signed zero,
// so skipping them gives the general kernel's values.
//
// One persistent launch runs the whole solve.  Each iteration is two passes
// separated by grid barriers:
//   cell pass: kLanes lanes per cell walk the cell's incidence entries
//     (ascending constraint order, lane l takes entries l, l + kLanes, ...),
//     each entry a coalesced read of its D row and the constraint's
//     gamma_old, and a read of the (gamma, g) pair of the previous iteration
//     from the constraint itself (entry 2c + side); gamma_k =
//     max(gamma_{k-1} - alpha g_{k-1}, 0) is formed on the fly, the lanes'
//     sums of F = D^T (gamma_k - gamma_old) and sigma = L^T gamma_k are combined
//     by a fixed shuffle tree, and the first lane forms U = M F, the growth
//     rate and its change;
//   constraint pass: a few constraints per thread in fixed chunks
//     (chunk_count, chunk_lo), phi_next = Phi + dt D U - dt L dldot, the new
//     (gamma_k, g_k) written over the constraint's previous pair, and the
//     three Barzilai-Borwein dot products and the residual reduced per chunk
//     by a fixed shuffle tree.
// The (gamma, g) pairs are updated in place: the cell pass reads them before
// the first barrier and the constraint pass rewrites them after it, and each
// constraint's pair is read and rewritten by the same thread.  Gathering the
// pairs costs a 32-byte sector per scattered read; pushing copies to the two
// incidence entries instead (sequential reads in the cell pass) cost the same
// sector per scattered 16-byte write and measured 1.5-1.65x slower per
// iteration once the constraint set is several times the L2.  On residual
// iterations (the only ones that can end the solve) the
// constraint pass also stores gamma_{k-1}, the iterate the reference returns,
// and phi_next, so nothing has to be kept from the previous iteration.
// After the second barrier every block reduces the chunk partials in the same
// fixed order (in the traced form the last block to arrive does, and
// publishes the step size and the convergence decision).  The
// work of a chunk and of a cell never depends on which block does it, so the
// result does not depend on the grid size.  This kernel streams its operands
// from memory at every iteration: it takes the constraint sets that are too
// large for the on-chip kernels (pcc_resident.cu, which give its values bit
// for bit) and the traced solves.
//
// Real = double is the plain FP64 method.  Real = float is the
// mixed-precision form: D, L, M, U and the D / M products in FP32, while
// gamma, the gradient, Phi / phi_next, sigma = L^T gamma, the BB dot products
// and the residual stay FP64.
#include <cfloat>
#include <cmath>

#include "pcc_bbpgd.cuh"
#include "pcc_kernels.hpp"

namespace pcc {

namespace {

// The untraced kernel has two forms, by the blocks per SM that share the
// registers: three blocks with four entries of a lane in flight in the cell
// pass, and four blocks with two.  The second takes sets of exactly
// kChunkTarget long chunks, which its 592 blocks reduce in one round, where 444
// blocks need two, the second round with one block on each SM.  Measured, us
// per iteration, three blocks / four, on the constraints of one detection of a
// dense packing: FP64 170,516 14.7 / 13.6, 207,223 15.6 / 15.2, 291,819 18.7 /
// 18.3, 360,205 21.4 / 21.5, 456,347 26.0 / 26.9, 519,809 31.7 / 30.6, 654,571
// 38.4 / 36.8, 1,101,179 57.0 / 54.5; mixed 13.1 / 11.5, 14.2 / 12.3, 16.0 /
// 15.3, 17.3 / 16.0, 19.4 / 17.6, 22.0 / 18.7, 25.6 / 21.7, 41.9 / 38.1.  Over
// whole ReLCP calls, whose later phases repeat pairs (named by the last phase's
// constraints; the earlier ones are smaller): FP64 466,000 16.3 / 18.9, 723,000
// 19.7 / 21.5, 958,000 29.3 / 26.6, 1,224,000 36.2 / 29.3, 1,844,000 49.4 /
// 49.0, 2,868,000 72.9 / 79.6; mixed 14.7 / 16.3, 16.0 / 16.8, 21.1 / 19.5,
// 29.4 / 23.7, 38.7 / 36.6, 53.6 / 55.1.  A step's phases start with one
// detection's set and grow from it, so the line lies between the two: from
// 350,000 constraints on instead, calls that end with 466,000 to 848,000 take
// 1-4 % longer, from 650,000 on those that end with 958,000 to 1,224,000
// 3-13 %.  Registers spilled within the loops cost more than either choice
// gives (their counters are 32-bit for that); what is left, 16 bytes stored with
// three blocks in FP64 and 116 with four, none in mixed precision, is in these
// figures.
constexpr int kFewBlocks = 3, kManyBlocks = 4;
constexpr long long kLongChunks = 500000;

template <class Real>
struct PT;
template <>
struct PT<double> {
  using V2 = double2;
  using V4 = double4;
};
template <>
struct PT<float> {
  using V2 = float2;
  using V4 = float4;
};

template <class V4>
__device__ __forceinline__ V4 mk4(double a, double b, double c, double d);
template <>
__device__ __forceinline__ double4 mk4<double4>(double a, double b, double c, double d) {
  return make_double4(a, b, c, d);
}
template <>
__device__ __forceinline__ float4 mk4<float4>(double a, double b, double c, double d) {
  return make_float4((float)a, (float)b, (float)c, (float)d);
}
template <class V2>
__device__ __forceinline__ V2 mk2(double a, double b);
template <>
__device__ __forceinline__ double2 mk2<double2>(double a, double b) {
  return make_double2(a, b);
}
template <>
__device__ __forceinline__ float2 mk2<float2>(double a, double b) {
  return make_float2((float)a, (float)b);
}

template <class Real>
struct PArgs {
  using V2 = typename PT<Real>::V2;
  using V4 = typename PT<Real>::V4;
  long long m, n;
  // per constraint
  const int2* ij;
  const V2 *nn, *tt, *ss;  // (n_x, n_y), (t_iz, t_jz), (s_i, s_j)
  double* phi;             // Phi on entry, phi_next of the returned iterate on exit
  double* gamma;           // gamma_0 on entry, gamma_{k-1} on exit
  double* phin;            // phi_next of the last residual iteration
  double2* gg;             // (gamma, g) of the last iteration
  // per incidence entry
  const int* inc_off;
  const V4* inc;           // (D_x, D_y, D_t, s) of that side
  const double* gold;      // gamma_old of the entry's constraint
  const int* ent;          // the entry's constraint and side (2c + side)
  // per cell
  const V4* cell;          // (M_lin, M_rot, len, ldot_prev)
  V4* u;                   // (u_x, u_y, w_z, dldot)
  const double* uext;      // rotational U_ext, 3 per cell (z used: monolayer kicks); null: zero
  double *U, *F, *sig, *ldot, *imp;  // general-layout outputs, written on residual iterations
  double dt, lambda, tau, tol;
  long long max_it;
  double4* partials;       // one per chunk: (sum dgam^2, sum dgam*dg, sum dg^2, max residual)
  long long nchunks;       // chunk_count(m)
  SolverScalars* sc;
  DevStatus* st_err;
  // BBPGD trace (-log_bbgd_trace), as in the general kernel
  int trace;
  double* tr_part;
  double* trace_out;
  long long trace_cap;
};

__device__ __forceinline__ double lane_add(double a, double b) { return add(a, b); }
__device__ __forceinline__ float lane_add(float a, float b) { return __fadd_rn(a, b); }

template <int kN>
struct Count {
  static constexpr int value = kN;
};

// Lane sums of one cell over its incidence entries.
template <class Real>
struct CellAcc {
  Real f0 = 0, f1 = 0, f5 = 0;
  double sg = 0.0, g0 = 0.0, g1 = 0.0, g5 = 0.0;
};

// Cell pass.  mode 0: gamma = gamma_0 (the initial gradient); mode 1: gamma_k
// projected from the entries' (gamma, g) with step alpha.  A lane group
// takes one cell per round and loads the next cell's incidence range and
// record while it walks the current cell's entries, so the two loads are in
// flight together; each cell's sums do not depend on which group takes it.
template <class Real, class U, int kTr, int kAhead>
__device__ __forceinline__ void cell_pass(const PArgs<Real>& a, int mode, double alpha, bool final, double* eq,
                                          double* eg, int set = 0) {
  using V4 = typename PT<Real>::V4;
  constexpr bool kF64 = sizeof(Real) == 8;
  const int lane = threadIdx.x & 31, gl = lane % kLanes;
  constexpr int kCellsPerWarp = 32 / kLanes;
  auto accumulate = [&](CellAcc<Real>& A, const V4& d, double go, double gc) {
    const double diff = sub(gc, go);
    if constexpr (kF64) {
      A.f0 = add(A.f0, mul(d.x, diff));
      A.f1 = add(A.f1, mul(d.y, diff));
      A.f5 = add(A.f5, mul(d.z, diff));
      A.sg = add(A.sg, mul(d.w, gc));
    } else {
      const float df = (float)diff;
      A.f0 = fmaf(d.x, df, A.f0);
      A.f1 = fmaf(d.y, df, A.f1);
      A.f5 = fmaf(d.z, df, A.f5);
      A.sg = fma((double)d.w, gc, A.sg);
    }
    if constexpr (kTr) {
      A.g0 = add(A.g0, mul((double)d.x, gc));
      A.g1 = add(A.g1, mul((double)d.y, gc));
      A.g5 = add(A.g5, mul((double)d.z, gc));
    }
  };
  // kN entries of a lane from k on: all loads, then the sums in order
  auto take_entries = [&](CellAcc<Real>& A, int k, auto count) {
    constexpr int kN = decltype(count)::value;
    int c[kN];
    double go[kN];
    V4 d[kN];
    double2 p[kN];
    if (mode != 0) {
#pragma unroll
      for (int q = 0; q < kN; ++q) c[q] = a.ent[k + q * kLanes] >> 1;
    }
#pragma unroll
    for (int q = 0; q < kN; ++q) {
      d[q] = ld256(a.inc + k + q * kLanes);
      go[q] = a.gold[k + q * kLanes];
    }
    if (mode != 0) {
#pragma unroll
      for (int q = 0; q < kN; ++q) p[q] = a.gg[c[q]];
    }
#pragma unroll
    for (int q = 0; q < kN; ++q) accumulate(A, d[q], go[q], mode != 0 ? project(p[q].x, p[q].y, alpha) : go[q]);
  };
  auto combine = [&](CellAcc<Real>& A) {  // fixed shuffle tree over the group's lanes
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) {
      A.f0 = lane_add(A.f0, __shfl_xor_sync(kFull, A.f0, o));
      A.f1 = lane_add(A.f1, __shfl_xor_sync(kFull, A.f1, o));
      A.f5 = lane_add(A.f5, __shfl_xor_sync(kFull, A.f5, o));
      A.sg = add(A.sg, __shfl_xor_sync(kFull, A.sg, o));
      if constexpr (kTr) {
        A.g0 = add(A.g0, __shfl_xor_sync(kFull, A.g0, o));
        A.g1 = add(A.g1, __shfl_xor_sync(kFull, A.g1, o));
        A.g5 = add(A.g5, __shfl_xor_sync(kFull, A.g5, o));
      }
    }
  };
  auto finish = [&](int p, const CellAcc<Real>& A, const V4& cl, double uez) {
    double ux, uy, wz;
    if constexpr (kF64) {
      ux = add(add(0.0, mul(cl.x, A.f0)), 0.0);
      uy = add(add(0.0, mul(cl.x, A.f1)), 0.0);
      wz = add(add(0.0, mul(cl.y, A.f5)), uez);  // U = U_ext + M F (HardModelGradient.cpp:21)
    } else {
      ux = cl.x * A.f0;
      uy = cl.x * A.f1;
      wz = (double)(cl.y * A.f5) + uez;
    }
    const double im = exp(vscale(-a.lambda, A.sg));
    const double ld = vscale(dvd(1.0, a.tau), mul((double)cl.z, im));
    a.u[p] = mk4<V4>(ux, uy, wz, sub(ld, (double)cl.w));
    if constexpr (kTr) {
      const double ml = cl.x, mr = cl.y;
      *eq = add(*eq, add(add(mul(A.g0, mul(ml, A.g0)), mul(A.g1, mul(ml, A.g1))), mul(A.g5, mul(mr, A.g5))));
      *eg = add(*eg, mul((double)cl.z, im));
    }
    if (final) {
      double* Up = a.U + 6 * (size_t)p;
      double* Fp = a.F + 6 * (size_t)p;
      Up[0] = ux;
      Up[1] = uy;
      Up[2] = 0.0;
      Up[3] = 0.0;
      Up[4] = 0.0;
      Up[5] = wz;
      Fp[0] = A.f0;
      Fp[1] = A.f1;
      Fp[2] = 0.0;
      Fp[3] = 0.0;
      Fp[4] = 0.0;
      Fp[5] = A.f5;
      a.sig[p] = A.sg;
      a.ldot[p] = ld;
      a.imp[p] = im;
    }
  };
  // Cell units: unit u is the cells [16 u, 16 u + 16), one per lane group of
  // a warp.  Warp w (of W) starts with unit w; the untraced multi-block pass
  // then draws its further units from kTakeGroups counters of counter set
  // `set` (warp w from counter w % kTakeGroups, whose units are W + (w % kTakeGroups) +
  // kTakeGroups j), so blocks that run fast take more cells and the pass ends
  // with the memory system still busy; the other forms keep the static order
  // w, w + W, w + 2W, ...  A unit is drawn one round ahead (the first draw
  // alongside the first unit's loads) and its cells' ranges are loaded one
  // round ahead of their use.  Which warp does a cell changes nothing in its
  // sums.
  constexpr bool kDyn = !kTr && U::kGrid;
  const int W = (int)U::warps(), units = (int)((a.n + kCellsPerWarp - 1) / kCellsPerWarp), n = (int)a.n;
  const int grp = (int)U::warp() % kTakeGroups;
  unsigned long long* take = kDyn ? &a.sc->take[set][grp][0] : nullptr;
  int ucur = (int)U::warp(), unext = ucur + W;
  int p = ucur * kCellsPerWarp + lane / kLanes;
  int b = 0, e = 0;
  V4 cl{};
  double uez = 0.0;
  if constexpr (kDyn) {
    unext = units;
    if (ucur < units && lane == 0) unext = W + grp + kTakeGroups * (int)atomicAdd(take, 1ULL);
  }
  if (p < n) {
    b = a.inc_off[p];
    e = a.inc_off[p + 1];
    cl = a.cell[p];
    if (a.uext) uez = a.uext[3 * (size_t)p + 2];
  }
  if constexpr (kDyn) unext = __shfl_sync(kFull, unext, 0);
  while (ucur < units) {
    int uafter = unext + W;
    if constexpr (kDyn) {
      uafter = units;
      if (unext < units && lane == 0) uafter = W + grp + kTakeGroups * (int)atomicAdd(take, 1ULL);
    }
    const int pn = unext * kCellsPerWarp + lane / kLanes;
    int bn = 0, en = 0;
    V4 cln{};
    double uezn = 0.0;
    if (pn < n) {
      bn = a.inc_off[pn];
      en = a.inc_off[pn + 1];
      cln = a.cell[pn];
      if (a.uext) uezn = a.uext[3 * (size_t)pn + 2];
    }
    CellAcc<Real> A;
    int k = b + gl;
    for (; k + (kAhead - 1) * kLanes < e; k += kAhead * kLanes) take_entries(A, k, Count<kAhead>());
    for (; k < e; k += kLanes) take_entries(A, k, Count<1>());
    combine(A);
    if (gl == 0 && p < n) finish(p, A, cl, uez);
    if constexpr (kDyn) uafter = __shfl_sync(kFull, uafter, 0);
    ucur = unext;
    unext = uafter;
    p = pn;
    b = bn;
    e = en;
    cl = cln;
    uez = uezn;
  }
}

// phi_next of constraint c given U and dldot (MatMult row c in ascending
// columns: gi < gj, so the i block first; VecMAXPY(phi_next, {dt, -dt}, ...)).
// Zeroes counter set `set` of the cell-unit counters.  Iteration k's cell
// pass draws from set k % 2; set (k + 1) % 2 was last drawn from by iteration
// k - 1, so one thread zeroes it between the two barriers of iteration k and
// the second barrier orders that before iteration k + 1 draws from it.
__device__ __forceinline__ void reset_take(SolverScalars* sc, int set) {
#pragma unroll
  for (int g = 0; g < kTakeGroups; ++g) sc->take[set][g][0] = 0;
}

template <class Real>
__device__ __forceinline__ double planar_grad(const PArgs<Real>& a, int c) {
  const int2 ij = a.ij[c];
  const auto n = a.nn[c];
  const auto t = a.tt[c];
  const auto s = a.ss[c];
  const auto ui = ld256w(a.u + ij.x);
  const auto uj = ld256w(a.u + ij.y);
  if constexpr (sizeof(Real) == 8) {
    double pd = 0.0;
    pd = add(pd, mul(n.x, ui.x));
    pd = add(pd, mul(n.y, ui.y));
    pd = add(pd, mul(t.x, ui.z));
    pd = add(pd, mul(-n.x, uj.x));
    pd = add(pd, mul(-n.y, uj.y));
    pd = add(pd, mul(t.y, uj.z));
    double gr = 0.0;
    gr = add(gr, mul(s.x, ui.w));
    gr = add(gr, mul(s.y, uj.w));
    return add(a.phi[c], add(mul(a.dt, pd), mul(-a.dt, gr)));
  } else {
    float pd = n.x * ui.x;
    pd = fmaf(n.y, ui.y, pd);
    pd = fmaf(t.x, ui.z, pd);
    pd = fmaf(-n.x, uj.x, pd);
    pd = fmaf(-n.y, uj.y, pd);
    pd = fmaf(t.y, uj.z, pd);
    const float gr = fmaf(s.y, uj.w, s.x * ui.w);
    return a.phi[c] + a.dt * ((double)pd - (double)gr);
  }
}

// Constraints of chunk ch, and how many of a block's chunks have them kept in
// shared memory (two 64-bit divisions otherwise).
constexpr int kBounds = 8;
__device__ __forceinline__ int2 chunk_range(int ch, long long m, long long nchunks) {
  return make_int2((int)chunk_lo(ch, m, nchunks), (int)chunk_lo(ch + 1, m, nchunks));
}

// Constraint pass: new (gamma, g) over the constraint's pair, chunk partials.
// mode 0 evaluates g at gamma_0 (residual only).
template <class Real, class U, int kTr>
__device__ __forceinline__ void constraint_pass(const PArgs<Real>& a, int mode, double alpha, bool check, double* sm,
                                                double* smt, const int2* bounds = nullptr) {
  double2* gg = a.gg;
  for (int ch = (int)U::unit(), round = 0; ch < (int)a.nchunks; ch += (int)U::units(), ++round) {
    double v[4] = {0, 0, 0, 0};
    double lin = 0.0;
    const int2 range = bounds && round < kBounds ? bounds[round] : chunk_range(ch, a.m, a.nchunks);
    const int hi = range.y;
#pragma unroll 2
    for (int c = range.x + U::t(); c < hi; c += kBlock) {
      const double2 s = gg[c];
      const double gam = mode == 0 ? s.x : project(s.x, s.y, alpha);
      const double g = planar_grad(a, c);
      const double2 r = make_double2(gam, g);
      gg[c] = r;
      if (mode != 0 && check) {  // what the solve returns if it ends here (Hard.cpp:170, BBPGD.cpp:124)
        a.gamma[c] = s.x;
        a.phin[c] = g;
      }
      if (mode != 0) {
        const double dgm = sub(gam, s.x), dg = sub(g, s.y);
        v[0] = add(v[0], mul(dgm, dgm));
        v[1] = add(v[1], mul(dgm, dg));
        v[2] = add(v[2], mul(dg, dg));
      }
      if (mode == 0 || check) {
        const double rr = proj_grad_abs(g, gam);
        v[3] = v[3] < rr ? rr : v[3];
      }
      if constexpr (kTr) lin = add(lin, mul(gam, a.phi[c]));
    }
    unit_reduce4<U>(v, sm);
    if (U::t() == 0) a.partials[ch] = make_double4(v[0], v[1], v[2], v[3]);
    if constexpr (kTr) {
      if (a.trace) {
        double w[4] = {lin, 0, 0, 0};
        block_reduce4(w, smt);
        if (threadIdx.x == 0) a.tr_part[2 * gridDim.x + ch] = w[0];
      }
    }
  }
}

__device__ __forceinline__ void trace_cells(double* smt, double eq, double eg, double* tr_part) {
  double v[4] = {eq, eg, 0, 0};
  block_reduce4(v, smt);
  if (threadIdx.x == 0) {
    tr_part[2 * blockIdx.x] = v[0];
    tr_part[2 * blockIdx.x + 1] = v[1];
  }
}

template <class Real, int kTr, int kBlocks>
__global__ void __launch_bounds__(kBlock, kTr ? 1 : kBlocks) k_bbpgd_planar(PArgs<Real> a) {
  __shared__ double sm[4 * (kBlock / 32)];
  __shared__ double smt[kTr ? 4 * kBlock : 1];
  constexpr int kAhead = kBlocks == kManyBlocks ? 2 : 4;
  const int TR = kTr ? a.trace : 0;
  const unsigned nb = gridDim.x;
  SolverScalars* sc = a.sc;
  GridBarrier bar{sc, a.st_err, nb};
  if constexpr (!kTr) {
    // Untraced: every block reduces the chunk partials itself after a plain
    // grid barrier, in the same fixed order, so every block holds the same
    // bits of the step size and of the convergence decision and nothing is
    // published between blocks.  Block 0 records the scalars for the host
    // and zeroes the cell-unit counters of the next iteration.
    __shared__ double s_v[4];
    __shared__ int2 s_bounds[kBounds];
    if (threadIdx.x < kBounds) s_bounds[threadIdx.x] = chunk_range(blockIdx.x + threadIdx.x * nb, a.m, a.nchunks);
    auto reduce_all = [&](double v[4]) {
      reduce_partials<GridUnits>(a.partials, a.nchunks, v, sm);
      if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) s_v[q] = v[q];
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = s_v[q];
    };
    const bool recorder = blockIdx.x == 0 && threadIdx.x == 0;
    cell_pass<Real, GridUnits, 0, kAhead>(a, 0, 0.0, false, nullptr, nullptr, 0);
    if (!bar.sync()) return;
    if (recorder) reset_take(sc, 1);
    constraint_pass<Real, GridUnits, 0>(a, 0, 0.0, true, sm, nullptr, s_bounds);
    if (!bar.sync()) return;
    double v[4];
    reduce_all(v);
    double alpha = 1.0 / v[3];
    if (recorder) {
      sc->res0 = v[3];
      sc->residual = v[3];
      sc->alpha = alpha;
    }
    long long it = 1;
    bool conv = false;
    while (it < a.max_it) {
      const bool check = (it % 10) == 0;
      cell_pass<Real, GridUnits, 0, kAhead>(a, 1, alpha, check, nullptr, nullptr, (int)(it & 1));
      if (!bar.sync()) return;
      if (recorder) reset_take(sc, (int)((it + 1) & 1));
      constraint_pass<Real, GridUnits, 0>(a, 1, alpha, check, sm, nullptr, s_bounds);
      if (!bar.sync()) return;
      reduce_all(v);
      if (check && v[3] <= a.tol) conv = true;
      if (!conv) alpha = bb_step(v, it);
      if (recorder) {
        if (check) sc->residual = v[3];
        sc->alpha = alpha;
        sc->converged = conv ? 1 : 0;
        sc->iterations = it;
      }
      if (conv) break;
      ++it;
    }
    if (recorder) sc->iterations = it;
    if (!conv) return;
    const long long tid = (long long)blockIdx.x * kBlock + threadIdx.x, stride = (long long)nb * kBlock;
    double most = 0.0;
    for (long long c = tid; c < a.m; c += stride) {
      const double phi = ldcg(a.phin + c);
      a.phi[c] = phi;
      most = overlap_of(most, phi);
    }
    fold_overlap(sc, most);
    return;
  }

  // gradient at gamma_0 and the initial residual (BBPGD.cpp:40-44)
  {
    double eq = 0.0, eg = 0.0;
    cell_pass<Real, GridUnits, kTr, kAhead>(a, 0, 0.0, false, &eq, &eg);
    if (TR) trace_cells(smt, eq, eg, a.tr_part);
  }
  if (!bar.sync()) return;
  constraint_pass<Real, GridUnits, kTr>(a, 0, 0.0, true, sm, smt);
  auto reduce_init = [&]() {
    double v[4];
    reduce_partials<GridUnits>(a.partials, a.nchunks, v, sm);
    if (threadIdx.x == 0) {
      sc->res0 = v[3];
      sc->residual = v[3];
      sc->alpha = 1.0 / v[3];
      sc->converged = 0;
    }
    if (TR)
      trace_record(smt, a.tr_part, nb, a.nchunks, a.dt, a.lambda, a.tau, 0, v[3], 1.0 / v[3], a.trace_out,
                   a.trace_cap);
  };
  if (!bar.sync_reduce(reduce_init)) return;

  long long it = 1;
  while (it < a.max_it) {
    const double alpha = *(volatile double*)&sc->alpha;
    // with the trace on the residual is evaluated (and tested) every iteration (BBPGD.cpp:73)
    const bool check = (it % 10) == 0 || TR;
    {
      double eq = 0.0, eg = 0.0;
      cell_pass<Real, GridUnits, kTr, kAhead>(a, 1, alpha, check, &eq, &eg);
      if (TR) trace_cells(smt, eq, eg, a.tr_part);
    }
    if (!bar.sync()) return;
    constraint_pass<Real, GridUnits, kTr>(a, 1, alpha, check, sm, smt);
    auto reduce_iter = [&]() {
      double v[4];
      reduce_partials<GridUnits>(a.partials, a.nchunks, v, sm);
      if (TR)
        trace_record(smt, a.tr_part, nb, a.nchunks, a.dt, a.lambda, a.tau, it, v[3], alpha, a.trace_out,
                     a.trace_cap);
      if (threadIdx.x == 0) {
        int conv = 0;
        if (check) {
          sc->residual = v[3];
          // a recording-only trace (trace == 2) keeps the every-10th test
          if (v[3] <= a.tol && (TR != 2 || it % 10 == 0)) conv = 1;
        }
        if (!conv) sc->alpha = bb_step(v, it);
        sc->converged = conv;
        sc->iterations = it;
      }
    };
    if (!bar.sync_reduce(reduce_iter)) return;
    if (*(volatile int*)&sc->converged) break;
    ++it;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) sc->iterations = it;
  if (!*(volatile int*)&sc->converged) return;
  // returned result (Hard.cpp:170 with BBPGD.cpp:124): gamma_{k-1} (stored by
  // the last constraint pass), phi of gamma_k
  const long long tid = (long long)blockIdx.x * kBlock + threadIdx.x, stride = (long long)nb * kBlock;
  double most = 0.0;
  for (long long c = tid; c < a.m; c += stride) {
    const double phi = ldcg(a.phin + c);
    a.phi[c] = phi;
    most = overlap_of(most, phi);
  }
  fold_overlap(sc, most);
}

// ---------------------------------------------------------------- packing
template <class Real>
__global__ void k_pack_planar_cons(ConsView cs, long long m, int2* __restrict__ ij,
                                   typename PT<Real>::V2* __restrict__ nn, typename PT<Real>::V2* __restrict__ tt,
                                   typename PT<Real>::V2* __restrict__ ss, double2* __restrict__ gg0) {
  using V2 = typename PT<Real>::V2;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m) return;
  ij[c] = make_int2(cs.gi[c], cs.gj[c]);
  nn[c] = mk2<V2>(cs.nx[c], cs.ny[c]);
  tt[c] = mk2<V2>(cs.tiz[c], cs.tjz[c]);
  ss[c] = mk2<V2>(cs.si[c], cs.sj[c]);
  gg0[c] = make_double2(cs.gamma[c], 0.0);
}

// Per incidence entry, from the unordered lists to its place in the ordered
// ones: the entry, its side's D row and the constraint's gamma_old.
template <class Real>
__global__ void k_pack_planar_inc(ConsView cs, const int* __restrict__ off, const int* __restrict__ raw, size_t ne,
                                  int* __restrict__ ents, typename PT<Real>::V4* __restrict__ inc,
                                  double* __restrict__ gold) {
  using V4 = typename PT<Real>::V4;
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ne) return;
  int at;
  const int ent = entry_place(cs.gi, cs.gj, off, raw, k, &at);
  const long long c = ent >> 1;
  ents[at] = ent;
  if ((ent & 1) == 0)
    inc[at] = mk4<V4>(cs.nx[c], cs.ny[c], cs.tiz[c], cs.si[c]);
  else
    inc[at] = mk4<V4>(-cs.nx[c], -cs.ny[c], cs.tjz[c], cs.sj[c]);
  gold[at] = cs.gamma[c];
}

template <class Real>
__global__ void k_pack_planar_cells(const double* __restrict__ Ml, const double* __restrict__ Mr,
                                    const double* __restrict__ len, const double* __restrict__ ldot_prev, long long n,
                                    typename PT<Real>::V4* __restrict__ cell) {
  using V4 = typename PT<Real>::V4;
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  cell[p] = mk4<V4>(Ml[p], Mr[p], len[p], ldot_prev[p]);
}

template <class Real>
struct PlanarBufs;
template <>
struct PlanarBufs<double> {
  static pcc::DevBuf<double2>& nn(pcc_ctx* c) { return c->p_n; }
  static pcc::DevBuf<double2>& tt(pcc_ctx* c) { return c->p_t; }
  static pcc::DevBuf<double2>& ss(pcc_ctx* c) { return c->p_s; }
  static pcc::DevBuf<double4>& inc(pcc_ctx* c) { return c->p_inc; }
  static pcc::DevBuf<double4>& cell(pcc_ctx* c) { return c->p_cell; }
  static pcc::DevBuf<double4>& u(pcc_ctx* c) { return c->p_u; }
};
template <>
struct PlanarBufs<float> {
  static pcc::DevBuf<float2>& nn(pcc_ctx* c) { return c->pf_n; }
  static pcc::DevBuf<float2>& tt(pcc_ctx* c) { return c->pf_t; }
  static pcc::DevBuf<float2>& ss(pcc_ctx* c) { return c->pf_s; }
  static pcc::DevBuf<float4>& inc(pcc_ctx* c) { return c->pf_inc; }
  static pcc::DevBuf<float4>& cell(pcc_ctx* c) { return c->pf_cell; }
  static pcc::DevBuf<float4>& u(pcc_ctx* c) { return c->pf_u; }
};

template <class Real>
cudaError_t launch(pcc_ctx* ctx, double dt, const PlanarTrace& tr, int* kind) {
  using B = PlanarBufs<Real>;
  cudaStream_t s = ctx->stream;
  const size_t n = ctx->n, m = ctx->ncons, ne = 2 * m;
  const size_t mm = m + 1, nn = n + 1;
  cudaError_t e;
  if ((e = ctx->p_ij.reserve(mm, 0, s)) || (e = ctx->p_gg.reserve(mm, 0, s)) || (e = ctx->p_phin.reserve(mm, 0, s)) ||
      (e = ctx->p_gold.reserve(ne + 1, 0, s)))
    return e;
  if ((e = B::nn(ctx).reserve(mm, 0, s)) || (e = B::tt(ctx).reserve(mm, 0, s)) || (e = B::ss(ctx).reserve(mm, 0, s)) ||
      (e = B::inc(ctx).reserve(ne + 1, 0, s)) || (e = B::cell(ctx).reserve(nn, 0, s)) ||
      (e = B::u(ctx).reserve(nn, 0, s)))
    return e;
  const long long nchunks = chunk_count((long long)m);
  if ((e = ctx->partials.reserve(4 * (nchunks + 1), 0, s))) return e;
  ConsView cv = ctx->cons.view();
  if (m) {
    k_pack_planar_cons<Real><<<grid_for((long long)m), kBlock, 0, s>>>(cv, (long long)m, ctx->p_ij.p, B::nn(ctx).p,
                                                                       B::tt(ctx).p, B::ss(ctx).p, ctx->p_gg.p);
    k_pack_planar_inc<Real><<<grid_for((long long)ne), kBlock, 0, s>>>(
        cv, ctx->inc_off.p, ctx->inc_raw.p, ne, ctx->inc_ent.p, B::inc(ctx).p, ctx->p_gold.p);
    ctx->launches += 2;
  }
  if (n) {
    k_pack_planar_cells<Real><<<grid_for((long long)n), kBlock, 0, s>>>(
        ctx->Mlin.p, ctx->Mrot.p, ctx->cells.len.p, ctx->cells.ldot.p, (long long)n, B::cell(ctx).p);
    ctx->launches++;
  }
  PArgs<Real> a;
  a.m = (long long)m;
  a.n = (long long)n;
  a.ij = ctx->p_ij.p;
  a.nn = B::nn(ctx).p;
  a.tt = B::tt(ctx).p;
  a.ss = B::ss(ctx).p;
  a.phi = cv.sd;
  a.gamma = cv.gamma;
  a.phin = ctx->p_phin.p;
  a.gg = ctx->p_gg.p;
  a.inc_off = ctx->inc_off.p;
  a.inc = B::inc(ctx).p;
  a.gold = ctx->p_gold.p;
  a.cell = B::cell(ctx).p;
  a.u = B::u(ctx).p;
  a.uext = ctx->uext_active ? ctx->uext.p : nullptr;
  a.U = ctx->U.p;
  a.F = ctx->F.p;
  a.sig = ctx->sig.p;
  a.ldot = ctx->ldot_new.p;
  a.imp = ctx->imp_new.p;
  a.dt = dt;
  a.lambda = ctx->params.lambda;
  a.tau = ctx->params.tau;
  a.tol = ctx->params.tolerance;
  a.max_it = ctx->params.max_bbpgd_iterations;
  a.partials = reinterpret_cast<double4*>(ctx->partials.p);
  a.nchunks = nchunks;
  a.ent = ctx->inc_ent.p;
  a.sc = &ctx->status->solver;
  a.st_err = ctx->status;
  a.trace = tr.trace;
  a.tr_part = tr.tr_part;
  a.trace_out = tr.trace_out;
  a.trace_cap = tr.trace_cap;
  void* args[] = {&a};
  if (ctx->profiling) cudaEventRecord(ctx->ev[0], s);
  const bool many = !tr.trace && nchunks == kChunkTarget && (long long)m >= kLongChunks;
  const void* kern = tr.trace ? (const void*)k_bbpgd_planar<Real, 1, kFewBlocks>
                     : many   ? (const void*)k_bbpgd_planar<Real, 0, kManyBlocks>
                              : (const void*)k_bbpgd_planar<Real, 0, kFewBlocks>;
  int& coop = ctx->coop_planar[sizeof(Real) == 8][tr.trace ? 0 : many ? 2 : 1];
  if (coop == 0) {
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlock, 0))) return e;
    const int cap = many ? kManyBlocks : kFewBlocks;
    coop = (per_sm < cap ? per_sm : cap) * ctx->num_sms;
  }
  long long want = (long long)grid_for((long long)n * kLanes);
  if (nchunks > want) want = nchunks;
  if (want > coop) want = coop;
  if (want < 1) want = 1;
  *kind = want > 1 ? 1 : 0;
  if (want == 1) return cudaLaunchKernel(kern, dim3(1), dim3(kBlock), args, 0, s);
  return cudaLaunchCooperativeKernel(kern, dim3((unsigned)want), dim3(kBlock), args, 0, s);
}

}  // namespace

long long planar_chunks(size_t m) { return chunk_count((long long)m); }

cudaError_t planar_bbpgd(pcc_ctx* ctx, double dt, bool mixed, const PlanarTrace& tr, int* kind) {
  return mixed ? launch<float>(ctx, dt, tr, kind) : launch<double>(ctx, dt, tr, kind);
}

}  // namespace pcc
