// Host launchers of the device kernels (internal to libpcc_gpu.so).
#pragma once

#include <cuda_runtime.h>

#include "pcc_ctx.hpp"

namespace pcc {

// Slots of ctx->pinned_ll for values copied back at a synchronisation point.
constexpr int kSlotRadius = 10;  // colony radius bits
constexpr int kSlotDivs = 11;    // divisions of the next step
constexpr int kSlotCrowded = 12;  // a crowded bucket of the x-sort

// ---- pcc_scan_sort.cu
// out[i] = sum in[0..i-1] for i in [0, n]; out has n+1 entries.  The sum of
// all goes to *total too (a device address) if given, and entries [0, n) to
// copy.
cudaError_t exclusive_scan(pcc_ctx* ctx, const int* in, int* out, size_t n, int* total = nullptr, int* copy = nullptr);
// Stable ascending sort of (keys, vals) by the low `bits` bits of keys;
// keys/vals are sorted in place (scratch from ctx).
cudaError_t radix_sort_pairs(pcc_ctx* ctx, unsigned long long* keys, int* vals, size_t n, int bits);

// ---- pcc_detect.cu
// Appends the contacts within tol of the resident cells to the constraint set
// (ctx->ncons grows by *added).  *max_overlap_new = max(-sd, 0) over them.
// reuse = true lets a later ReLCP phase of the same step re-test the
// candidate lists of the previous full pass instead of rebinning; callers
// pass it only when the cells changed by constraint motion alone since.
cudaError_t detect_contacts(pcc_ctx* ctx, double tol, int phase, bool reuse, size_t* added,
                            double* max_overlap_new);
// Cell -> incident constraint sides for ctx->ncons: the offsets and, with
// order, the entries in ascending constraint order (inc_ent); without, the
// entries of each cell in no order (inc_raw), for order_incidence or a solver
// that orders them as it packs them.
cudaError_t build_incidence(pcc_ctx* ctx, bool order);
cudaError_t order_incidence(pcc_ctx* ctx);

// out[3 k + d] = component d of vector k, for n vectors.
cudaError_t interleave3(pcc_ctx* ctx, const double* x, const double* y, const double* z, size_t n, double* out);

// ---- pcc_solver.cu
// Draws the Brownian U_ext of every cell (temperature > 0) from the context's
// generator and sets ctx->uext_active; a no-op at temperature 0.
cudaError_t brownian_draw(pcc_ctx* ctx);
// One BBPGD solve on the current constraint set (hard model).  With defer,
// only launches it (ctx->bbpgd_pending);
// bbpgd_collect reads them after the caller's next synchronisation that also
// copied the device status.  It sets ctx->solved_overlap.  Expects the
// incidence without order.
cudaError_t bbpgd_solve(pcc_ctx* ctx, double dt, long long* iterations, double* residual, int* status,
                        bool defer = false);
void bbpgd_collect(pcc_ctx* ctx, long long* iterations, double* residual, int* status);
// Moves cells with the solver's velocities and writes back gamma / phi.
cudaError_t apply_hard_solution(pcc_ctx* ctx, double dt);
// Soft model: Hertz forces, motion and growth parameters.
cudaError_t soft_forces_and_move(pcc_ctx* ctx, double dt);
// Soft model force assembly only (frozen microbench).
cudaError_t soft_assemble(pcc_ctx* ctx);

// ---- pcc_planar.cu
// BBPGD trace buffers handed to the planar solver (trace = 0: none).
struct PlanarTrace {
  int trace;
  double* tr_part;
  double* trace_out;
  long long trace_cap;
};
// Constraint chunks of the planar solver's reductions for m constraints.
long long planar_chunks(size_t m);
// Packs the planar operands and launches the planar BBPGD solve on the
// context's stream (FP64, or mixed precision); *kind = 1 for the multi-block
// cooperative kernel, 0 for a one-block launch.
cudaError_t planar_bbpgd(pcc_ctx* ctx, double dt, bool mixed, const PlanarTrace& tr, int* kind);

// ---- pcc_resident.cu
// Launches the on-chip BBPGD solve (and the ordering of the incidence lists) if
// the constraint set fits it (*taken);
// full: six D components.  *kind as for planar_bbpgd.
cudaError_t resident_bbpgd(pcc_ctx* ctx, double dt, bool full, bool mixed, bool* taken, int* kind);

// ---- pcc_update.cu
cudaError_t reset_ldot(pcc_ctx* ctx);
// Growth; with step_end also the colony radius and the division flags of the
// next step (read by step_end_collect after the caller's synchronisation).
cudaError_t grow_cells(pcc_ctx* ctx, double dt, bool step_end);
// Division of every cell with len >= 2 l0, daughters appended; returns count.
// Uses the flags counted at the end of the previous step when ctx->div_known.
cudaError_t divide_cells(pcc_ctx* ctx, size_t* added);
// End of a step: the offsets and the count of the divisions flagged by
// grow_cells and, unless dt is fixed, the adaptDt median, all into the device
// status, whose one copy to ctx->status_host is queued; step_end_collect reads
// it after the caller's synchronisation (radius, divisions of the next step)
// and adapts ctx->params.dt.
cudaError_t step_end_enqueue(pcc_ctx* ctx);
void step_end_collect(pcc_ctx* ctx);
// Sort cells by x (stable) and renumber.
cudaError_t sort_cells_by_x(pcc_ctx* ctx);
cudaError_t colony_radius(pcc_ctx* ctx, double* out);
// Per-cell mobilities for the streaming solvers, unless ctx->mobility_known.
cudaError_t mobility(pcc_ctx* ctx);

// ---- pcc_vtk.cu
// Waits for and stops the context's VTK writer thread.
void vtk_writer_shutdown(pcc_ctx* ctx);
// Removes <dir>/<prefix>*.pvtu and <dir>/data/<prefix>*.vtu (a new logger's reset).
void vtk_clear_prefix(const std::string& dir, const std::string& prefix);
// bbpgdtrace_<index> files of BBPGDLogger::log, indices first_index, first_index + 1, ...
bool vtk_write_trace(const std::string& dir, unsigned long long first_index,
                     const std::vector<pcc_bbpgd_trace_step>& steps);

}  // namespace pcc
