// Host-side launchers of the step kernels (implemented in gop_kernels.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "gamera_op.h"
#include "gop_device.cuh"

namespace gop {

// per-step work arrays, each field fs elements, element type R
template <typename R>
struct Work {
  R* Wh;   // 6 half-step primitives
  R* Ms;   // 3 cell-centred B at step start (PDM limiter reference)
  R* Msh;  // 3 half-step cell-centred B
  R* Bh;   // 3 half-step face fields
  R* V;    // 6 centre-to-edge first-sweep velocities (2 per edge direction)
  R* E;    // 3 edge EMFs
  R* F;    // 27 face fluxes (9 per direction)
  R* Wl;   // FP32 path: 6 step-start primitives in R (the limiters' reference)
  R* Bl;   // FP32 path: 3 step-start face fields in R
  const R* tab;  // the per-axis tables in R (same layout as Params::tab)
  const R* fw;   // the packed face records in R (tab + fw_offset(tmax))
};
constexpr int WORK_FIELDS = 6 + 3 + 3 + 3 + 6 + 3 + 27;
// the FP32 path adds the R copies of the step-start state (Wl, Bl)
constexpr int work_fields(bool mixed) { return WORK_FIELDS + (mixed ? 9 : 0); }

int64_t launches();
void count_launches(int64_t n);  // kernels run by graph replays

// kernel groups of one step, for event timing
enum Group : int { G_BEGIN = 0, G_AB2, G_C2C, G_EMF, G_FLUX, G_UPDATE, G_GHOST, G_END, NGROUP };

// launch shapes of the tunable kernels: AB2, C2C x3 (places of gop_autotune's
// result alone: their launch has one shape), EMF x3, FLUX x3, UPDATE
enum TuneSlot : int { K_AB2 = 0, K_C2C0, K_C2C1, K_C2C2, K_EMF0, K_EMF1, K_EMF2,
                      K_FLUX0, K_FLUX1, K_FLUX2, K_UPDATE, NTUNE };
struct Tune {
  dim3 blk[NTUNE];
  // the stage's fluxes / edge EMFs from the tile-staged sweep kernels
  // (gop_sweep.cu) instead of the per-point kernels, where the sweeps apply
  bool flux_sweep;
  bool emf_sweep;
  bool update_sweep;  // the update from tiles as well
  // order of the axes (independent) in the flux and EMF stages
  int flux_order[3];
  int emf_order[3];
  Tune();
};

// Tensor maps and launch data of an instance's tile-staged flux sweeps
// (gop_sweep.cu); null when they could not be made (the per-face kernels run)
struct SweepSet;
template <typename R>
SweepSet* sweep_create(const Params& P, const Work<R>& w);
void sweep_destroy(SweepSet* s);
// The fluxes (edge EMFs) of the three axes by the sweep kernels, their tiles
// in the given order; false (nothing launched) where the sweep does not apply
// (no maps; for the flux, the entropy channel is live)
template <typename R>
bool launch_flux_sweep(const SweepSet* sw, const Params& P, const Work<R>& w, const int order[3],
                       cudaStream_t st);
template <typename R>
bool launch_emf_sweep(const SweepSet* sw, const Params& P, const Work<R>& w, const int order[3],
                      cudaStream_t st);

// the update from TMA-filled tiles; false as above, on small grids, and on
// spherical ones with the pole ring average or on the mixed path
template <typename R>
bool update_sweep_applies(const SweepSet* sw, const Params& P);
template <typename R>
bool launch_update_sweep(const SweepSet* sw, const Params& P, const Work<R>& w, cudaStream_t st);

// points covered by the launch of one slot (x, y, z extents); none for K_C2C0..2,
// which are one launch of a fixed shape within launch_step_body
dim3 launch_space(const Params& P, int slot);

// launches one tunable kernel; pdl false: without programmatic dependent
// launch
template <typename R>
void launch_slot(const Params& P, int coord, const Work<R>& w, int slot, dim3 blk,
                 cudaStream_t st, bool pdl = true);

// optional timing hook: mark(ctx, group, start) records an event on the stream
struct Hook {
  void (*mark)(void* ctx, int group, int start) = nullptr;
  void* ctx = nullptr;
  void operator()(int g, int s) const {
    if (mark) mark(ctx, g, s);
  }
};
// arm a gop_step call: stop after time tstop or after `budget` steps; opens
// the first step
void launch_arm(const Params& P, double tstop, double budget, cudaStream_t st);
// CFL dt (in the form and arithmetic of the step's own estimate) and
// max|div B| of the current state
void launch_dt(const Params& P, int coord, bool mixed, cudaStream_t st);
// P.scal[S_PSNZ] <- 1 if p_S is nonzero in either state buffer, and with an
// uploaded history S_HISTG <- 1 if its periodic ghosts do not repeat its active
// cells (both must be 0 before)
void launch_state_check(const Params& P, bool history, cudaStream_t st);
template <typename R>
void launch_step_body(const Params& P, int coord, const Work<R>& w, cudaStream_t st,
                      const Tune& tune, const SweepSet* sw, const Hook& hook = Hook());
// what fills the ghost layers of each face (gas_bc_*, gem_bc_*: GOP_BC_*) and
// which axes are periodic
struct GhostFill {
  char gas[6], gem[6];
  bool per[3];
};
// which = 0: the buffer being written this step, and the turn to the next
// step; 1: the current state
void launch_ghosts(const Params& P, const char bc[6], const char gem_bc[6], int which,
                   cudaStream_t st);
// one field between the reference layout and the device's
void launch_from_ref(const Params& P, const double* src, double* dst, cudaStream_t st);
void launch_to_ref(const Params& P, const double* src, double* dst, cudaStream_t st);
template <typename R>
void launch_widen(const Params& P, int nf, const R* src, double* dst, cudaStream_t st);
void launch_mags(const Params& P, const double* B, double* out, cudaStream_t st);
// pole ring average (spherical grids reaching a pole): the pole-edge EMFs
// before the update; the ring averages of the new state after it (scratch:
// 2 fields of doubles)
template <typename R>
void launch_pole_emf(const Params& P, const Work<R>& w, cudaStream_t st);
void launch_ring_average(const Params& P, double* scratch, cudaStream_t st);
// background field B0 of a built-in kind into the background block out
// (BG_NF fields, zero beforehand); aux: 12 fields of doubles of scratch
void launch_background(const Params& P, const gop_background& bg, int sph, double* out, double* aux,
                       cudaStream_t st);
// problem p's initial state in buffer 0 (cells, face field; ghosts left for
// the ghost fill); scratch: 3 fields of doubles for the edge integrals
void launch_problem_init(const Params& P, const gop_problem& p, int sph, double* scratch,
                         cudaStream_t st);

}  // namespace gop
