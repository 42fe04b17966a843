// Interface between the ghost-cell translation unit (ghostmac.cu) and the cut-cell one
// (cutcell.cu): a pressure-only handle built over a cut-cell geometry runs the boundary-
// corrected separable inverse of the ghost path (rectangle transforms, column solves, Schur
// band chain, residual checks and refinement sweeps) on the cut-cell Poisson operator.
#pragma once
#include <cuda_runtime.h>

#include <array>
#include <cstdint>
#include <functional>
#include <string>

#include "../../include/ghostmac.h"
#include "geometry.hpp"
#include "kernels.cuh"

struct gm_handle;

// the per-thread message of a failed call made without a handle (gm_last_error(NULL))
void gm_internal_set_error(const char* msg);

namespace gmi {

// Pressure-only handle over `g` (filled by gm::build_cutcell_geometry); GM_OK or an error
// class with the message in err.  FP64 operator and inverse; three residual checks per solve.
int pressure_create(gm::Geometry&& g, gm_handle** out, std::string& err);
void pressure_destroy(gm_handle* h);
const gm::Geometry& geometry(const gm_handle* h);
cudaStream_t stream(gm_handle* h);
// streams that capture the bodies of conditional graph nodes
cudaStream_t body_stream(gm_handle* h, int level);
// while set, pressure_solve queues (or records) as many gated refinement sweeps as its slot holds; a solve
// that needs more raises gmk::ERR_SWEEPS with the slot as the gate word
void hold_sweeps(gm_handle* h, bool on);
int checks(const gm_handle* h);            // residual checks of a solve at most
// Monitored solve of A x = b (full pressure grids on the device, inactive cells ignored in b
// and zero in x) in control slot `slot` (gmk::S_P0..S_P2), then its pressure gate.
void pressure_solve(gm_handle* h, const double* b, double* x, int slot);
// b - A x after the last solve's final check (pressure grid)
const double* pressure_residual(gm_handle* h);
gmk::StepCtl* control(gm_handle* h);
// GM_OK or the class of a failed gate / CUDA error recorded in the control block (message in err)
int check(gm_handle* h, const char* where, std::string& err);
int failed_gate(const gm_handle* h);       // the gate word that check read
// The held sweeps (HeldCount): one more for a slot; a slot's, set; those of every slot; the sweeps that a slot's
// solve ran, of the control block that check read; and `count` solves of a slot that ran at most `used` each.
// What is captured or queued from here on holds the new counts.
void add_sweep(gm_handle* h, int slot);
void set_sweeps(gm_handle* h, int slot, int n);
std::array<int, 5> held_sweeps(const gm_handle* h);
int sweeps_run(const gm_handle* h, int slot);
void note_sweeps(gm_handle* h, int slot, int used, int count);
int64_t schur_rank(const gm_handle* h);
// surface point-pressure reconstruction (rows = quadrature points, columns = pressure cells)
struct SurfaceCsr {
  int n;
  const int64_t* ptr;
  const int64_t* col;
  const double* val;
  const double* nwx;
  const double* nwy;
};
SurfaceCsr surface(const gm_handle* h);

}  // namespace gmi

// The legacy step's launches on a stream, without synchronisation (legacy.cu); arrays of the
// state are device memory.
namespace gml {
// doubles of device scratch the calls below need
size_t scratch_doubles(const gm_legacy_state& s);
// Every call returns once *err is set (device memory; null: never).
// u*, v* (predictor_rhs_cpp), ghost velocities, the AB2 step (centred), ghost velocities, and
// the Poisson right-hand side into s.rhs, in the row scaling of the pressure system
void predict(const gm_legacy_state& s, double dt, double* scratch, const int32_t* cell_type, const double* ikappa,
             const int* err, cudaStream_t st);
// the corrector (with the ghost-cell branch's ghost velocities and boundary faces), then
// p = phi (centred) or p += phi
void correct(const gm_legacy_state& s, double dt, double* scratch, const int* err, cudaStream_t st);
// the step's record: forces (fx_p, fy_p, fx_v, fy_v), the bits of max |residual| of the solve in `slot`, and
// one more than its refinement sweeps, into out[0..5] (device)
void forces(const gm_legacy_state& s, double* scratch, double* out, const gmk::StepCtl* ctl, int slot, int nchk,
            cudaStream_t st);
}  // namespace gml
