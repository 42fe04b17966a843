// The reference's native MAC kernels of its legacy staircase path, on the GPU.
//
// solver/src/bindings.cpp:47-390 (module mac_engine) holds four OpenMP loops that the
// reference's legacy immersed/staircase step calls (solver/main.py:303-381):
//   predictor_rhs_cpp          upwind or centred momentum predictor u*, v* with staircase wall
//                              reflections, and the Poisson right-hand side rho/dt div u*;
//   corrector_cpp              u = u* - dt/rho grad phi with the exact Dirichlet outlet;
//   calculate_mac_forces_cpp   staircase pressure and shear force sums over the solid cells;
//   calculate_mac_divergence_cpp  fluid-cell divergence statistics.
// Here each is one or two grid-parallel kernels; gm_mac_ab2_rhs adds the loop's own AB2 step on
// u*, v* and its recomputed Poisson right-hand side (solver/main.py:315-339).  The per-point arithmetic is written in the
// reference's order and this file is compiled without FMA contraction, so u*, v*, rhs, u and v
// are bit-identical to the reference's compiled code; the force and divergence sums are
// reduced per block and then over blocks in a fixed order (deterministic, and equal to the
// sequential sums up to reassociation).
//
// Arrays may be host or device memory: host arrays are staged through a per-thread device
// buffer (grown on demand) on the caller's stream, and every call returns after its results
// are in the caller's arrays.
#include <cuda_runtime.h>

#include <cmath>
#include <algorithm>
#include <cstring>
#include <vector>

#include "../../include/ghostmac.h"
#include "exactdiv.cuh"
#include "internal.hpp"

namespace gmk {
void kernel_launch_adjust(long long delta);  // the library's launch counter (kernels.cu)
}
void gm_internal_set_error(const char* msg);  // defined in ghostmac.cu

namespace {
using gmk::div_by;

constexpr int LT = 256;

// Steps of the legacy loop queue behind each other without a host check between them: every kernel that
// writes the state returns once the control block's sticky error word is set (null: no control block).
__device__ __forceinline__ bool stopped(const int* err) { return err && *(const volatile int*)err != 0; }
// (row, column), in 32 bits where the index allows it
struct RowCol { int j, i; };
__device__ __forceinline__ RowCol row_col(long long t, int n) {
  if (t >> 32) return {(int)(t / n), (int)(t % n)};
  const unsigned q = (unsigned)t / (unsigned)n;
  return {(int)q, (int)((unsigned)t - q * (unsigned)n)};
}
// spacings and their reciprocals: the predictor's six divides a face, all by constants, were two thirds
// of its FP64 instructions (17 us a component at 350x213)
struct Spacing {
  double dx, dy, dx2, dy2, rho, idx, idy, idx2, idy2, irho;
};
Spacing spacing_of(double dx, double dy, double rho) {
  using gmk::reciprocal_of;
  return {dx, dy, dx * dx, dy * dy, rho, reciprocal_of(dx), reciprocal_of(dy), reciprocal_of(dx * dx), reciprocal_of(dy * dy),
          reciprocal_of(rho)};
}

#define P_(j, i) p[(size_t)(j) * nx + (i)]
#define M_(j, i) mask[(size_t)(j) * nx + (i)]
#define U_(j, i) u[(size_t)(j) * (nx + 1) + (i)]
#define V_(j, i) v[(size_t)(j) * nx + (i)]
#define US_(j, i) us[(size_t)(j) * (nx + 1) + (i)]
#define VS_(j, i) vs[(size_t)(j) * nx + (i)]
#define PHI_(j, i) phi[(size_t)(j) * nx + (i)]

// (a - 2 b + c) / h^2; 2 b is exact, so the fused form rounds as the two operations do.  (So do the factors
// 1/2 and 1/4 of the transport terms, which are taken out of the products and quotients.)
__device__ __forceinline__ double second_difference(double a, double b, double c, double hh, double ihh) {
  return div_by(__fma_rn(-2.0, b, a) + c, hh, ihh);
}
struct PredictArgs {
  const double *u, *v, *p, *inlet;  // p null: zero
  const uint8_t* mask;
  int nx, ny;
  Spacing h;
  double dt, nu;
  int slip, centered;
};
// u* on every vertical face (bindings.cpp:98-139): interior faces by the predictor, the inlet
// column from the inlet profile, the outlet column from the previous u
__device__ __forceinline__ double predict_u(const PredictArgs& a, int j, int i) {
  const double *u = a.u, *v = a.v, *p = a.p;
  const uint8_t* mask = a.mask;
  const int nx = a.nx, ny = a.ny, slip = a.slip;
  const Spacing& h = a.h;
  if (i == 0) return a.inlet[j];
  if (i == nx) return U_(j, nx - 1);
  if (M_(j, i - 1) || M_(j, i)) return 0.0;
  const double uc = U_(j, i);
  double ub, ut;
  if (j == 0) ub = slip ? uc : -uc;
  else ub = (M_(j - 1, i - 1) && M_(j - 1, i)) ? -uc : U_(j - 1, i);
  if (j == ny - 1) ut = slip ? uc : -uc;
  else ut = (M_(j + 1, i - 1) && M_(j + 1, i)) ? -uc : U_(j + 1, i);
  const double lap = second_difference(U_(j, i + 1), uc, U_(j, i - 1), h.dx2, h.idx2) + second_difference(ut, uc, ub, h.dy2, h.idy2);
  double conv;
  if (a.centered) {
    const double e = uc + U_(j, i + 1), w = uc + U_(j, i - 1);
    conv = .25 * (div_by(e * e - w * w, h.dx, h.idx) +
                  div_by((uc + ut) * (V_(j + 1, i - 1) + V_(j + 1, i)) - (uc + ub) * (V_(j, i - 1) + V_(j, i)), h.dy, h.idy));
  } else {
    const double vavg = 0.25 * (V_(j, i - 1) + V_(j, i) + V_(j + 1, i - 1) + V_(j + 1, i));
    const double dudx = div_by((uc > 0.0) ? uc - U_(j, i - 1) : U_(j, i + 1) - uc, h.dx, h.idx);
    const double dudy = div_by((vavg > 0.0) ? uc - ub : ut - uc, h.dy, h.idy);
    conv = uc * dudx + vavg * dudy;
  }
  double r = -conv + a.nu * lap;
  if (p) r = r - div_by(div_by(P_(j, i) - P_(j, i - 1), h.dx, h.idx), h.rho, h.irho);
  return uc + a.dt * r;
}

// v* on every horizontal face (bindings.cpp:142-193): walls zero
__device__ __forceinline__ double predict_v(const PredictArgs& a, int j, int i) {
  const double *u = a.u, *v = a.v, *p = a.p;
  const uint8_t* mask = a.mask;
  const int nx = a.nx, ny = a.ny;
  const Spacing& h = a.h;
  if (j == 0 || j == ny) return 0.0;
  if (M_(j - 1, i) || M_(j, i)) return 0.0;
  const double vc = V_(j, i);
  double vl, vr;
  if (i == 0) vl = -vc;
  else vl = (M_(j - 1, i - 1) && M_(j, i - 1)) ? -vc : V_(j, i - 1);
  if (i == nx - 1) vr = vc;
  else vr = (M_(j - 1, i + 1) && M_(j, i + 1)) ? -vc : V_(j, i + 1);
  const double lap = second_difference(vr, vc, vl, h.dx2, h.idx2) + second_difference(V_(j + 1, i), vc, V_(j - 1, i), h.dy2, h.idy2);
  double conv;
  if (a.centered) {
    const double n = vc + V_(j + 1, i), s = vc + V_(j - 1, i);
    conv = .25 * (div_by(n * n - s * s, h.dy, h.idy) +
                  div_by((vc + vr) * (U_(j - 1, i + 1) + U_(j, i + 1)) - (vc + vl) * (U_(j - 1, i) + U_(j, i)), h.dx, h.idx));
  } else {
    const double uavg = 0.25 * (U_(j - 1, i) + U_(j, i) + U_(j - 1, i + 1) + U_(j, i + 1));
    const double dvdx = div_by((uavg > 0.0) ? vc - vl : vr - vc, h.dx, h.idx);
    const double dvdy = div_by((vc > 0.0) ? vc - V_(j - 1, i) : V_(j + 1, i) - vc, h.dy, h.idy);
    conv = uavg * dvdx + vc * dvdy;
  }
  double r = -conv + a.nu * lap;
  if (p) r = r - div_by(div_by(P_(j, i) - P_(j - 1, i), h.dy, h.idy), h.rho, h.irho);
  return vc + a.dt * r;
}

// The predictor on every face, with the loop's AB2 step on the interior faces (solver/main.py:315-322)
// behind it when ab2 >= 0: d = (u* - u) / dt, u* += dt alpha (d - d_prev) when a previous step exists
// (ab2 = 1), d_prev = d.  The FP64 pipe is the bound; predictor and AB2 in three kernels took 40 us at
// 350x213, 17 as one with divides by known divisors.
__global__ void k_predict(PredictArgs a, double* __restrict__ us, double* __restrict__ vs, int ab2, double idt,
                          double dt_alpha, double* __restrict__ pdu, double* __restrict__ pdv, const int* err) {
  if (stopped(err)) return;
  const int nx = a.nx, ny = a.ny;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nu_ = (long long)ny * (nx + 1);
  if (t >= nu_ + (long long)(ny + 1) * nx) return;
  const bool isu = t < nu_;
  const long long f = isu ? t : t - nu_;
  const auto [j, i] = row_col(f, isu ? nx + 1 : nx);
  double s = isu ? predict_u(a, j, i) : predict_v(a, j, i);
  if (ab2 >= 0 && (isu ? i >= 1 && i < nx : j >= 1 && j < ny)) {
    const double d = div_by(s - (isu ? a.u : a.v)[f], a.dt, idt);
    double* prev = isu ? pdu : pdv;
    if (ab2) s = s + dt_alpha * (d - prev[f]);
    prev[f] = d;
  }
  (isu ? us : vs)[f] = s;
}

// Poisson right-hand side rho/dt div u* on the fluid cells (bindings.cpp:201-215)
__global__ void k_poisson_rhs(const double* __restrict__ us, const double* __restrict__ vs,
                              const uint8_t* __restrict__ mask, double* __restrict__ rhs, int nx, int ny,
                              Spacing h, double inv_dt) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)ny * nx) return;
  const int j = (int)(t / nx), i = (int)(t - (long long)j * nx);
  if (M_(j, i)) { rhs[t] = 0.0; return; }
  const double div = div_by(US_(j, i + 1) - US_(j, i), h.dx, h.idx) + div_by(VS_(j + 1, i) - VS_(j, i), h.dy, h.idy);
  rhs[t] = inv_dt * div;
}

// The same AB2 step by itself (the ghost-cell branch sets its ghost faces in between): d = (u* - u) / dt,
// u* += dt alpha (d - d_prev) when a previous step exists, d_prev = d
__global__ void k_ab2(const double* __restrict__ u, const double* __restrict__ v, double* __restrict__ us,
                      double* __restrict__ vs, double* __restrict__ pdu, double* __restrict__ pdv, int nx, int ny,
                      double dt, double dt_alpha, int has_prev, const int* err) {
  if (stopped(err)) return;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nu_ = (long long)ny * (nx + 1), nv_ = (long long)(ny + 1) * nx;
  if (t < nu_) {
    const int i = (int)(t % (nx + 1));
    if (i < 1 || i > nx - 1) return;
    const double d = (us[t] - u[t]) / dt;
    if (has_prev) us[t] = us[t] + dt_alpha * (d - pdu[t]);
    pdu[t] = d;
  } else if (t < nu_ + nv_) {
    const long long f = t - nu_;
    const int j = (int)(f / nx);
    if (j < 1 || j > ny - 1) return;
    const double d = (vs[f] - v[f]) / dt;
    if (has_prev) vs[f] = vs[f] + dt_alpha * (d - pdv[f]);
    pdv[f] = d;
  }
}

// the recomputed Poisson right-hand side of the legacy loop (solver/main.py:337-339):
// rho/dt ((u*_e - u*_w)/dx + (v*_n - v*_s)/dy), zero on masked cells; with cell_type in the row
// scaling of the pressure system (1 / kappa on cut cells, zero on covered ones)
__global__ void k_legacy_rhs(const double* __restrict__ us, const double* __restrict__ vs,
                             const uint8_t* __restrict__ mask, double* __restrict__ rhs, int nx, int ny, Spacing h,
                             double rho_dt, const int32_t* __restrict__ cell_type, const double* __restrict__ ikappa,
                             const int* err) {
  if (stopped(err)) return;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)ny * nx) return;
  const auto [j, i] = row_col(t, nx);
  if (M_(j, i) || (cell_type && cell_type[t] == -1)) { rhs[t] = 0.0; return; }
  const double r = rho_dt * (div_by(US_(j, i + 1) - US_(j, i), h.dx, h.idx) + div_by(VS_(j + 1, i) - VS_(j, i), h.dy, h.idy));
  rhs[t] = cell_type ? r * ikappa[t] : r;
}

// ---- the legacy loop's ghost-cell branch (solver/ghost_cell.py:32-234, solver/main.py:347-370) --
// Image-point ghost velocities g = wall - gamma (ip - wall), ip the bilinear value at the image
// point.  The reference sets the ghost faces one after another, so a face may read a ghost face
// set earlier in the same pass (its new value) or a later one (its old value): the host orders
// the faces into levels (a face is one level above every earlier ghost face it reads), the old
// values are saved first, and each level is one launch.
__global__ void k_ghost_save(const double* __restrict__ f, long long nf, const long long* __restrict__ target,
                             long long n, double* __restrict__ snap, const int* err) {
  if (stopped(err)) return;
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < n) {
    const long long t = target[g];
    snap[g] = (t >= 0 && t < nf) ? f[t] : 0.0;
  }
}
// one level of ghost faces; entries whose indexes fall outside the field or the table are skipped
__global__ void k_ghost_level(double* __restrict__ f, long long nf, const long long* __restrict__ target,
                              const long long* __restrict__ src, const int* __restrict__ snap_of,
                              const double* __restrict__ w, const double* __restrict__ gamma,
                              const int* __restrict__ level, long long n, int lvl, const double* __restrict__ snap,
                              double wall, const int* err) {
  if (stopped(err)) return;
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n || level[g] != lvl) return;
  const long long t = target[g];
  if (t < 0 || t >= nf) return;
  double v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int sidx = snap_of[4 * g + q];
    const long long c = src[4 * g + q];
    if (sidx >= n || c < 0 || c >= nf) return;
    v[q] = sidx >= 0 ? snap[sidx] : f[c];
  }
  // the reference's order: w00 f00 + w10 f10 + w01 f01 + w11 f11, then the reflection
  const double ip = w[4 * g] * v[0] + w[4 * g + 1] * v[1] + w[4 * g + 2] * v[2] + w[4 * g + 3] * v[3];
  f[t] = wall - gamma[g] * (ip - wall);
}

// the ghost branch's corrector (solver/main.py:347-366): u = u* on interior faces, minus
// dt/rho grad phi on faces between two fluid cells, zero between two masked cells, the inlet
// and the Dirichlet outlet; v likewise with zero wall rows
__global__ void k_ghost_correct(double* __restrict__ u, double* __restrict__ v, const double* __restrict__ us,
                                const double* __restrict__ vs, const double* __restrict__ phi,
                                const uint8_t* __restrict__ mask, const double* __restrict__ inlet, int nx, int ny,
                                double dx, double dy, double dt_over_rho, const int* err) {
  if (stopped(err)) return;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nu_ = (long long)ny * (nx + 1);
  if (t < nu_) {
    const int j = (int)(t / (nx + 1)), i = (int)(t - (long long)j * (nx + 1));
    if (i == 0) U_(j, 0) = inlet[j];
    else if (i == nx) U_(j, nx) = US_(j, nx) + dt_over_rho * 2.0 * PHI_(j, nx - 1) / dx;
    else {
      const bool l = M_(j, i - 1), r = M_(j, i);
      double val = US_(j, i);
      if (!l && !r) val -= dt_over_rho * (PHI_(j, i) - PHI_(j, i - 1)) / dx;
      else if (l && r) val = 0.0;
      U_(j, i) = val;
    }
  } else if (t < nu_ + (long long)(ny + 1) * nx) {
    const long long f = t - nu_;
    const int j = (int)(f / nx), i = (int)(f - (long long)j * nx);
    if (j == 0 || j == ny) { V_(j, i) = 0.0; return; }
    const bool b = M_(j - 1, i), a = M_(j, i);
    double val = VS_(j, i);
    if (!a && !b) val -= dt_over_rho * (PHI_(j, i) - PHI_(j - 1, i)) / dy;
    else if (a && b) val = 0.0;
    V_(j, i) = val;
  }
}
// faces between a fluid and a masked cell keep u* (solver/main.py:368-370); the pressure update
__global__ void k_ghost_boundary(double* __restrict__ u, double* __restrict__ v, const double* __restrict__ us,
                                 const double* __restrict__ vs, const uint8_t* __restrict__ mask, int nx, int ny, double* __restrict__ p,
                                 const double* __restrict__ phi, int add, const int* err) {
  if (stopped(err)) return;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nu_ = (long long)ny * (nx + 1);
  if (p && t < (long long)ny * nx) p[t] = add ? p[t] + phi[t] : phi[t];
  if (t < nu_) {
    const int j = (int)(t / (nx + 1)), i = (int)(t - (long long)j * (nx + 1));
    if (i >= 1 && i <= nx - 1 && M_(j, i - 1) != M_(j, i)) U_(j, i) = US_(j, i);
  } else if (t < nu_ + (long long)(ny + 1) * nx) {
    const long long f = t - nu_;
    const int j = (int)(f / nx), i = (int)(f - (long long)j * nx);
    if (j >= 1 && j <= ny - 1 && M_(j - 1, i) != M_(j, i)) V_(j, i) = VS_(j, i);
  }
}

// A step's record behind its four forces: max |residual| of the pressure solve's last check (out[4], its bits)
// and, as a mark that the step is complete, one more than the refinement sweeps that the solve ran (out[5]).
struct StepRecord {
  const gmk::StepCtl* ctl;  // null: no record
  int slot, nchk;
  __device__ const int* err() const { return ctl ? &ctl->err : nullptr; }
  __device__ void close(double* out) const {
    if (!ctl) return;
    const gmk::SolveCtl* sc = &ctl->solve[slot];
    const int k = gmk::last_check(sc, nchk);
    out[4] = gmk::bits2d(sc->rmax[k]);
    out[5] = 1.0 + k;
  }
};

// bilinear value of a staggered field at (y, x): the linear RegularGridInterpolator of the
// reference (solver/ghost_cell.py:199-201), zero outside the grid
__device__ double grid_linear(const double* __restrict__ f, int nxf, int nyf, double x0, double y0, double hx,
                              double hy, double y, double x) {
  const double gx = (x - x0) / hx, gy = (y - y0) / hy;
  if (!(gx >= 0.0 && gx <= nxf - 1 && gy >= 0.0 && gy <= nyf - 1)) return 0.0;
  int i = (int)floor(gx), j = (int)floor(gy);
  if (i > nxf - 2) i = nxf - 2;
  if (j > nyf - 2) j = nyf - 2;
  const double tx = (x - (x0 + i * hx)) / hx, ty = (y - (y0 + j * hy)) / hy;
  const double* r0 = f + (size_t)j * nxf;
  const double* r1 = r0 + nxf;
  return (r0[i] * (1.0 - tx) + r0[i + 1] * tx) * (1.0 - ty) + (r1[i] * (1.0 - tx) + r1[i + 1] * tx) * ty;
}

// surface forces on the true circle (extract_true_surface_forces, solver/ghost_cell.py:186-234):
// pressure and probed central-difference velocity gradients at n points; one block, sums in a
// fixed order; out = fx_p, fy_p, fx_v, fy_v
__global__ void k_ghost_forces(const double* __restrict__ u, const double* __restrict__ v, const double* __restrict__ p,
                               int nx, int ny, double dx, double dy, double xc, double yc, double radius, int n,
                               double mu, double* __restrict__ out, StepRecord rec) {
  if (stopped(rec.err())) return;
  __shared__ double sh[4][256];
  double ax = 0.0, ay = 0.0, bx = 0.0, by = 0.0;
  const double eps = 1e-4 * dx;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const double th = k * (2 * M_PI / n);  // np.linspace(0, 2 pi, n, endpoint=False)
    const double c = cos(th), s = sin(th);
    const double x = xc + radius * c, y = yc + radius * s;
    const double pk = grid_linear(p, nx, ny, 0.5 * dx, 0.5 * dy, dx, dy, y, x);
    auto U = [&](double yy, double xx) { return grid_linear(u, nx + 1, ny, 0.0, 0.5 * dy, dx, dy, yy, xx); };
    auto V = [&](double yy, double xx) { return grid_linear(v, nx, ny + 1, 0.5 * dx, 0.0, dx, dy, yy, xx); };
    const double dudx = (U(y, x + eps) - U(y, x - eps)) / (2.0 * eps);
    const double dudy = (U(y + eps, x) - U(y - eps, x)) / (2.0 * eps);
    const double dvdx = (V(y, x + eps) - V(y, x - eps)) / (2.0 * eps);
    const double dvdy = (V(y + eps, x) - V(y - eps, x)) / (2.0 * eps);
    const double txx = 2.0 * mu * dudx, tyy = 2.0 * mu * dvdy, txy = mu * (dudy + dvdx);
    ax += pk * c;
    ay += pk * s;
    bx += txx * c + txy * s;
    by += txy * c + tyy * s;
  }
  sh[0][threadIdx.x] = ax; sh[1][threadIdx.x] = ay; sh[2][threadIdx.x] = bx; sh[3][threadIdx.x] = by;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st)
      for (int q = 0; q < 4; ++q) sh[q][threadIdx.x] += sh[q][threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double ds = radius * (2 * M_PI / n);
    out[0] = -sh[0][0] * ds;
    out[1] = -sh[1][0] * ds;
    out[2] = sh[2][0] * ds;
    out[3] = sh[3][0] * ds;
    rec.close(out);
  }
}

// u = u* - dt/rho d phi/dx, v = v* - dt/rho d phi/dy (bindings.cpp:248-281); with p also the loop's pressure
// update, p = phi (add = 0) or p += phi
__global__ void k_correct(double* __restrict__ u, double* __restrict__ v, const double* __restrict__ us,
                          const double* __restrict__ vs, const double* __restrict__ phi,
                          const uint8_t* __restrict__ mask, const double* __restrict__ inlet, int nx, int ny,
                          Spacing h, double dt_over_rho, double* __restrict__ p, int add, const int* err) {
  if (stopped(err)) return;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nu_ = (long long)ny * (nx + 1);
  if (p && t < (long long)ny * nx) p[t] = add ? p[t] + phi[t] : phi[t];
  if (t < nu_) {
    const auto [j, i] = row_col(t, nx + 1);
    if (i == 0) U_(j, 0) = inlet[j];
    else if (i == nx) U_(j, nx) = US_(j, nx) + div_by(dt_over_rho * 2.0 * PHI_(j, nx - 1), h.dx, h.idx);
    else if (M_(j, i - 1) || M_(j, i)) U_(j, i) = 0.0;
    else U_(j, i) = US_(j, i) - div_by(dt_over_rho * (PHI_(j, i) - PHI_(j, i - 1)), h.dx, h.idx);
    return;
  }
  const long long r = t - nu_;
  if (r >= (long long)(ny + 1) * nx) return;
  const auto [j, i] = row_col(r, nx);
  if (j == 0 || j == ny) V_(j, i) = 0.0;
  else if (M_(j - 1, i) || M_(j, i)) V_(j, i) = 0.0;
  else V_(j, i) = VS_(j, i) - div_by(dt_over_rho * (PHI_(j, i) - PHI_(j - 1, i)), h.dy, h.idy);
}

template <int NF>
__device__ void block_sum(double (&val)[NF], double* __restrict__ out /* NF per block */) {
  __shared__ double sm[NF][LT];
#pragma unroll
  for (int f = 0; f < NF; ++f) sm[f][threadIdx.x] = val[f];
  __syncthreads();
  for (int s = LT / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s)
#pragma unroll
      for (int f = 0; f < NF; ++f) sm[f][threadIdx.x] += sm[f][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0)
#pragma unroll
    for (int f = 0; f < NF; ++f) out[(size_t)blockIdx.x * NF + f] = sm[f][0];
}

// staircase traction of every solid cell's fluid-facing sides (bindings.cpp:310-338)
__global__ void k_forces_part(const double* __restrict__ u, const double* __restrict__ v,
                              const double* __restrict__ p, const uint8_t* __restrict__ mask, int nx, int ny,
                              double dx, double dy, double mu, double* __restrict__ part) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double f[4] = {0.0, 0.0, 0.0, 0.0};  // fx_p, fy_p, fx_v, fy_v
  if (t < (long long)ny * nx) {
    const int j = (int)(t / nx), i = (int)(t - (long long)j * nx);
    if (M_(j, i)) {
      if (i > 0 && !M_(j, i - 1)) {
        f[0] += P_(j, i - 1) * dy;
        const double vf = 0.5 * (V_(j, i - 1) + V_(j + 1, i - 1));
        f[3] += mu * (vf / (0.5 * dx)) * dy;
      }
      if (i < nx - 1 && !M_(j, i + 1)) {
        f[0] -= P_(j, i + 1) * dy;
        const double vf = 0.5 * (V_(j, i + 1) + V_(j + 1, i + 1));
        f[3] += mu * (vf / (0.5 * dx)) * dy;
      }
      if (j > 0 && !M_(j - 1, i)) {
        f[1] += P_(j - 1, i) * dx;
        const double uf = 0.5 * (U_(j - 1, i) + U_(j - 1, i + 1));
        f[2] += mu * (uf / (0.5 * dy)) * dx;
      }
      if (j < ny - 1 && !M_(j + 1, i)) {
        f[1] -= P_(j + 1, i) * dx;
        const double uf = 0.5 * (U_(j + 1, i) + U_(j + 1, i + 1));
        f[2] += mu * (uf / (0.5 * dy)) * dx;
      }
    }
  }
  block_sum<4>(f, part);
}

// divergence of every fluid cell: max |div|, sum div^2, count, core sum, core count
// (bindings.cpp:343-390)
__global__ void k_div_part(const double* __restrict__ u, const double* __restrict__ v,
                           const uint8_t* __restrict__ mask, int nx, int ny, double dx, double dy,
                           double* __restrict__ part) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double s[4] = {0.0, 0.0, 0.0, 0.0};  // sum div^2, count, core sum, core count
  double mx = 0.0;
  if (t < (long long)ny * nx) {
    const int j = (int)(t / nx), i = (int)(t - (long long)j * nx);
    if (!M_(j, i)) {
      const double d = (U_(j, i + 1) - U_(j, i)) / dx + (V_(j + 1, i) - V_(j, i)) / dy;
      mx = fabs(d);
      s[0] = d * d;
      s[1] = 1.0;
      const bool core = !((i > 0 && M_(j, i - 1)) || (i < nx - 1 && M_(j, i + 1)) || (j > 0 && M_(j - 1, i)) ||
                          (j < ny - 1 && M_(j + 1, i)));
      if (core) {
        s[2] = d * d;
        s[3] = 1.0;
      }
    }
  }
  __shared__ double smx[LT];
  smx[threadIdx.x] = mx;
  __syncthreads();
  for (int k = LT / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) smx[threadIdx.x] = fmax(smx[threadIdx.x], smx[threadIdx.x + k]);
    __syncthreads();
  }
  double* out = part + (size_t)gridDim.x * 4;  // maxima after the sums
  if (threadIdx.x == 0) out[blockIdx.x] = smx[0];
  block_sum<4>(s, part);
}

// per-field sums of the block partials (one block of LT threads: thread t adds the partials of
// blocks t, t + LT, ... in order, then a tree in a fixed order; the same sums every run); the
// maximum of the divergence after them when nmax is set
__global__ void k_fold(const double* __restrict__ part, int nblocks, int nmax, double* __restrict__ out, StepRecord rec) {
  if (stopped(rec.err())) return;
  constexpr int NF = 4;
  __shared__ double sh[NF + 1][LT];
  double a[NF + 1] = {0.0, 0.0, 0.0, 0.0, 0.0};
  for (int b = threadIdx.x; b < nblocks; b += LT) {
#pragma unroll
    for (int f = 0; f < NF; ++f) a[f] = a[f] + part[(size_t)b * NF + f];
    if (nmax) a[NF] = fmax(a[NF], part[(size_t)nblocks * NF + b]);
  }
#pragma unroll
  for (int f = 0; f <= NF; ++f) sh[f][threadIdx.x] = a[f];
  __syncthreads();
  for (int k = LT / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) {
#pragma unroll
      for (int f = 0; f < NF; ++f) sh[f][threadIdx.x] = sh[f][threadIdx.x] + sh[f][threadIdx.x + k];
      sh[NF][threadIdx.x] = fmax(sh[NF][threadIdx.x], sh[NF][threadIdx.x + k]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    for (int f = 0; f < NF + (nmax ? 1 : 0); ++f) out[f] = sh[f][0];
    rec.close(out);
  }
}


int fail(int code, const char* msg) {
  gm_internal_set_error(msg);
  return code;
}

bool is_device(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  return (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) && a.device == dev;
}

// Device views of the call's arrays: device arrays pass through; host arrays get a slice of a
// per-thread device buffer, copied in (inputs) before and out (outputs) after the kernels.
struct Staging {
  struct Arena {
    void* p = nullptr;
    size_t cap = 0;
    int dev = -1;
  };
  static Arena& arena() {
    static thread_local Arena a;
    return a;
  }
  struct Item {
    const void* host;
    void* dev;
    size_t bytes;
    bool in, out;
  };
  std::vector<Item> items;
  size_t total = 0;
  cudaStream_t st;
  explicit Staging(cudaStream_t s) : st(s) {}
  // registers an array; returns its index
  int add(const void* p, size_t bytes, bool in, bool out) {
    if (is_device(p)) {
      items.push_back({p, const_cast<void*>(p), bytes, false, false});
    } else {
      items.push_back({p, nullptr, bytes, in, out});
      total += (bytes + 255) & ~(size_t)255;
    }
    return (int)items.size() - 1;
  }
  cudaError_t begin(size_t extra_bytes, double** extra) {
    Arena& a = arena();
    int dev = 0;
    cudaGetDevice(&dev);
    const size_t need = total + ((extra_bytes + 255) & ~(size_t)255);
    if (a.dev != dev || a.cap < need) {
      if (a.p && a.dev == dev) cudaFree(a.p);
      a.p = nullptr;
      a.cap = 0;
      cudaError_t e = cudaMalloc(&a.p, need);
      if (e != cudaSuccess) return e;
      a.cap = need;
      a.dev = dev;
    }
    size_t off = 0;
    char* base = static_cast<char*>(a.p);
    for (auto& it : items) {
      if (it.dev) continue;
      it.dev = base + off;
      off += (it.bytes + 255) & ~(size_t)255;
      if (it.in) {
        cudaError_t e = cudaMemcpyAsync(it.dev, it.host, it.bytes, cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return e;
      }
    }
    *extra = reinterpret_cast<double*>(base + off);
    return cudaSuccess;
  }
  cudaError_t finish() {
    for (auto& it : items)
      if (it.out && it.host != it.dev) {
        cudaError_t e = cudaMemcpyAsync(const_cast<void*>(it.host), it.dev, it.bytes, cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) return e;
      }
    return cudaStreamSynchronize(st);
  }
  template <typename T>
  T* dev(int k) const { return static_cast<T*>(items[k].dev); }
};

int check_grid(int nx, int ny, double dx, double dy) {
  if (nx < 2 || ny < 2) return fail(GM_EVALUE, "mask must be a 2D grid with at least 2 cells per direction");
  if (!(std::isfinite(dx) && dx > 0 && std::isfinite(dy) && dy > 0))
    return fail(GM_EVALUE, "dx and dy must be finite and positive");
  return GM_OK;
}
int check_step(double dt, double rho) {
  if (!(std::isfinite(dt) && dt > 0 && std::isfinite(rho) && rho > 0))
    return fail(GM_EVALUE, "dt and rho must be finite and positive");
  return GM_OK;
}
int cuda_fail(cudaError_t e) {
  cudaGetLastError();
  return fail(GM_ECUDA, cudaGetErrorString(e));
}
unsigned blocks(long long n) { return (unsigned)((n + LT - 1) / LT); }

void ghost_pass(const gm_legacy_state& s, int k, double* field, double* snap, const int* err, cudaStream_t st) {
  const long long n = s.n_ghost[k];
  if (n <= 0) return;
  const long long nf = k == 0 ? (long long)s.ny * (s.nx + 1) : (long long)(s.ny + 1) * s.nx;
  const long long* tg = reinterpret_cast<const long long*>(s.target[k]);
  k_ghost_save<<<blocks(n), LT, 0, st>>>(field, nf, tg, n, snap, err);
  for (int l = 0; l < s.n_levels[k]; ++l)
    k_ghost_level<<<blocks(n), LT, 0, st>>>(field, nf, tg, reinterpret_cast<const long long*>(s.src[k]), s.snap_of[k],
                                            s.weights[k], s.gamma[k], s.level[k], n, l, snap, 0.0, err);
  gmk::kernel_launch_adjust(1 + s.n_levels[k]);
}

}  // namespace

namespace gml {

size_t scratch_doubles(const gm_legacy_state& s) {
  const long long nP = (long long)s.ny * s.nx;
  const long long ng = std::max<long long>(s.ghost ? std::max(s.n_ghost[0], s.n_ghost[1]) : 0, 1);
  return (size_t)(ng + (long long)blocks(nP) * 4 + 16);
}

void predict(const gm_legacy_state& s, double dt, double* scratch, const int32_t* cell_type, const double* ikappa,
             const int* err, cudaStream_t st) {
  const int nx = s.nx, ny = s.ny;
  const long long nU = (long long)ny * (nx + 1), nV = (long long)(ny + 1) * nx, nP = (long long)ny * nx;
  const PredictArgs a{s.u, s.v, s.centered ? nullptr : s.p, s.inlet, s.mask, nx, ny, spacing_of(s.dx, s.dy, s.rho), dt, s.nu,
                      s.slip_walls ? 1 : 0, s.centered ? 1 : 0};
  const bool hp = s.has_prev != 0;
  const double dta = hp ? dt * (dt / (2 * s.prev_dt)) : 0.0;
  k_predict<<<blocks(nU + nV), LT, 0, st>>>(a, s.u_star, s.v_star, s.ghost || !s.centered ? -1 : hp ? 1 : 0, gmk::reciprocal_of(dt), dta,
                                            s.prev_du, s.prev_dv, err);
  gmk::kernel_launch_adjust(1);
  if (s.ghost) {
    ghost_pass(s, 0, s.u_star, scratch, err, st);
    ghost_pass(s, 1, s.v_star, scratch, err, st);
    if (s.centered) {
      k_ab2<<<blocks(nU + nV), LT, 0, st>>>(s.u, s.v, s.u_star, s.v_star, s.prev_du, s.prev_dv, nx, ny, dt, dta, hp ? 1 : 0, err);
      gmk::kernel_launch_adjust(1);
      ghost_pass(s, 0, s.u_star, scratch, err, st);
      ghost_pass(s, 1, s.v_star, scratch, err, st);
    }
  }
  k_legacy_rhs<<<blocks(nP), LT, 0, st>>>(s.u_star, s.v_star, s.mask, s.rhs, nx, ny, a.h, s.rho / dt, cell_type, ikappa, err);
  gmk::kernel_launch_adjust(1);
}

void correct(const gm_legacy_state& s, double dt, double* scratch, const int* err, cudaStream_t st) {
  const int nx = s.nx, ny = s.ny;
  const long long n = (long long)ny * (nx + 1) + (long long)(ny + 1) * nx;
  if (s.ghost) {
    k_ghost_correct<<<blocks(n), LT, 0, st>>>(s.u, s.v, s.u_star, s.v_star, s.phi, s.mask, s.inlet, nx, ny, s.dx,
                                              s.dy, dt / s.rho, err);
    ghost_pass(s, 0, s.u, scratch, err, st);
    ghost_pass(s, 1, s.v, scratch, err, st);
    k_ghost_boundary<<<blocks(n), LT, 0, st>>>(s.u, s.v, s.u_star, s.v_star, s.mask, nx, ny, s.p, s.phi, s.centered ? 0 : 1, err);
    gmk::kernel_launch_adjust(2);
  } else {
    k_correct<<<blocks(n), LT, 0, st>>>(s.u, s.v, s.u_star, s.v_star, s.phi, s.mask, s.inlet, nx, ny,
                                        spacing_of(s.dx, s.dy, s.rho), dt / s.rho, s.p, s.centered ? 0 : 1, err);
    gmk::kernel_launch_adjust(1);
  }
}

void forces(const gm_legacy_state& s, double* scratch, double* out, const gmk::StepCtl* ctl, int slot, int nchk,
            cudaStream_t st) {
  const int nx = s.nx, ny = s.ny;
  const double mu = s.nu * s.rho;
  const StepRecord rec{ctl, slot, nchk};
  if (s.ghost) {
    k_ghost_forces<<<1, 256, 0, st>>>(s.u, s.v, s.p, nx, ny, s.dx, s.dy, s.xc, s.yc, s.radius, s.n_theta, mu, out, rec);
    gmk::kernel_launch_adjust(1);
    return;
  }
  const unsigned nb = blocks((long long)ny * nx);
  double* part = scratch + 1;
  k_forces_part<<<nb, LT, 0, st>>>(s.u, s.v, s.p, s.mask, nx, ny, s.dx, s.dy, mu, part);
  k_fold<<<1, LT, 0, st>>>(part, (int)nb, 0, out, rec);
  gmk::kernel_launch_adjust(2);
}

}  // namespace gml

extern "C" {

int gm_mac_predictor_rhs(const double* u, const double* v, double* u_star, double* v_star, double* rhs,
                         const double* p, const uint8_t* mask, const double* inlet, int32_t nx, int32_t ny, double dx,
                         double dy, double dt, double nu, double rho, int32_t slip_walls, int32_t centered,
                         void* stream) {
  if (!u || !v || !u_star || !v_star || !rhs || !p || !mask || !inlet) return fail(GM_EVALUE, "null argument");
  if (int rc = check_grid(nx, ny, dx, dy)) return rc;
  if (int rc = check_step(dt, rho)) return rc;
  if (!(std::isfinite(nu) && nu >= 0)) return fail(GM_EVALUE, "nu must be finite and nonnegative");
  const size_t nU = (size_t)ny * (nx + 1), nV = (size_t)(ny + 1) * nx, nP = (size_t)ny * nx;
  Staging sg(static_cast<cudaStream_t>(stream));
  const int iu = sg.add(u, nU * 8, true, false), iv = sg.add(v, nV * 8, true, false);
  const int ius = sg.add(u_star, nU * 8, false, true), ivs = sg.add(v_star, nV * 8, false, true);
  const int ir = sg.add(rhs, nP * 8, false, true), ip = sg.add(p, nP * 8, true, false);
  const int im = sg.add(mask, nP, true, false), ii = sg.add(inlet, (size_t)ny * 8, true, false);
  double* extra = nullptr;
  if (cudaError_t e = sg.begin(0, &extra)) return cuda_fail(e);
  cudaStream_t st = sg.st;
  const Spacing h = spacing_of(dx, dy, rho);
  const PredictArgs a{sg.dev<double>(iu), sg.dev<double>(iv), sg.dev<double>(ip), sg.dev<double>(ii), sg.dev<uint8_t>(im), nx, ny, h,
                      dt, nu, slip_walls ? 1 : 0, centered ? 1 : 0};
  k_predict<<<blocks((long long)(nU + nV)), LT, 0, st>>>(a, sg.dev<double>(ius), sg.dev<double>(ivs), -1, 0.0, 0.0, nullptr, nullptr,
                                                       nullptr);
  k_poisson_rhs<<<blocks((long long)nP), LT, 0, st>>>(sg.dev<double>(ius), sg.dev<double>(ivs), sg.dev<uint8_t>(im),
                                                      sg.dev<double>(ir), nx, ny, h, rho / dt);
  gmk::kernel_launch_adjust(2);
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(e);
  if (cudaError_t e = sg.finish()) return cuda_fail(e);
  return GM_OK;
}

int gm_mac_corrector(double* u, double* v, const double* u_star, const double* v_star, const double* phi,
                     const uint8_t* mask, const double* inlet, int32_t nx, int32_t ny, double dx, double dy, double dt,
                     double rho, int32_t slip_walls, void* stream) {
  (void)slip_walls;  // accepted for the reference's signature; the walls are no-slip v = 0 either way
  if (!u || !v || !u_star || !v_star || !phi || !mask || !inlet) return fail(GM_EVALUE, "null argument");
  if (int rc = check_grid(nx, ny, dx, dy)) return rc;
  if (int rc = check_step(dt, rho)) return rc;
  const size_t nU = (size_t)ny * (nx + 1), nV = (size_t)(ny + 1) * nx, nP = (size_t)ny * nx;
  Staging sg(static_cast<cudaStream_t>(stream));
  const int iu = sg.add(u, nU * 8, false, true), iv = sg.add(v, nV * 8, false, true);
  const int ius = sg.add(u_star, nU * 8, true, false), ivs = sg.add(v_star, nV * 8, true, false);
  const int iph = sg.add(phi, nP * 8, true, false), im = sg.add(mask, nP, true, false);
  const int ii = sg.add(inlet, (size_t)ny * 8, true, false);
  double* extra = nullptr;
  if (cudaError_t e = sg.begin(0, &extra)) return cuda_fail(e);
  k_correct<<<blocks((long long)(nU + nV)), LT, 0, sg.st>>>(sg.dev<double>(iu), sg.dev<double>(iv),
                                                              sg.dev<double>(ius), sg.dev<double>(ivs),
                                                              sg.dev<double>(iph), sg.dev<uint8_t>(im),
                                                              sg.dev<double>(ii), nx, ny, spacing_of(dx, dy, rho), dt / rho, nullptr, 0, nullptr);
  gmk::kernel_launch_adjust(1);
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(e);
  if (cudaError_t e = sg.finish()) return cuda_fail(e);
  return GM_OK;
}

int gm_mac_ab2_rhs(const double* u, const double* v, double* u_star, double* v_star, double* prev_du,
                   double* prev_dv, double* rhs, const uint8_t* mask, int32_t nx, int32_t ny, double dx, double dy,
                   double dt, double rho, double alpha, int32_t has_prev, int32_t what, void* stream) {
  if (!u || !v || !u_star || !v_star || !prev_du || !prev_dv || !rhs || !mask) return fail(GM_EVALUE, "null argument");
  if (int rc = check_grid(nx, ny, dx, dy)) return rc;
  if (int rc = check_step(dt, rho)) return rc;
  if (has_prev && !std::isfinite(alpha)) return fail(GM_EVALUE, "alpha must be finite");
  const size_t nU = (size_t)ny * (nx + 1), nV = (size_t)(ny + 1) * nx, nP = (size_t)ny * nx;
  Staging sg(static_cast<cudaStream_t>(stream));
  const int iu = sg.add(u, nU * 8, true, false), iv = sg.add(v, nV * 8, true, false);
  const int ius = sg.add(u_star, nU * 8, true, true), ivs = sg.add(v_star, nV * 8, true, true);
  const int idu = sg.add(prev_du, nU * 8, true, true), idv = sg.add(prev_dv, nV * 8, true, true);
  const int ir = sg.add(rhs, nP * 8, true, true), im = sg.add(mask, nP, true, false);
  double* extra = nullptr;
  if (cudaError_t e = sg.begin(0, &extra)) return cuda_fail(e);
  cudaStream_t st = sg.st;
  if (what & 1) {
    k_ab2<<<blocks((long long)(nU + nV)), LT, 0, st>>>(sg.dev<double>(iu), sg.dev<double>(iv), sg.dev<double>(ius),
                                                       sg.dev<double>(ivs), sg.dev<double>(idu), sg.dev<double>(idv),
                                                       nx, ny, dt, dt * alpha, has_prev ? 1 : 0, nullptr);
    gmk::kernel_launch_adjust(1);
  }
  if (what & 2) {
    k_legacy_rhs<<<blocks((long long)nP), LT, 0, st>>>(sg.dev<double>(ius), sg.dev<double>(ivs),
                                                       sg.dev<uint8_t>(im), sg.dev<double>(ir), nx, ny, spacing_of(dx, dy, rho),
                                                       rho / dt, nullptr, nullptr, nullptr);
    gmk::kernel_launch_adjust(1);
  }
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(e);
  if (cudaError_t e = sg.finish()) return cuda_fail(e);
  return GM_OK;
}

int gm_mac_ghost_apply(double* field, int64_t field_size, int64_t n_ghost, const int64_t* target, const int64_t* src,
                       const int32_t* snap_of, const double* weights, const double* gamma, const int32_t* level,
                       int32_t n_levels, double wall, void* stream) {
  if (n_ghost < 0 || field_size <= 0 || n_levels < 0) return fail(GM_EVALUE, "invalid ghost table sizes");
  if (n_ghost == 0) return GM_OK;
  if (!field || !target || !src || !snap_of || !weights || !gamma || !level) return fail(GM_EVALUE, "null argument");
  if (!std::isfinite(wall)) return fail(GM_EVALUE, "the wall velocity must be finite");
  const size_t ng = (size_t)n_ghost;
  Staging sg(static_cast<cudaStream_t>(stream));
  const int iff = sg.add(field, (size_t)field_size * 8, true, true);
  const int it = sg.add(target, ng * 8, true, false), is = sg.add(src, 4 * ng * 8, true, false);
  const int io = sg.add(snap_of, 4 * ng * 4, true, false), iw = sg.add(weights, 4 * ng * 8, true, false);
  const int ig = sg.add(gamma, ng * 8, true, false), il = sg.add(level, ng * 4, true, false);
  double* snap = nullptr;
  if (cudaError_t e = sg.begin(ng * 8, &snap)) return cuda_fail(e);
  const unsigned nb = blocks((long long)n_ghost);
  const long long* tg = sg.dev<const long long>(it);
  k_ghost_save<<<nb, LT, 0, sg.st>>>(sg.dev<double>(iff), field_size, tg, n_ghost, snap, nullptr);
  for (int l = 0; l < n_levels; ++l)
    k_ghost_level<<<nb, LT, 0, sg.st>>>(sg.dev<double>(iff), field_size, tg, sg.dev<const long long>(is),
                                        sg.dev<const int>(io), sg.dev<const double>(iw), sg.dev<const double>(ig),
                                        sg.dev<const int>(il), n_ghost, l, snap, wall, nullptr);
  gmk::kernel_launch_adjust(1 + n_levels);
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(e);
  if (cudaError_t e = sg.finish()) return cuda_fail(e);
  return GM_OK;
}

int gm_mac_ghost_correct(double* u, double* v, const double* u_star, const double* v_star, const double* phi,
                         const uint8_t* mask, const double* inlet, int32_t nx, int32_t ny, double dx, double dy,
                         double dt, double rho, int32_t boundary_faces, void* stream) {
  if (!u || !v || !u_star || !v_star || !phi || !mask || !inlet) return fail(GM_EVALUE, "null argument");
  if (int rc = check_grid(nx, ny, dx, dy)) return rc;
  if (int rc = check_step(dt, rho)) return rc;
  const size_t nU = (size_t)ny * (nx + 1), nV = (size_t)(ny + 1) * nx, nP = (size_t)ny * nx;
  Staging sg(static_cast<cudaStream_t>(stream));
  const int iu = sg.add(u, nU * 8, true, true), iv = sg.add(v, nV * 8, true, true);
  const int ius = sg.add(u_star, nU * 8, true, false), ivs = sg.add(v_star, nV * 8, true, false);
  const int iph = sg.add(phi, nP * 8, true, false), im = sg.add(mask, nP, true, false);
  const int ii = sg.add(inlet, (size_t)ny * 8, true, false);
  double* extra = nullptr;
  if (cudaError_t e = sg.begin(0, &extra)) return cuda_fail(e);
  const long long n = (long long)(nU + nV);
  if (boundary_faces)
    k_ghost_boundary<<<blocks(n), LT, 0, sg.st>>>(sg.dev<double>(iu), sg.dev<double>(iv), sg.dev<double>(ius),
                                                  sg.dev<double>(ivs), sg.dev<uint8_t>(im), nx, ny, nullptr, nullptr, 0, nullptr);
  else
    k_ghost_correct<<<blocks(n), LT, 0, sg.st>>>(sg.dev<double>(iu), sg.dev<double>(iv), sg.dev<double>(ius),
                                                 sg.dev<double>(ivs), sg.dev<double>(iph), sg.dev<uint8_t>(im),
                                                 sg.dev<double>(ii), nx, ny, dx, dy, dt / rho, nullptr);
  gmk::kernel_launch_adjust(1);
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(e);
  if (cudaError_t e = sg.finish()) return cuda_fail(e);
  return GM_OK;
}

int gm_mac_ghost_forces(const double* u, const double* v, const double* p, int32_t nx, int32_t ny, double dx,
                        double dy, double xc, double yc, double radius, int32_t n_theta, double mu, double out[4],
                        void* stream) {
  if (!u || !v || !p || !out) return fail(GM_EVALUE, "null argument");
  if (int rc = check_grid(nx, ny, dx, dy)) return rc;
  if (n_theta <= 0) return fail(GM_EVALUE, "n_theta must be positive");
  if (!(std::isfinite(mu) && mu >= 0)) return fail(GM_EVALUE, "mu must be finite and nonnegative");
  if (!(std::isfinite(xc) && std::isfinite(yc) && std::isfinite(radius) && radius > 0))
    return fail(GM_EVALUE, "the circle must be finite with a positive radius");
  const size_t nU = (size_t)ny * (nx + 1), nV = (size_t)(ny + 1) * nx, nP = (size_t)ny * nx;
  Staging sg(static_cast<cudaStream_t>(stream));
  const int iu = sg.add(u, nU * 8, true, false), iv = sg.add(v, nV * 8, true, false);
  const int ip = sg.add(p, nP * 8, true, false);
  double* res = nullptr;
  if (cudaError_t e = sg.begin(8 * 8, &res)) return cuda_fail(e);
  k_ghost_forces<<<1, 256, 0, sg.st>>>(sg.dev<double>(iu), sg.dev<double>(iv), sg.dev<double>(ip), nx, ny, dx, dy,
                                       xc, yc, radius, n_theta, mu, res, StepRecord{});
  gmk::kernel_launch_adjust(1);
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(e);
  if (cudaError_t e = cudaMemcpyAsync(out, res, 4 * sizeof(double), cudaMemcpyDeviceToHost, sg.st))
    return cuda_fail(e);
  if (cudaError_t e = sg.finish()) return cuda_fail(e);
  return GM_OK;
}

int gm_mac_forces(const double* u, const double* v, const double* p, const uint8_t* mask, int32_t nx, int32_t ny,
                  double dx, double dy, double mu, double out[4], void* stream) {
  if (!u || !v || !p || !mask || !out) return fail(GM_EVALUE, "null argument");
  if (int rc = check_grid(nx, ny, dx, dy)) return rc;
  if (!(std::isfinite(mu) && mu >= 0)) return fail(GM_EVALUE, "mu must be finite and nonnegative");
  const size_t nU = (size_t)ny * (nx + 1), nV = (size_t)(ny + 1) * nx, nP = (size_t)ny * nx;
  const unsigned nb = blocks((long long)nP);
  Staging sg(static_cast<cudaStream_t>(stream));
  const int iu = sg.add(u, nU * 8, true, false), iv = sg.add(v, nV * 8, true, false);
  const int ip = sg.add(p, nP * 8, true, false), im = sg.add(mask, nP, true, false);
  double* part = nullptr;
  if (cudaError_t e = sg.begin(((size_t)nb * 4 + 8) * 8, &part)) return cuda_fail(e);
  double* res = part + (size_t)nb * 4;
  k_forces_part<<<nb, LT, 0, sg.st>>>(sg.dev<double>(iu), sg.dev<double>(iv), sg.dev<double>(ip), sg.dev<uint8_t>(im),
                                      nx, ny, dx, dy, mu, part);
  k_fold<<<1, LT, 0, sg.st>>>(part, (int)nb, 0, res, StepRecord{});
  gmk::kernel_launch_adjust(2);
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(e);
  if (cudaError_t e = cudaMemcpyAsync(out, res, 4 * sizeof(double), cudaMemcpyDeviceToHost, sg.st))
    return cuda_fail(e);
  if (cudaError_t e = sg.finish()) return cuda_fail(e);
  return GM_OK;
}

int gm_mac_divergence(const double* u, const double* v, const uint8_t* mask, int32_t nx, int32_t ny, double dx,
                      double dy, double out[3], int64_t counts[2], void* stream) {
  if (!u || !v || !mask || !out || !counts) return fail(GM_EVALUE, "null argument");
  if (int rc = check_grid(nx, ny, dx, dy)) return rc;
  const size_t nU = (size_t)ny * (nx + 1), nV = (size_t)(ny + 1) * nx, nP = (size_t)ny * nx;
  const unsigned nb = blocks((long long)nP);
  Staging sg(static_cast<cudaStream_t>(stream));
  const int iu = sg.add(u, nU * 8, true, false), iv = sg.add(v, nV * 8, true, false);
  const int im = sg.add(mask, nP, true, false);
  double* part = nullptr;
  if (cudaError_t e = sg.begin(((size_t)nb * 5 + 8) * 8, &part)) return cuda_fail(e);
  double* res = part + (size_t)nb * 5;
  k_div_part<<<nb, LT, 0, sg.st>>>(sg.dev<double>(iu), sg.dev<double>(iv), sg.dev<uint8_t>(im), nx, ny, dx, dy, part);
  k_fold<<<1, LT, 0, sg.st>>>(part, (int)nb, 1, res, StepRecord{});
  gmk::kernel_launch_adjust(2);
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(e);
  double r[5];
  if (cudaError_t e = cudaMemcpyAsync(r, res, sizeof r, cudaMemcpyDeviceToHost, sg.st)) return cuda_fail(e);
  if (cudaError_t e = sg.finish()) return cuda_fail(e);
  out[0] = r[4];
  out[1] = r[0];
  out[2] = r[2];
  counts[0] = (int64_t)std::llround(r[1]);
  counts[1] = (int64_t)std::llround(r[3]);
  return GM_OK;
}

}  // extern "C"
