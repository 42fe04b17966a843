// Cut-cell (embedded-boundary) AB2/CN step on the GPU: MAC_CylinderFlow(boundary='cut_cell',
// time_scheme='ab2_cn') of the reference (solver/cut_cell_solver.py:790-1015 with
// solver/time_integration.py:7-145).
//
// State and every vector of the step live on the face grid (u then v, ny x (nx+1) and
// (ny+1) x nx, C order) with the non-unknown faces held at zero: the inlet column, covered
// faces and the channel-wall rows of v.  The packed unknown vector of the reference is this
// grid restricted to its active faces, so dot products and norms over the grid equal the
// reference's over q.
//
// Momentum right-hand side (compute_momentum_rhs, solver/cut_cell_solver.py:790-957), one
// evaluation = three launches:
//   k_cc_flux    the four face-flux families on the aperture-weighted staggered faces
//   k_cc_fix     curved faces near the cylinder, one warp per face: advective fluxes from the
//                streamfunction fit at Gauss points, or viscous fluxes from the fitted /
//                ring-corrected gradient, then the wall shear at the circle's Gauss points
//   k_cc_rhs     flux differences into the staggered control volumes (natural outlet row), the
//                wall shear added in the reference's order and the covered-volume transfers
//                (on the few flagged faces), division by rho * owned volume, small-cell
//                merging, covered faces zero, and the packed output (or the CN operator
//                x - dt/2 a for GMRES)
// The CN system is solved by GMRES(30) without a preconditioner (scipy.sparse.linalg.gmres of
// solver/time_integration.py:99-101, rtol 1e-12, atol 1e-13) with its control on the device, over
// an operator on packed vectors that takes one pass (k_cn_eval, k_cn_apply).  The three pressure solves per step use the pressure-only handle of ghostmac.cu
// over the cut-cell Poisson operator (internal.hpp).  One step is one CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "../../include/ghostmac.h"
#include "geometry.hpp"
#include "heldcount.hpp"
#include "internal.hpp"
#include "kernels.cuh"

using namespace gmk;

namespace {

struct CcFail : std::exception {
  int cls;
  std::string msg;
  CcFail(int c, std::string m) : cls(c), msg(std::move(m)) {}
  const char* what() const noexcept override { return msg.c_str(); }
};

#define CCK(call)                                                                                   \
  do {                                                                                              \
    cudaError_t e_ = (call);                                                                        \
    if (e_ != cudaSuccess) throw CcFail(GM_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

template <typename T>
struct Buf {
  T* p = nullptr;
  size_t n = 0;
  Buf() = default;
  Buf(const Buf&) = delete;
  Buf& operator=(const Buf&) = delete;
  ~Buf() { if (p) cudaFree(p); }
  void alloc(size_t count) {
    if (p) { cudaFree(p); p = nullptr; }
    n = count;
    if (count) CCK(cudaMalloc(&p, count * sizeof(T)));
  }
  void upload(const std::vector<T>& v, cudaStream_t st) {
    alloc(v.size());
    if (!v.empty()) CCK(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
  }
  void zero(cudaStream_t st) { if (n) CCK(cudaMemsetAsync(p, 0, n * sizeof(T), st)); }
};

constexpr int CC_TPB = 256;
constexpr int CC_FORCE_THREADS = 512;
inline unsigned nblk(int64_t n, int t = CC_TPB) { return (unsigned)std::max<int64_t>(1, (n + t - 1) / t); }
inline void counted() { note_launch_ext(); }

enum : uint8_t { F_ACTIVE = 1, F_FLUID = 2, F_SOLID = 4, F_AUX = 8 };

// geometry of the face grid (kernel argument)
// GB300 issues FP64 at 1/64 of the FP32 rate, so every per-point factor that does not depend on
// the field is folded on the host: the kernels multiply, they never divide.
struct CcGeo {
  int nx, ny;
  int64_t usize, vsize, psize, F;
  double dx, dy, idx, idy;
  const double *ax, *ay;
  // viscous flux factors (aperture x face length / spacing): F = rho nu (difference) c
  const double *cxx, *cyy;   // ny x nx: ax_mid dy / dx, ay_mid dx / dy
  const double *cxy, *cyx;   // (ny+1) x (nx+1): ay_u dx / dy, ax_v dy / dx
  // advective flux factors (rho x aperture x face length): F = -(transported product) a
  const double *axx, *ayy;   // ny x nx: rho ax_mid dy, rho ay_mid dx
  const double *axy, *ayx;   // (ny+1) x (nx+1): rho ay_u dx, rho ax_v dy
  const double* aout;        // ny: rho ax[:, nx] dy (natural outlet)
  const uint8_t* flags;      // F: F_ACTIVE unknown, F_FLUID divided by its own volume, F_SOLID covered face
  const int32_t* cell_type;  // psize
  const double* kappa;       // psize: fluid fraction
  const double* ikappa;      // psize: 1 / fluid fraction on cut cells, 1 elsewhere
  const double* ivol_rho;    // F: 1 / (rho * owned volume)
  const int32_t* merge_of;   // F: the last merge that writes the face, or -1
  const int64_t* ms;         // merges: small face, master face (face-grid flat), 1 / (rho * merged volume)
  const int64_t* mm;
  const double* imvol_rho;
};

// curved-face flux overrides, the four families concatenated (0 F_xx, 1 F_xy, 2 F_yx, 3 F_yy)
struct CcFix {
  int n_dif;
  const uint8_t* dfam;
  const int64_t* dface;
  const int64_t* dptr;
  const int64_t* dcol;
  const double* dval;
  int n_adv;
  const uint8_t* afam;
  const int64_t* aface;
  const int64_t* apptr;  // n_adv + 1: each face's Gauss points
  const int64_t* uptr;
  const int64_t* ucol;
  const double* uval;
  const int64_t* vptr;
  const int64_t* vcol;
  const double* vval;
  const double* alen;
};

struct CcWall {
  int n;  // Gauss points on the circle
  const int64_t* ptr;
  const int64_t* col;
  const double* val;
  const double* tx;
  const double* ty;
  const double* ds;
  int n_tgt;  // faces receiving wall shear, each with its points in the reference's order
  const int64_t* tgt;
  const int64_t* tptr;
  const int32_t* tk;
  int n_own;  // owners of covered volumes, each with its donors in order
  const int64_t* own;
  const int64_t* optr;
  const int64_t* odon;
  int n_don;
  const int64_t* don;
  double* tau;  // n scratch
  // faces flagged F_AUX (wall targets, owners, donors), sorted, with their target and owner
  // list entries (-1: none) and whether they are donors
  int n_aux;
  const int64_t* aux_face;
  const int32_t* aux_tgt;
  const int32_t* aux_own;
  const uint8_t* aux_don;
};

struct CcFlux {
  double *xx, *xy, *yx, *yy;
};

// Per-step device diagnostics (maxima as the bits of non-negative doubles)
struct CcDiagDev {
  unsigned long long rhs_max, mres, coupled, umax, vmax, divmax;
  unsigned long long pdiv[3];  // predicted divergence of the start-up, first and second solve
  double forces[6];
  double res_linf, res_l2;     // the legacy step's pressure residual b - A phi (unscaled rows)
};

// (row, column) of flat index t on a grid of n columns, in 32 bits (faces are fewer than 2^31): a 64-bit
// division by a run-time value costs some 80 instructions, more than most of these kernels' arithmetic
struct RowCol { int j, i; };
__device__ __forceinline__ RowCol row_col(int64_t t, int n) {
  const unsigned q = (unsigned)t / (unsigned)n;
  return {(int)q, (int)((unsigned)t - q * (unsigned)n)};
}

// field value c of the concatenated face grid, with the inlet column from `inl` when given
__device__ __forceinline__ double fld(const CcGeo& g, const double* __restrict__ X, const double* __restrict__ inl,
                                      int64_t c) {
  if (inl && c < g.usize) {
    const auto [j, i] = row_col(c, g.nx + 1);
    if (i == 0) return inl[j];
  }
  return X[c];
}

// Maxima of |v| run on the bits (non-negative doubles order like them, a NaN above all): integer
// comparisons keep the FP64 pipe, 1/64 of the FP32 rate, for the arithmetic.
using MaxBits = unsigned long long;
__device__ __forceinline__ MaxBits max_abs(MaxBits m, double v) {
  const MaxBits b = (MaxBits)__double_as_longlong(v) & 0x7fffffffffffffffull;
  return b > m ? b : m;
}
// the block's maximum committed with one atomic: warp maxima, then the first warp over the block's warps
__device__ __forceinline__ void block_commit_max(MaxBits m, unsigned long long* out) {
  __shared__ MaxBits wm[32];
  auto warp_max = [](MaxBits v) {
    for (int o = 16; o; o >>= 1) {
      const MaxBits q = __shfl_xor_sync(0xffffffffu, v, o);
      v = q > v ? q : v;
    }
    return v;
  };
  m = warp_max(m);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();  // an earlier call's readers are done with wm
  if (lane == 0) wm[w] = m;
  __syncthreads();
  if (w == 0) {
    m = warp_max(lane < (int)((blockDim.x + 31) >> 5) ? wm[lane] : 0);
    if (lane == 0) atomicMax(out, m);
  }
}

// One CSR row times the field by a whole warp: lanes stride over the row's entries, then a
// butterfly sum leaves the same total in every lane (the pairs add in mirrored order, which
// IEEE addition does not distinguish), in a fixed order from run to run.
__device__ __forceinline__ double warp_row_dot(const int64_t* __restrict__ ptr, const int64_t* __restrict__ col,
                                               const double* __restrict__ val, int64_t r, const CcGeo& g,
                                               const double* __restrict__ X, const double* __restrict__ inl,
                                               int lane) {
  double acc = 0.0;
  for (int64_t e = ptr[r] + lane; e < ptr[r + 1]; e += 32) acc += val[e] * fld(g, X, inl, col[e]);
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// ---- momentum right-hand side -------------------------------------------------------------
// One thread per vertex (j, i) of the (ny+1) x (nx+1) grid: F_xx and F_yy of cell (j, i),
// F_xy and F_yx of vertex (j, i) (solver/cut_cell_solver.py:808-914).  ADV: the advective
// form (nu = 0: no viscous part), with the transported velocity centred or, UPW, taken from
// the upwind side of the face's advecting velocity (transport='upwind'); otherwise the
// viscous form without advection.
template <bool ADV, bool UPW = false>
__global__ void k_cc_flux(CcGeo g, const double* __restrict__ X, const double* __restrict__ inl, double rnu,
                          int slip, CcFlux F) {
  const int nx = g.nx, ny = g.ny;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)(ny + 1) * (nx + 1)) return;
  const auto [j, i] = row_col(t, nx + 1);
  const double* V = X + g.usize;
  auto U = [&](int jj, int ii) -> double {
    const int64_t f = (int64_t)jj * (nx + 1) + ii;
    return (ii == 0 && inl) ? inl[jj] : X[f];
  };
  auto W = [&](int jj, int ii) -> double { return V[(int64_t)jj * nx + ii]; };
  if (j < ny && i < nx) {
    const int64_t c = (int64_t)j * nx + i;
    const double ul = U(j, i), ur = U(j, i + 1), vb = W(j, i), vt = W(j + 1, i);
    if (ADV) {
      const double uf = 0.5 * (ul + ur), vf = 0.5 * (vb + vt);
      const double ua = UPW ? (uf >= 0.0 ? ul : ur) : uf, va = UPW ? (vf >= 0.0 ? vb : vt) : vf;
      F.xx[c] = -(uf * ua * g.axx[c]);
      F.yy[c] = -(vf * va * g.ayy[c]);
    } else {
      F.xx[c] = rnu * (ur - ul) * g.cxx[c];
      F.yy[c] = rnu * (vt - vb) * g.cyy[c];
    }
  }
  {
    double f;
    if (j == 0) f = (ADV || slip) ? 0.0 : rnu * U(0, i) * (2.0 * g.cxy[t]);
    else if (j == ny) f = (ADV || slip) ? 0.0 : -(rnu * U(ny - 1, i) * (2.0 * g.cxy[t]));
    else if (ADV) {
      const double vf = i == 0 ? W(j, 0) : (i == nx ? W(j, nx - 1) : 0.5 * (W(j, i - 1) + W(j, i)));
      const double ua = UPW ? (vf >= 0.0 ? U(j - 1, i) : U(j, i)) : 0.5 * (U(j - 1, i) + U(j, i));
      f = -(vf * ua * g.axy[t]);
    } else {
      f = rnu * (U(j, i) - U(j - 1, i)) * g.cxy[t];
    }
    F.xy[t] = f;
  }
  {
    double f;
    if (i == 0) {
      f = ADV ? 0.0 : rnu * W(j, 0) * (2.0 * g.cyx[t]);
    } else if (i == nx) {
      f = 0.0;
      if (ADV) {
        const double uo = j == 0 ? U(0, nx) : (j == ny ? U(ny - 1, nx) : 0.5 * (U(j - 1, nx) + U(j, nx)));
        f = -(uo * W(j, nx - 1) * g.ayx[t]);
      }
    } else if (ADV) {
      const double uf = j == 0 ? U(0, i) : (j == ny ? U(ny - 1, i) : 0.5 * (U(j - 1, i) + U(j, i)));
      const double va = UPW ? (uf >= 0.0 ? W(j, i - 1) : W(j, i)) : 0.5 * (W(j, i - 1) + W(j, i));
      f = -(uf * va * g.ayx[t]);
    } else {
      f = rnu * (W(j, i) - W(j, i - 1)) * g.cyx[t];
    }
    F.yx[t] = f;
  }
}

// Curved faces (solver/staggered_wall.py:134-140 and the viscous correction of
// solver/cut_cell_solver.py:822-825), one warp per face: ADV: -rho * sum over the face's Gauss
// points of length * (u u | u v | v v) with u, v from the fit; otherwise rho nu (gradient row .
// field), and then one warp per wall Gauss point for its shear stress (wscale = -rho nu).
template <bool ADV>
__global__ void k_cc_fix(CcGeo g, CcFix fx, CcWall w, const double* __restrict__ X, const double* __restrict__ inl,
                         double rnu, double rho, double wscale, CcFlux F) {
  const int lane = threadIdx.x & 31;
  const int r = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  double* fam[4] = {F.xx, F.xy, F.yx, F.yy};
  if (!ADV) {
    if (r < fx.n_dif) {
      const double acc = warp_row_dot(fx.dptr, fx.dcol, fx.dval, r, g, X, inl, lane);
      if (lane == 0) fam[fx.dfam[r]][fx.dface[r]] = rnu * acc;
    } else if (r < fx.n_dif + w.n) {
      // wall shear stress -rho nu (rate . field) at Gauss point k (solver/cut_cell_solver.py:921-924)
      const int k = r - fx.n_dif;
      const double acc = warp_row_dot(w.ptr, w.col, w.val, k, g, X, inl, lane);
      if (lane == 0) w.tau[k] = wscale * acc;
    }
  } else {
    if (r >= fx.n_adv) return;
    const int fm = fx.afam[r];
    double s = 0.0;
    for (int64_t p = fx.apptr[r]; p < fx.apptr[r + 1]; ++p) {
      const double ue = warp_row_dot(fx.uptr, fx.ucol, fx.uval, p, g, X, inl, lane);
      const double ve = warp_row_dot(fx.vptr, fx.vcol, fx.vval, p, g, X, inl, lane);
      const double prod = fm == 0 ? ue * ue : (fm == 3 ? ve * ve : ue * ve);
      s += fx.alen[p] * prod;
    }
    if (lane == 0) fam[fm][fx.aface[r]] = -(rho * s);
  }
}

// Flux differences of face f (solver/cut_cell_solver.py:853-861, 916-917; the natural outlet
// row of u at :857-861)
template <bool ADV>
__device__ __forceinline__ double rhs_base(const CcGeo& g, const CcFlux& F, const double* __restrict__ X, int64_t f) {
  const int nx = g.nx, ny = g.ny;
  if (f < g.usize) {
    const auto [j, i] = row_col(f, nx + 1);
    if (i >= 1 && i < nx)
      return (F.xx[(int64_t)j * nx + i] - F.xx[(int64_t)j * nx + i - 1]) + (F.xy[f + nx + 1] - F.xy[f]);
    if (i == nx) {
      double ext = 0.0;
      if (ADV) {
        const double un = X[f];
        ext = -(un * un * g.aout[j]);
      }
      return (ext - F.xx[(int64_t)j * nx + nx - 1]) + 0.5 * (F.xy[f + nx + 1] - F.xy[f]);
    }
    return 0.0;
  }
  const int64_t c = f - g.usize;
  const auto [j, i] = row_col(c, nx);
  if (j >= 1 && j < ny)
    return (F.yx[(int64_t)j * (nx + 1) + i + 1] - F.yx[(int64_t)j * (nx + 1) + i]) + (F.yy[c] - F.yy[c - nx]);
  return 0.0;
}

__device__ __forceinline__ int aux_find(const CcWall& w, int64_t f) {
  int lo = 0, hi = w.n_aux - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (w.aux_face[mid] < f) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// right-hand side of face f after the wall shear (added in the order of the Gauss points,
// np.add.at of solver/cut_cell_solver.py:922-924)
template <bool ADV>
__device__ double rhs_walled(const CcGeo& g, const CcFlux& F, const CcWall& w, const double* __restrict__ X,
                             int64_t f, int shear, int a) {
  double r = rhs_base<ADV>(g, F, X, f);
  const int t = a >= 0 ? w.aux_tgt[a] : -1;
  if (shear && t >= 0) {
    const double* dir = f < g.usize ? w.tx : w.ty;
    for (int64_t q = w.tptr[t]; q < w.tptr[t + 1]; ++q) {
      const int k = w.tk[q];
      r += w.tau[k] * dir[k] * w.ds[k];
    }
  }
  return r;
}

// the full right-hand side of face f: flux differences, wall shear, then the covered-volume
// transfers (donors give their whole value to their owner in donor order and hold zero;
// solid/staggered_wall.py:302-304)
template <bool ADV>
__device__ double rhs_full(const CcGeo& g, const CcFlux& F, const CcWall& w, const double* __restrict__ X, int64_t f,
                           int shear) {
  if (!(g.flags[f] & F_AUX)) return rhs_base<ADV>(g, F, X, f);
  const int a = aux_find(w, f);
  if (w.aux_don[a]) return 0.0;
  double r = rhs_walled<ADV>(g, F, w, X, f, shear, a);
  const int o = w.aux_own[a];
  if (o >= 0)
    for (int64_t q = w.optr[o]; q < w.optr[o + 1]; ++q) {
      const int64_t d = w.odon[q];
      r += rhs_walled<ADV>(g, F, w, X, d, shear, (g.flags[d] & F_AUX) ? aux_find(w, d) : -1);
    }
  return r;
}

// Right-hand side and accelerations in one pass (solver/cut_cell_solver.py:853-955): flux
// differences, wall shear and covered transfers (flagged faces only), division by rho x owned
// volume (a multiply by the host-formed reciprocal), small-cell merging, covered faces zero.
// mode 0: Y = packed a; 1: Y = packed (X - hdt a) (the CN operator); 2: Y = a and Rout = rhs,
// both unpacked.
template <bool ADV>
__global__ void k_cc_rhs(CcGeo g, CcFlux F, CcWall w, const double* __restrict__ X, int shear, double hdt, int mode,
                         double* __restrict__ Y, double* __restrict__ Rout) {
  const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= g.F) return;
  const uint8_t fl = g.flags[f];
  const double r = rhs_full<ADV>(g, F, w, X, f, shear);
  double a = 0.0;
  if (fl & F_FLUID) a = r * g.ivol_rho[f];
  const int m = g.merge_of[f];
  if (m >= 0) {
    const int64_t fs = g.ms[m], fm = g.mm[m];
    const double rs = fs == f ? r : rhs_full<ADV>(g, F, w, X, fs, shear);
    const double rm = fm == f ? r : rhs_full<ADV>(g, F, w, X, fm, shear);
    a = (rs + rm) * g.imvol_rho[m];
  }
  if (fl & F_SOLID) a = 0.0;
  if (mode == 0) Y[f] = (fl & F_ACTIVE) ? a : 0.0;
  else if (mode == 1) Y[f] = (fl & F_ACTIVE) ? X[f] - hdt * a : 0.0;
  else {
    Y[f] = a;
    Rout[f] = (fl & F_SOLID) ? 0.0 : r;
  }
}

// ---- projection pieces ----------------------------------------------------------------------
// (rho / dt) times the aperture-weighted divergence of the unpacked field, zero on covered
// cells (compute_rhs, solver/cut_cell_solver.py:732-738), divided by kappa on cut cells (the row
// scaling of the pressure system built by gm::build_cutcell_geometry)
__global__ void k_cc_divrhs(CcGeo g, const double* __restrict__ X, const double* __restrict__ inl, double inv_dt,
                            double* __restrict__ B) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.psize) return;
  if (g.cell_type[c] == -1) { B[c] = 0.0; return; }
  const int nx = g.nx;
  const auto [j, i] = row_col(c, nx);
  const int64_t fu = (int64_t)j * (nx + 1) + i;
  const double uw = (i == 0 && inl) ? inl[j] : X[fu];
  const double* V = X + g.usize;
  const double fx = (g.ax[fu + 1] * X[fu + 1] - g.ax[fu] * uw) * g.idx;
  const double fy = (g.ay[c + nx] * V[c + nx] - g.ay[c] * V[c]) * g.idy;
  B[c] = inv_dt * (fx + fy) * g.ikappa[c];
}
// a caller's right-hand side in the row scaling of the pressure system: cut cells / kappa,
// covered cells zero
__global__ void k_cc_scale_rhs(CcGeo g, double* __restrict__ B) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.psize) return;
  B[c] = g.cell_type[c] == -1 ? 0.0 : B[c] * g.ikappa[c];
}

// corrector (solver/cut_cell_solver.py:740-753), packed output; sx = dt / (rho dx), sy = dt / (rho dy).
// With a residual: also the predicted divergence dt/rho max_fluid |res| / kappa (:721-722; the residual
// of the row-scaled system already carries the 1 / kappa).
__global__ void k_cc_correct(CcGeo g, const double* __restrict__ X, const double* __restrict__ phi, double sx,
                             double sy, double* __restrict__ Y, const double* __restrict__ res, double scale,
                             unsigned long long* out) {
  const int nx = g.nx, ny = g.ny;
  MaxBits m = 0;
  for (int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; f < g.F; f += (int64_t)gridDim.x * blockDim.x) {
    double r = 0.0;
    if (f < g.usize) {
      const auto [j, i] = row_col(f, nx + 1);
      const int64_t c = (int64_t)j * nx + i;
      if (i >= 1 && i < nx) r = g.ax[f] > 0.0 ? X[f] - sx * (phi[c] - phi[c - 1]) : 0.0;
      else if (i == nx) r = X[f] + (2.0 * sx) * phi[c - 1];
    } else {
      const int64_t c = f - g.usize;
      const int j = row_col(c, nx).j;
      if (j >= 1 && j < ny) r = g.ay[c] > 0.0 ? X[f] - sy * (phi[c] - phi[c - nx]) : 0.0;
    }
    Y[f] = (g.flags[f] & F_ACTIVE) ? r : 0.0;
    if (res && f < g.psize && g.cell_type[f] != -1) m = max_abs(m, scale * res[f]);
  }
  if (res) block_commit_max(m, out);
}

// pressure gradient / rho at face f (advance_ab2_cn's gradient, solver/cut_cell_solver.py:979-984), zero on
// faces that are not unknown; gx = 1 / (rho dx), gy = 1 / (rho dy)
__device__ __forceinline__ double face_grad(const CcGeo& g, const double* __restrict__ P, double gx, double gy, int64_t f) {
  if (!(g.flags[f] & F_ACTIVE)) return 0.0;
  const int nx = g.nx, ny = g.ny;
  if (f < g.usize) {
    const auto [j, i] = row_col(f, nx + 1);
    const int64_t c = (int64_t)j * nx + i;
    if (i >= 1 && i < nx) return (P[c] - P[c - 1]) * gx;
    return i == nx ? -2.0 * P[c - 1] * gx : 0.0;
  }
  const int64_t c = f - g.usize;
  const int j = row_col(c, nx).j;
  return j >= 1 && j < ny ? (P[c] - P[c - nx]) * gy : 0.0;
}

// face f of the unpacked field: inlet column, packed values on the unknown faces, zero elsewhere
__device__ __forceinline__ double unpacked(const CcGeo& g, const double* __restrict__ X, const double* __restrict__ inl,
                                           int64_t f) {
  if (f < g.usize) {
    const auto [j, i] = row_col(f, g.nx + 1);
    if (i == 0) return inl[j];
  }
  return (g.flags[f] & F_ACTIVE) ? X[f] : 0.0;
}
// pack (X = masked U) and unpack (U = X with the inlet column)
__global__ void k_cc_pack(CcGeo g, const double* __restrict__ U, double* __restrict__ X) {
  const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (f < g.F) X[f] = (g.flags[f] & F_ACTIVE) ? U[f] : 0.0;
}
__global__ void k_cc_unpack(CcGeo g, const double* __restrict__ X, const double* __restrict__ inl,
                            double* __restrict__ U) {
  const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= g.F) return;
  U[f] = unpacked(g, X, inl, f);
}

// max |a - b| (b may be null), max |(a - b) + s c| with c set
__global__ void k_cc_maxdiff(int64_t n, const double* __restrict__ a, const double* __restrict__ b,
                             const double* __restrict__ c, double s, unsigned long long* out) {
  MaxBits m = 0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    double v = b ? a[t] - b[t] : a[t];
    if (c) v = v + s * c[t];
    m = max_abs(m, v);
  }
  block_commit_max(m, out);
}
// predicted divergence dt/rho max_fluid |res| / kappa (solver/cut_cell_solver.py:721-722); the
// residual of the row-scaled system already carries the 1 / kappa
__global__ void k_cc_pdiv(CcGeo g, const double* __restrict__ res, double scale, unsigned long long* out) {
  MaxBits m = 0;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < g.psize; c += (int64_t)gridDim.x * blockDim.x)
    if (g.cell_type[c] != -1) m = max_abs(m, scale * res[c]);
  block_commit_max(m, out);
}
// step gate quantities of solver/main.py:416-424: max_fluid |flux divergence| / kappa, max |u|, max |v|
__global__ void k_cc_stepmax(CcGeo g, const double* __restrict__ U, unsigned long long* divmax,
                             unsigned long long* umax, unsigned long long* vmax) {
  const int nx = g.nx;
  MaxBits dm = 0, um = 0, vm = 0;
  const double* V = U + g.usize;
  for (int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; f < g.F; f += (int64_t)gridDim.x * blockDim.x) {
    if (f < g.usize) um = max_abs(um, U[f]);
    else vm = max_abs(vm, U[f]);
    if (f < g.psize && g.cell_type[f] != -1) {
      const int64_t c = f;
      const auto [j, i] = row_col(c, nx);
      const int64_t fu = (int64_t)j * (nx + 1) + i;
      const double d = (g.ax[fu + 1] * U[fu + 1] - g.ax[fu] * U[fu]) * g.idx +
                       (g.ay[c + nx] * V[c + nx] - g.ay[c] * V[c]) * g.idy;
      dm = max_abs(dm, d * g.ikappa[c]);
    }
  }
  block_commit_max(dm, divmax);
  block_commit_max(um, umax);
  block_commit_max(vm, vmax);
}

// The legacy predictor (advance_momentum_predictor, solver/cut_cell_solver.py:1017-1033) and
// apply_predictor_boundary (:663-670): a = advective + viscous acceleration, u* = u + dt a
// (forward Euler) or u + dt ((1 + alpha) a - alpha a_prev) (AB2), a_prev = a; then the inlet
// column, zero on closed faces and on the channel-wall v rows.
__global__ void k_cc_legacy_pred(CcGeo g, const double* __restrict__ U, const double* __restrict__ aa,
                                 const double* __restrict__ ad, double* __restrict__ prev,
                                 const double* __restrict__ inl, double dt, double alpha, int ab2,
                                 double* __restrict__ star) {
  const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= g.F) return;
  const double a = aa[f] + ad[f];
  double s = ab2 ? U[f] + dt * ((1 + alpha) * a - alpha * prev[f]) : U[f] + dt * a;
  prev[f] = a;
  if (f < g.usize) {
    const auto [j, i] = row_col(f, g.nx + 1);
    if (i == 0) s = inl[j];
    if (g.ax[f] == 0.0) s = 0.0;
  } else {
    const int64_t c = f - g.usize;
    const int j = row_col(c, g.nx).j;
    if (g.ay[c] == 0.0 || j == 0 || j == g.ny) s = 0.0;
  }
  star[f] = s;
}

// max |r| and sum r^2 of the pressure residual in the unscaled rows (the row-scaled residual
// times kappa), per block, then folded by one block in a fixed order (deterministic)
constexpr int CC_RES_BLOCKS = 152;
__global__ void k_cc_resnorm_part(CcGeo g, const double* __restrict__ res, double* __restrict__ part) {
  __shared__ double smax[CC_TPB], ssum[CC_TPB];
  double m = 0.0, q = 0.0;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < g.psize; c += (int64_t)gridDim.x * blockDim.x)
    if (g.cell_type[c] != -1) {
      const double r = res[c] * g.kappa[c];
      m = (r != r) ? r : fmax(m, fabs(r));
      q += r * r;
    }
  smax[threadIdx.x] = m;
  ssum[threadIdx.x] = q;
  __syncthreads();
  for (int k = CC_TPB / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) {
      const double o = smax[threadIdx.x + k];
      smax[threadIdx.x] = (o != o) ? o : fmax(smax[threadIdx.x], o);
      ssum[threadIdx.x] += ssum[threadIdx.x + k];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = smax[0];
    part[2 * blockIdx.x + 1] = ssum[0];
  }
}
__global__ void k_cc_resnorm_fold(const double* __restrict__ part, int nb, double* __restrict__ linf,
                                  double* __restrict__ l2) {
  __shared__ double smax[CC_TPB], ssum[CC_TPB];
  double m = 0.0, q = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const double o = part[2 * b];
    m = (o != o) ? o : fmax(m, o);
    q += part[2 * b + 1];
  }
  smax[threadIdx.x] = m;
  ssum[threadIdx.x] = q;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) {
      const double o = smax[threadIdx.x + k];
      smax[threadIdx.x] = (o != o) ? o : fmax(smax[threadIdx.x], o);
      ssum[threadIdx.x] += ssum[threadIdx.x + k];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *linf = smax[0];
    *l2 = sqrt(ssum[0]);
  }
}

// fixed-order block sum of one value per thread, the same in every thread (at most 32 warps)
__device__ double block_sum(double v, double* sh) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  v = (int)(threadIdx.x & 31) < (int)(blockDim.x >> 5) ? sh[threadIdx.x & 31] : 0.0;
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  return v;
}

// mu (rate . field) at every wall Gauss point and the pressure at every surface point, one warp each
__global__ void k_cc_wall_points(gmi::SurfaceCsr S, CcWall w, const double* __restrict__ U, const double* __restrict__ P,
                                 double mu, double* __restrict__ tau, double* __restrict__ pb) {
  const int lane = threadIdx.x & 31;
  const int k = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (k >= w.n + S.n) return;  // whole warps leave together
  const bool wall = k < w.n;
  const double acc = wall ? warp_row_dot(w.ptr, w.col, w.val, k, CcGeo{}, U, nullptr, lane)
                          : warp_row_dot(S.ptr, S.col, S.val, k - w.n, CcGeo{}, P, nullptr, lane);
  if (lane == 0) {
    if (wall) tau[k] = mu * acc;
    else pb[k - w.n] = acc;
  }
}

// Forces on the true circle (extract_true_surface_forces, solver/cut_cell_solver.py:755-765):
// pressure from the point reconstruction with its mean removed, shear mu (rate . field) at
// the wall Gauss points.  One block; out = fx, fy, fx_p, fy_p, fx_v, fy_v.
__global__ void k_cc_forces(gmi::SurfaceCsr S, CcWall w, const double* __restrict__ tau, const double* __restrict__ pb,
                            double* __restrict__ out) {
  __shared__ double sh[CC_FORCE_THREADS];
  const int tid = threadIdx.x, nt = blockDim.x;
  double s = 0.0;
  for (int k = tid; k < S.n; k += nt) s += pb[k];
  const double mean = block_sum(s, sh) / S.n;
  double px = 0.0, py = 0.0;
  for (int k = tid; k < S.n; k += nt) {
    const double d = pb[k] - mean;
    px += d * S.nwx[k];
    py += d * S.nwy[k];
  }
  double vx = 0.0, vy = 0.0;
  for (int k = tid; k < w.n; k += nt) {
    const double t = tau[k] * w.ds[k];
    vx += t * w.tx[k];
    vy += t * w.ty[k];
  }
  const double fxp = -block_sum(px, sh), fyp = -block_sum(py, sh);
  const double fxv = block_sum(vx, sh), fyv = block_sum(vy, sh);
  if (tid == 0) {
    out[0] = fxp + fxv;
    out[1] = fyp + fyv;
    out[2] = fxp;
    out[3] = fyp;
    out[4] = fxv;
    out[5] = fyv;
  }
}

// calculate_cut_cell_divergence (solver/cut_cell_solver.py:219-260): max |div|, sum div^2,
// fluid count, max |net flux|, one block in a fixed order
__global__ void k_cc_divstats(CcGeo g, const double* __restrict__ U, double* __restrict__ out) {
  __shared__ double sh[CC_FORCE_THREADS];
  const int nx = g.nx;
  const double* V = U + g.usize;
  double mdiv = 0.0, sq = 0.0, cnt = 0.0, mflux = 0.0;
  for (int64_t c = threadIdx.x; c < g.psize; c += blockDim.x) {
    if (g.cell_type[c] == -1) continue;
    const auto [j, i] = row_col(c, nx);
    const int64_t fu = (int64_t)j * (nx + 1) + i;
    const double fx = g.ax[fu + 1] * g.dy * U[fu + 1] - g.ax[fu] * g.dy * U[fu];
    const double fy = g.ay[c + nx] * g.dx * V[c + nx] - g.ay[c] * g.dx * V[c];
    const double net = fx + fy;
    const double vol = g.kappa[c] * g.dx * g.dy;  // diagnostics only: the reference's division
    const double d = vol > 0.0 ? net / vol : 0.0;
    mdiv = fmax(mdiv, fabs(d));
    mflux = fmax(mflux, fabs(net));
    sq += d * d;
    cnt += 1.0;
  }
  const double tsq = block_sum(sq, sh), tcnt = block_sum(cnt, sh);
  sh[threadIdx.x] = mdiv;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + s]);
    __syncthreads();
  }
  const double tmd = sh[0];
  __syncthreads();
  sh[threadIdx.x] = mflux;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = tmd;
    out[1] = tsq;
    out[2] = tcnt;
    out[3] = sh[0];
  }
}

// ---- the viscous operator of the CN step --------------------------------------------------
// L x on packed vectors (zero on faces that are not unknown; the inlet's part is the constant vector
// `offset`).  By flux arrays it is three kernels (k_cc_flux, k_cc_fix, k_cc_rhs: 45 us at 800x410, four
// arrays through L2 and three launches); as an operator on packed vectors it is one pass, because
// every face near the body is one sparse row formed at set-up (curved fluxes, wall shear, covered
// transfers and merging are linear), and every other face is a five-point stencil: the constant one
// where apertures and volumes are full, the structured one at the channel's edges.  16 us with the vector
// step behind it at 800x410; the FP64 pipe is the bound (5 multiply-adds a regular face).
struct CnOp {
  const uint8_t* cls;    // per face: CN_ZERO, CN_REGULAR, CN_EDGE or CN_ROW
  int n_row;             // rows near the body
  const int32_t* face;
  const int64_t* ptr;
  const int32_t* col;
  const double* val;
  double kx, ky;         // nu / dx^2, nu / dy^2 of the regular faces
  double rnu;
  int slip;
};
enum : uint8_t { CN_ZERO = 0, CN_REGULAR = 1, CN_EDGE = 2, CN_ROW = 3 };

// (L x)(f) of a face at the channel's edge, or with apertures or a volume of its own
__device__ double cn_edge(const CcGeo& g, const CnOp& L, const double* __restrict__ X, int64_t f) {
  if (!(g.flags[f] & F_FLUID) || (g.flags[f] & F_SOLID)) return 0.0;
  const int nx = g.nx, ny = g.ny;
  double r = 0.0;
  if (f < g.usize) {
    const auto [j, i] = row_col(f, nx + 1);
    const int64_t c = (int64_t)j * nx + i;
    if (i == 0) return 0.0;
    const double fs = j == 0 ? (L.slip ? 0.0 : X[f] * (2.0 * g.cxy[f])) : (X[f] - X[f - nx - 1]) * g.cxy[f];
    const double fn = j == ny - 1 ? (L.slip ? 0.0 : -(X[f] * (2.0 * g.cxy[f + nx + 1])))
                                  : (X[f + nx + 1] - X[f]) * g.cxy[f + nx + 1];
    const double fw = (X[f] - X[f - 1]) * g.cxx[c - 1];
    r = i == nx ? 0.5 * (fn - fs) - fw : ((X[f + 1] - X[f]) * g.cxx[c] - fw) + (fn - fs);
  } else {
    const int64_t c = f - g.usize;
    const auto [j, i] = row_col(c, nx);
    if (j == 0 || j == ny) return 0.0;
    const int64_t t = (int64_t)j * (nx + 1) + i;
    const double fw = i == 0 ? X[f] * (2.0 * g.cyx[t]) : (X[f] - X[f - 1]) * g.cyx[t];
    const double fe = i + 1 == nx ? 0.0 : (X[f + 1] - X[f]) * g.cyx[t + 1];
    r = (fe - fw) + ((X[f + nx] - X[f]) * g.cyy[c] - (X[f] - X[f - nx]) * g.cyy[c - nx]);
  }
  return L.rnu * r * g.ivol_rho[f];
}

// the stencil of H on regular faces: H x = c x - x_w (west + east) - y (south + north)
struct CnH {
  double hdt, c, x, y;
};
inline CnH cn_h(const CnOp& L, double hdt) { return {hdt, 1.0 + 2.0 * (hdt * L.kx + hdt * L.ky), hdt * L.kx, hdt * L.ky}; }

// Every face once over the whole grid of threads: f(face, x, value), value = L x (H = false) or
// s (x - hdt L x) (H = true, the stencil h holding the factor s); faces that are not unknown report 0, 0.  The rows near the body, a warp
// each (its lane 0 reports), go to blocks of their own: their chain of loads would otherwise come on
// top of those warps' share of the sweep.
template <bool H, class Fn>
__device__ __forceinline__ void cn_sweep(const CcGeo& g, const CnOp& L, const double* __restrict__ X, const CnH& h, double s,
                                         Fn&& fn) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int rb = min((L.n_row + nw - 1) / nw, (int)(gridDim.x / 4));  // at least one when there are rows (gridDim >= 4)
  if ((int)blockIdx.x < rb) {
    for (int r = blockIdx.x * nw + (threadIdx.x >> 5); r < L.n_row; r += rb * nw) {
      double a = 0.0;
      for (int64_t e = L.ptr[r] + lane, e1 = L.ptr[r + 1]; e < e1; e += 32) a += L.val[e] * X[L.col[e]];
      for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (lane == 0) {
        const int64_t f = L.face[r];
        const double x = X[f];
        fn(f, x, H ? s * (x - h.hdt * a) : a);
      }
    }
    return;
  }
  for (int64_t f = (int64_t)(blockIdx.x - rb) * blockDim.x + threadIdx.x; f < g.F; f += (int64_t)(gridDim.x - rb) * blockDim.x) {
    const uint8_t k = L.cls[f];
    if (k == CN_ROW) continue;
    double x = 0.0, v = 0.0;
    if (k == CN_REGULAR) {
      const int up = f < g.usize ? g.nx + 1 : g.nx;
      x = X[f];
      const double ew = X[f - 1] + X[f + 1], ns = X[f - up] + X[f + up];
      if (H) v = (h.c * x - h.x * ew) - h.y * ns;
      else v = L.kx * (ew - 2.0 * x) + L.ky * (ns - 2.0 * x);
    } else if (k == CN_EDGE) {
      x = X[f];
      const double a = cn_edge(g, L, X, f);
      v = H ? s * (x - h.hdt * a) : a;
    }
    fn(f, x, v);
  }
}

// The vector steps around the operator (solver/time_integration.py:7-145), one pass each:
// CN_MID     out = x + dt ((a + d) - grad p), d = L x + offset      (projected midpoint start-up; dt is its half step)
// CN_RHS     out = (x + dt ((e + d / 2) - grad p)) + hdt offset, out2 = x (the first iterate),
//            e = (1 + s) a - s b (AB2) or a (b null); max |out|
// CN_CHECK   max |H x - a|
// CN_ACTION  out = H x, out2 = x + (a - H x)                           (projected result plus the momentum defect)
// CN_H       out = H x; CN_L: out = L x + offset
enum CnMode { CN_MID, CN_RHS, CN_CHECK, CN_ACTION, CN_H, CN_L };
struct CnEval {
  const double *x, *a, *b, *offset, *p;
  double dt, hdt, s, gx, gy;
  CnH h;
  double *out, *out2;
  unsigned long long* mx;
};
template <int MODE>
__global__ void k_cn_eval(CcGeo g, CnOp L, CnEval e) {
  constexpr bool H = MODE == CN_CHECK || MODE == CN_ACTION || MODE == CN_H;
  MaxBits m = 0;
  cn_sweep<H>(g, L, e.x, e.h, 1.0, [&](int64_t f, double x, double v) {
    if (MODE == CN_MID || MODE == CN_RHS) {
      const double d = v + e.offset[f], gp = face_grad(g, e.p, e.gx, e.gy, f);
      if (MODE == CN_MID) e.out[f] = x + e.dt * ((e.a[f] + d) - gp);
      else {
        const double ex = e.b ? (1 + e.s) * e.a[f] - e.s * e.b[f] : e.a[f];
        const double r = (x + e.dt * ((ex + 0.5 * d) - gp)) + e.hdt * e.offset[f];
        e.out[f] = r;
        e.out2[f] = x;
        m = max_abs(m, r);
      }
    } else if (MODE == CN_CHECK) {
      m = max_abs(m, v - e.a[f]);
    } else if (MODE == CN_ACTION) {
      e.out[f] = v;
      e.out2[f] = x + (e.a[f] - v);
    } else {
      e.out[f] = MODE == CN_L ? v + e.offset[f] : v;
    }
  });
  if (MODE == CN_RHS || MODE == CN_CHECK) block_commit_max(m, e.mx);
}

// ---- GMRES(30) of the CN system ---------------------------------------------------------------
// H x = b from x0 = x (solver/time_integration.py:99-101: rtol 1e-12, atol 1e-13, restart 30, at most
// 100 cycles), no preconditioner, two classical Gram-Schmidt passes, Givens rotations.  An Arnoldi
// step is three kernels: k_cn_apply (operator and the first pass's dots while w is in registers),
// k_cn_pass<false> (first update, second pass's dots) and k_cn_pass<true> (second update, |w|^2).  The
// last block of the third to finish holds the whole column, so it does the rotations, the
// convergence test and the next scale: basis vectors stay unscaled in memory (v_i = sc[i] V_i), the
// scales enter the coefficients.  A step is bound by the FP64 pipe (some 6 + 3 nv multiply-adds a
// face) and the basis in L2.
// A step graph holds `steps` Arnoldi steps, each gated by `go`, and no conditional node (8 us each
// even when its body does not run: 30 of them and the loop were 250 of 590 us).  A system that needs
// more stops the step (ERR_SWEEPS) before any state is written and the host repeats it with more;
// beyond 30 the cycle runs in a WHILE node.  At 800x410 (5 Arnoldi steps) the solve took 588 us, now 306;
// one block of 512 threads an SM, as two cost 12 us more (twice the sums to fold).
constexpr int CN_BLOCKS = 152;
constexpr int CN_THREADS = 512;
constexpr int CN_M = 30;
constexpr int CN_SHORT = 5;  // gate word of ERR_SWEEPS when the Arnoldi steps did not suffice (below: solve slots)
struct CnDev {
  double H[CN_M * CN_M];     // R of the rotated Hessenberg matrix, row i column j at i M + j
  double cs[CN_M], sn[CN_M], g[CN_M + 1], sc[CN_M + 1], d1[CN_M], coef[CN_M];
  double tol;
  int jend, cycle, its, converged, go, nv;
  unsigned ticket;
};

// Block sums of NA values a thread, value i of this block to part[i CN_BLOCKS + block].  An FP64 warp
// instruction occupies the pipe for 16 cycles, so the sums take as few as they can: up to four values
// go through shared memory to a warp each (21 additions a value instead of 5 a warp and value); for
// more, lanes exchange halves of their values (about NA + 5 additions a warp instead of 5 NA).
template <int NA>
__device__ __forceinline__ void cn_partials_few(double (&acc)[NA], double* __restrict__ part) {
  __shared__ double red[NA][CN_THREADS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NA; ++i) red[i][threadIdx.x] = acc[i];
  __syncthreads();
  if (warp >= NA) return;
  double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < CN_THREADS / 32; ++q) a[q & 3] += red[warp][32 * q + lane];
  double v = (a[0] + a[1]) + (a[2] + a[3]);
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) part[(int64_t)warp * CN_BLOCKS + blockIdx.x] = v;
}
template <int NA>
__device__ __forceinline__ void cn_partials(double (&acc)[NA], int na, double* __restrict__ part) {
  if constexpr (NA <= 4) {
    cn_partials_few(acc, part);
    return;
  }
  __shared__ double red[NA][CN_THREADS / 32];
  constexpr int K = NA > 16 ? 5 : NA > 8 ? 4 : NA > 4 ? 3 : NA > 2 ? 2 : NA > 1 ? 1 : 0;  // 2^K >= NA
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int o = 16 >> k, half = k < K ? 1 << (K - 1 - k) : 0;  // lane bit o takes the upper half of the values
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < (k < K ? half : 1); ++i) {
      if (i < NA) {
        const bool pair = k < K && i + half < NA;
        const double other = pair ? acc[pair ? i + half : 0] : acc[i];
        const double send = pair && !up ? other : acc[i], keep = pair && up ? other : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
  const int i = lane >> (5 - K);
  if ((lane & ((1 << (5 - K)) - 1)) == 0 && i < NA) red[i][warp] = acc[0];
  __syncthreads();
  for (int q = threadIdx.x; q < na; q += CN_THREADS) {
    double a = 0.0;
    for (int w = 0; w < CN_THREADS / 32; ++w) a += red[q][w];
    part[(int64_t)q * CN_BLOCKS + blockIdx.x] = a;
  }
}
// sum over the blocks of value i, by one warp in a fixed order
__device__ __forceinline__ double cn_fold(const double* part, int i, int lane) {
  double a = 0.0;
  for (int b = lane; b < CN_BLOCKS; b += 32) a += __ldcg(part + (int64_t)i * CN_BLOCKS + b);
  for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}
// whether this block is the last of the grid to get here; what the others wrote before is then visible
__device__ __forceinline__ bool cn_last_block(CnDev* gd) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&gd->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last) __threadfence();
  return last != 0;
}

// V_0 = b - H x, and the start of a cycle
__global__ void __launch_bounds__(CN_THREADS) k_cn_start(CcGeo g, CnOp L, const double* __restrict__ x, CnH h,
                                                         const double* __restrict__ b, double* __restrict__ V,
                                                         double* part, CnDev* gd, int first) {
  double acc[2] = {0.0, 0.0};
  cn_sweep<true>(g, L, x, h, 1.0, [&](int64_t f, double, double v) {
    const double bf = b[f], r = bf - v;
    V[f] = r;
    acc[0] += r * r;
    acc[1] += bf * bf;
  });
  cn_partials(acc, 2, part);
  if (!cn_last_block(gd)) return;
  if (threadIdx.x >= 32) return;
  const double r2 = cn_fold(part, 0, threadIdx.x), b2 = cn_fold(part, 1, threadIdx.x);
  if (threadIdx.x != 0) return;
  const double beta = sqrt(r2), tol = fmax(1e-12 * sqrt(b2), 1e-13);
  if (first) gd->cycle = gd->its = gd->converged = 0;
  const bool go = beta > tol;
  if (!go) gd->converged = isfinite(beta) ? 1 : 0;
  gd->tol = tol;
  gd->jend = -1;
  gd->nv = 0;
  gd->sc[0] = 1.0 / beta;
  gd->g[0] = beta;
  gd->go = go ? 1 : 0;
  gd->ticket = 0;
}

// w = H v_j (v_j = sc[j] V_j, nv = j + 1) and the partial dots of the unscaled basis with w
template <int NV>
__global__ void __launch_bounds__(CN_THREADS, 1) k_cn_apply(CcGeo g, CnOp L, const double* __restrict__ V, int nv,
                                                             CnH h, double* __restrict__ w, double* __restrict__ part,
                                                             const CnDev* __restrict__ gd) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!gd->go) return;
  const int64_t n = g.F;
  __shared__ CnH hs;
  const double s = gd->sc[nv - 1];
  if (threadIdx.x == 0) hs = CnH{h.hdt, s * h.c, s * h.x, s * h.y};
  __syncthreads();
  double acc[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) acc[i] = 0.0;
  cn_sweep<true>(g, L, V + (int64_t)(nv - 1) * n, hs, s, [&](int64_t f, double, double y) {
    w[f] = y;
    const double* p = V + f;
#pragma unroll
    for (int i = 0; i < NV; ++i, p += n)
      if (NV <= 8 || i < nv) acc[i] += *p * y;
  });
  cn_partials(acc, nv, part);
}

// w -= V c, c from the partials of the previous kernel; then the partials of V^T w (NORM = false) or of
// |w|^2 and the end of the Arnoldi step (NORM = true).  ctl is set on the last step that the graph
// holds when it may be followed by more.
template <int NV, bool NORM>
__global__ void __launch_bounds__(CN_THREADS, 1) k_cn_pass(const double* __restrict__ V, int64_t n, int nv,
                                                            const double* __restrict__ part_in, double* __restrict__ w,
                                                            double* part_out, CnDev* gd, int last_step, StepCtl* ctl) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!gd->go) return;
  __shared__ double cf[NV], ck[NV];  // coefficients in the scaled and in the unscaled basis
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = warp; i < nv; i += CN_THREADS / 32) {
    const double s = gd->sc[i], c = s * cn_fold(part_in, i, lane);
    if (lane == 0) { cf[i] = c; ck[i] = s * c; }
  }
  __syncthreads();
  if (!NORM && blockIdx.x == 0 && threadIdx.x < nv) gd->d1[threadIdx.x] = cf[threadIdx.x];
  constexpr int NA = NORM ? 1 : NV;
  double acc[NA];
#pragma unroll
  for (int i = 0; i < NA; ++i) acc[i] = 0.0;
  for (int64_t t = (int64_t)blockIdx.x * CN_THREADS + threadIdx.x; t < n; t += (int64_t)CN_BLOCKS * CN_THREADS) {
    double v[NV <= 8 ? NV : 1];  // wider bases are read twice (the second time from L1)
    double s = 0.0;
    const double* p = V + t;
#pragma unroll
    for (int i = 0; i < NV; ++i, p += n)
      if (NV <= 8 || i < nv) {
        const double vi = *p;
        if (NV <= 8) v[NV <= 8 ? i : 0] = vi;
        s += ck[i] * vi;
      }
    const double wt = w[t] - s;
    w[t] = wt;
    if (NORM) acc[0] += wt * wt;
    else {
      p = V + t;
#pragma unroll
      for (int i = 0; i < NA; ++i, p += n)
        if (NV <= 8 || i < nv) acc[i] += (NV <= 8 ? v[NV <= 8 ? i : 0] : *p) * wt;
    }
  }
  cn_partials(acc, NORM ? 1 : nv, part_out);
  if (!NORM) return;
  if (!cn_last_block(gd)) return;
  if (threadIdx.x >= 32) return;
  // the end of Arnoldi step j (one warp): column j of H, the rotations, the residual estimate
  const int j = nv - 1;
  __shared__ double hc[CN_M + 1], cs[CN_M], sn[CN_M];
  const double w2 = cn_fold(part_out, 0, lane);
  if (lane < nv) hc[lane] = __ldcg(&gd->d1[lane]) + cf[lane];
  if (lane < j) { cs[lane] = gd->cs[lane]; sn[lane] = gd->sn[lane]; }
  __syncwarp();
  __shared__ int stop;
  if (lane == 0) {
    const double h = sqrt(w2);
    double below = h;
    for (int i = 0; i < j; ++i) {
      const double a = cs[i] * hc[i] + sn[i] * hc[i + 1];
      hc[i + 1] = -sn[i] * hc[i] + cs[i] * hc[i + 1];
      hc[i] = a;
    }
    const double den = hypot(hc[j], below), inv = 1.0 / den, c = den > 0 ? hc[j] * inv : 1.0, s = den > 0 ? below * inv : 0.0;
    hc[j] = den;
    gd->cs[j] = c;
    gd->sn[j] = s;
    const double gj = gd->g[j], r = -s * gj;
    gd->g[j + 1] = r;
    gd->g[j] = c * gj;
    gd->sc[j + 1] = h > 0 ? 1.0 / h : 1.0;
    gd->its += 1;
    gd->jend = j;
    bool go = true;
    if (!isfinite(r)) go = false;
    else if (fabs(r) <= gd->tol) { gd->converged = 1; go = false; }
    const bool more = go && last_step && ctl;
    if (more) raise_gate(ctl, ERR_SWEEPS, CN_SHORT);
    if (go && last_step) go = false;
    gd->go = go ? 1 : 0;
    gd->ticket = 0;
    stop = !go && !more;
  }
  __syncwarp();
  if (lane <= j) gd->H[lane * CN_M + j] = hc[lane];
  __syncwarp();
  if (!stop) return;
  // y = R^-1 g (lane i keeps g_i), as coefficients of the unscaled basis
  double gi = lane <= j ? gd->g[lane] : 0.0;
  for (int k = j; k >= 0; --k) {
    const double hik = lane <= k ? gd->H[lane * CN_M + k] : 1.0;
    const double yk = __shfl_sync(0xffffffffu, gi / hik, k);
    if (lane < k) gi -= hik * yk;
    else if (lane == k) gd->coef[k] = yk * gd->sc[k];
  }
  if (lane == 0) gd->nv = nv;
}

// x += V coef
__global__ void k_cn_combine(const double* __restrict__ V, int64_t n, const CnDev* __restrict__ gd, double* __restrict__ x) {
  const int nv = gd->nv;
  if (nv == 0) return;
  __shared__ double cf[CN_M];
  if (threadIdx.x < nv) cf[threadIdx.x] = gd->coef[threadIdx.x];
  __syncthreads();
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    double a = 0.0;
#pragma unroll 4
    for (int i = 0; i < nv; ++i) a += cf[i] * V[(int64_t)i * n + t];
    x[t] += a;
  }
}
// the next restart cycle runs while not converged, a step was taken and fewer than 100 cycles ran
__global__ void k_cn_cycle(CnDev* gd, cudaGraphConditionalHandle cycle) {
  const bool go = gd->jend >= 0 && !gd->converged && ++gd->cycle < 100;
  cudaGraphSetConditional(cycle, go ? 1u : 0u);
}

template <int NV>
void cn_arnoldi_nv(const CcGeo& g, const CnOp& L, double* V, int nv, const CnH& h, double* part1, double* part2, CnDev* gd,
                   int last_step, StepCtl* ctl, cudaStream_t st) {
  double* w = V + (int64_t)nv * g.F;
  counted();
  launch_pdl_ext(k_cn_apply<NV>, dim3(CN_BLOCKS), dim3(CN_THREADS), 0, st, g, L, V, nv, h, w, part1, gd);
  counted();
  launch_pdl_ext(k_cn_pass<NV, false>, dim3(CN_BLOCKS), dim3(CN_THREADS), 0, st, V, g.F, nv, part1, w, part2, gd, 0, nullptr);
  counted();
  launch_pdl_ext(k_cn_pass<NV, true>, dim3(CN_BLOCKS), dim3(CN_THREADS), 0, st, V, g.F, nv, part2, w, part1, gd, last_step, ctl);
}
// Arnoldi step nv - 1.  Up to eight basis vectors the kernels keep a face's values in registers; beyond
// (steps that few systems reach) the size is rounded up and the vectors are read again.
void cn_arnoldi(const CcGeo& g, const CnOp& L, double* V, int nv, const CnH& h, double* part1, double* part2, CnDev* gd,
                int last_step, StepCtl* ctl, cudaStream_t st) {
#define CN_CASE(K) if (nv <= K) return cn_arnoldi_nv<K>(g, L, V, nv, h, part1, part2, gd, last_step, ctl, st)
  CN_CASE(1); CN_CASE(2); CN_CASE(3); CN_CASE(4); CN_CASE(5); CN_CASE(6); CN_CASE(7); CN_CASE(8);
  CN_CASE(12); CN_CASE(20); CN_CASE(CN_M);
#undef CN_CASE
}

// ---- the end of a step ------------------------------------------------------------------------
// Pressure (half = p + inc, next = half + factor inc), unpacked velocity, advection history, the
// coupled residual max |(H q - rhs) + dt grad inc| and the gate quantities of solver/main.py:416-424
// (max_fluid |flux divergence| / kappa, max |u|, max |v|) in one pass; nothing is written when a solve
// ran out of its graph's sweeps or Arnoldi steps (the host repeats the step).
struct CcEnd {
  const double *q, *inl, *now, *action, *rhs, *p, *inc;
  double factor, dt, gx, gy;
  double *U, *prev_adv, *half, *P;
  const int* err;
  CcDiagDev* d;
};
__global__ void k_cc_step_end(CcGeo g, CcEnd e) {
  if (*e.err == ERR_SWEEPS) return;
  const int nx = g.nx;
  MaxBits dm = 0, um = 0, vm = 0, cm = 0;
  for (int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; f < g.F; f += (int64_t)gridDim.x * blockDim.x) {
    const bool isu = f < g.usize;
    const auto [fj, fi] = row_col(isu ? f : f - g.usize, isu ? nx + 1 : nx);
    const bool act = (g.flags[f] & F_ACTIVE) != 0;
    const double u = isu && fi == 0 ? e.inl[fj] : act ? e.q[f] : 0.0;
    e.U[f] = u;
    if (isu) um = max_abs(um, u);
    else vm = max_abs(vm, u);
    e.prev_adv[f] = e.now[f];
    // (face_grad of inc)
    double gp = 0.0;
    if (act) {
      const int64_t c = isu ? (int64_t)fj * nx + fi : f - g.usize;
      if (isu) gp = fi == 0 ? 0.0 : fi < nx ? (e.inc[c] - e.inc[c - 1]) * e.gx : -2.0 * e.inc[c - 1] * e.gx;
      else if (fj >= 1 && fj < g.ny) gp = (e.inc[c] - e.inc[c - nx]) * e.gy;
    }
    cm = max_abs(cm, (e.action[f] - e.rhs[f]) + e.dt * gp);
    // the cell east of a u face: this thread has its west face, the packed field the others
    if (isu && fi < nx) {
      const int64_t c = (int64_t)fj * nx + fi, fv = g.usize + c;
      if (g.cell_type[c] != -1) {
        auto val = [&](int64_t t) { return (g.flags[t] & F_ACTIVE) ? e.q[t] : 0.0; };
        const double d = (g.ax[f + 1] * val(f + 1) - g.ax[f] * u) * g.idx + (g.ay[c + nx] * val(fv + nx) - g.ay[c] * val(fv)) * g.idy;
        dm = max_abs(dm, d * g.ikappa[c]);
      }
      const double inc = e.inc[c], h = e.p[c] + inc;
      e.half[c] = h;
      e.P[c] = h + e.factor * inc;
    }
  }
  block_commit_max(cm, &e.d->coupled);
  block_commit_max(dm, &e.d->divmax);
  block_commit_max(um, &e.d->umax);
  block_commit_max(vm, &e.d->vmax);
}

}  // namespace

// =============================================================================================
// handle
// =============================================================================================
struct gm_cc {
  std::string err;
  gm_handle* P = nullptr;  // pressure-only handle (stream, Poisson inverse, control block)
  cudaStream_t st = nullptr;
  int nx = 0, ny = 0;
  int64_t usize = 0, vsize = 0, psize = 0, F = 0;
  double dx = 0, dy = 0, rho = 1, nu = 0, D = 1, U_ref = 1;
  int slip = 0;
  int64_t n_active = 0;
  std::vector<int64_t> act_idx;  // face-grid flat indices of the unknowns (packed order)
  // geometry on the device
  Buf<double> ax, ay, kappa, ikappa, vol_rho, mvol_rho, inlet;
  Buf<double> cxx, cyy, cxy, cyx, axx, ayy, axy, ayx, aout;
  Buf<uint8_t> flags;
  Buf<int32_t> cell_type, merge_of;
  Buf<int64_t> ms, mm, d_act;
  // overrides
  Buf<uint8_t> dfam, afam;
  Buf<int64_t> dface, dptr, dcol, aface, apptr, uptr, ucol, vptr, vcol;
  Buf<double> dval, uval, vval, alen;
  // wall and transfers
  Buf<int64_t> wptr, wcol, tgt, tptr, own, optr, odon, don;
  Buf<int32_t> tk, aux_tgt, aux_own;
  Buf<int64_t> aux_face;
  Buf<uint8_t> aux_don;
  Buf<double> wval, wtx, wty, wds, tau;
  CcGeo geo{};
  CcFix fix{};
  CcWall wall{};
  // state: U (unpacked face grid), P; history
  Buf<double> U, Pst, prev_adv, halfp;
  bool has_history = false;
  double prev_dt = 0;
  // work vectors (face grid) and pressure-grid work
  Buf<double> q0, now, mid, halfq, expl, offset, rhs, star, w, result, action, tmp, zero;
  Buf<double> fxx, fxy, fyx, fyy;
  Buf<double> B, phi, inc, pb, io_f, io_p;
  // the legacy predictor: advective and viscous accelerations, scratch, previous acceleration,
  // predicted field, residual-norm partials; its history
  Buf<double> la, ld, lr, lprev, lstar, lres;
  Buf<double> ftau;  // the wall shear of the forces, per Gauss point
  bool l_has_prev = false;
  double l_prev_dt = 0;
  CcFlux flux{};
  // the CN operator on packed vectors and its GMRES(30)
  Buf<uint8_t> ncls;
  Buf<int32_t> nface, ncol;
  Buf<int64_t> nptr;
  Buf<double> nval;
  CnOp cn{};
  bool offset_stale = true;  // the inlet changed since offset was formed
  HeldCount arnoldi{6, 1};   // Arnoldi steps that a step graph holds; above CN_M: restart cycles in a WHILE node
  bool counts_known = false; // a first step, which holds plenty, has set them and the pressure solves' sweeps
  long long repeats = 0;     // steps repeated for a refinement sweep or Arnoldi steps more
  Buf<double> V, gpart, gpart2;
  Buf<CnDev> gdev;
  // per-step diagnostics
  Buf<CcDiagDev> diag;
  CcDiagDev* host_diag = nullptr;
  // step graphs keyed by (dt, history, previous dt) and what they hold
  struct Graph {
    cudaGraphExec_t exec = nullptr;
    double dt = 0, prev_dt = 0;
    bool hist = false;
    std::array<int, 5> sweeps{};
    int arnoldi = 0;
    long long outer = 0, per_cycle = 0;
  };
  Graph graphs[3];
  int next_graph = 0;
  // optional phase events inside the step graph (environment GHOSTMAC_PHASE_TIMING=1 at create)
  static constexpr int NPHASE = 8;
  bool phase_on = false;
  cudaEvent_t pev[NPHASE + 1] = {};
  double phase_ms[NPHASE] = {};
};

namespace {

int guarded(gm_cc* c, const std::function<void()>& f) {
  try {
    f();
    return GM_OK;
  } catch (const CcFail& e) {
    if (c) c->err = e.msg;
    else gm_internal_set_error(e.msg.c_str());
    return e.cls;
  } catch (const std::exception& e) {
    if (c) c->err = e.what();
    else gm_internal_set_error(e.what());
    return GM_ECUDA;
  }
}

// copies n doubles from a host or device pointer into a device buffer
void copy_in(double* dst, const double* src, size_t n, cudaStream_t st) {
  CCK(cudaMemcpyAsync(dst, src, n * sizeof(double), cudaMemcpyDefault, st));
}

// ---- momentum evaluation (three launches) ---------------------------------------------------
void momentum(gm_cc* c, bool adv, const double* X, const double* inl, double nu, int mode, double hdt, double* Y,
              double* Rout, cudaStream_t st, bool upwind = false) {
  const double rnu = c->rho * nu;
  const int64_t nv = (int64_t)(c->ny + 1) * (c->nx + 1);
  const bool shear = !adv && nu != 0.0;
  counted();
  if (adv && upwind) k_cc_flux<true, true><<<nblk(nv), CC_TPB, 0, st>>>(c->geo, X, inl, rnu, c->slip, c->flux);
  else if (adv) k_cc_flux<true><<<nblk(nv), CC_TPB, 0, st>>>(c->geo, X, inl, rnu, c->slip, c->flux);
  else k_cc_flux<false><<<nblk(nv), CC_TPB, 0, st>>>(c->geo, X, inl, rnu, c->slip, c->flux);
  const int nrows = adv ? c->fix.n_adv : c->fix.n_dif + (shear ? c->wall.n : 0);
  if (nrows > 0) {
    counted();
    const unsigned nb = nblk((int64_t)nrows * 32, 256);
    if (adv) k_cc_fix<true><<<nb, 256, 0, st>>>(c->geo, c->fix, c->wall, X, inl, rnu, c->rho, 0.0, c->flux);
    else k_cc_fix<false><<<nb, 256, 0, st>>>(c->geo, c->fix, c->wall, X, inl, rnu, c->rho, (-c->rho) * nu, c->flux);
  }
  counted();
  if (adv) k_cc_rhs<true><<<nblk(c->F), CC_TPB, 0, st>>>(c->geo, c->flux, c->wall, X, 0, hdt, mode, Y, Rout);
  else k_cc_rhs<false><<<nblk(c->F), CC_TPB, 0, st>>>(c->geo, c->flux, c->wall, X, shear ? 1 : 0, hdt, mode, Y, Rout);
}

// project(q, step) of advance_ab2_cn (solver/cut_cell_solver.py:993-1002): q -> out (packed),
// phi; slot selects the control block entry and the predicted-divergence record
void project(gm_cc* c, const double* q, double step, double* out, double* phi, int slot, int rec, cudaStream_t st) {
  counted();
  k_cc_divrhs<<<nblk(c->psize), CC_TPB, 0, st>>>(c->geo, q, c->inlet.p, c->rho / step, c->B.p);
  gmi::pressure_solve(c->P, c->B.p, phi, slot);
  counted();
  k_cc_correct<<<std::min<unsigned>(nblk(c->F), 1216), CC_TPB, 0, st>>>(
      c->geo, q, phi, (step / c->rho) / c->dx, (step / c->rho) / c->dy, out, gmi::pressure_residual(c->P), step / c->rho,
      &c->diag.p->pdiv[rec]);
}

// forces on the circle into diag->forces: the wall shear and pressure of every point (one warp each),
// then the one-block sums
void forces(gm_cc* c, const double* U, const double* P, double mu, cudaStream_t st) {
  const gmi::SurfaceCsr S = gmi::surface(c->P);
  if (c->wall.n + S.n > 0) {
    counted();
    k_cc_wall_points<<<nblk((int64_t)(c->wall.n + S.n) * 32, 256), 256, 0, st>>>(S, c->wall, U, P, mu, c->ftau.p, c->pb.p);
  }
  counted();
  k_cc_forces<<<1, CC_FORCE_THREADS, 0, st>>>(S, c->wall, c->ftau.p, c->pb.p, c->diag.p->forces);
}

template <int MODE>
void cn_eval(gm_cc* c, CnEval e, cudaStream_t st) {
  e.offset = c->offset.p;
  e.h = cn_h(c->cn, e.hdt);
  e.gx = 1.0 / (c->rho * c->dx);
  e.gy = 1.0 / (c->rho * c->dy);
  counted();
  k_cn_eval<MODE><<<std::max(4u, std::min<unsigned>(nblk(c->F), 1216)), CC_TPB, 0, st>>>(c->geo, c->cn, e);
}
// the inlet's part of the viscous operator, by the flux arrays (mode 0 of momentum on the zero vector)
void refresh_offset(gm_cc* c) {
  if (!c->offset_stale) return;
  momentum(c, false, c->zero.p, c->inlet.p, c->nu, 0, 0.0, c->offset.p, nullptr, c->st);
  c->offset_stale = false;
}

cudaGraphNode_t add_cond(cudaStream_t st, cudaGraphConditionalHandle cond, cudaGraphConditionalNodeType type,
                         cudaGraph_t* body) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t graph;
  const cudaGraphNode_t* deps = nullptr;
  size_t nd = 0;
  CCK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &graph, &deps, nullptr, &nd));
  cudaGraphNodeParams cp{};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = cond;
  cp.conditional.type = type;
  cp.conditional.size = 1;
  cudaGraphNode_t node;
  CCK(cudaGraphAddNode(&node, graph, deps, nullptr, nd, &cp));
  *body = cp.conditional.phGraph_out[0];
  CCK(cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
  return node;
}

// the CN solve (see k_cn_start), captured on st: x holds the first iterate and the solution
void gmres(gm_cc* c, const double* b, double* x, double dt, gm_cc::Graph& gr, cudaStream_t st) {
  const CnH h = cn_h(c->cn, 0.5 * dt);
  auto cycle = [&](int first, int steps, StepCtl* ctl, cudaStream_t s) {
    counted();
    k_cn_start<<<CN_BLOCKS, CN_THREADS, 0, s>>>(c->geo, c->cn, x, h, b, c->V.p, c->gpart.p, c->gdev.p, first);
    for (int nv = 1; nv <= steps; ++nv)
      cn_arnoldi(c->geo, c->cn, c->V.p, nv, h, c->gpart.p, c->gpart2.p, c->gdev.p, nv == steps, ctl, s);
    counted();
    k_cn_combine<<<std::min<unsigned>(nblk(c->F), 1216), CC_TPB, 0, s>>>(c->V.p, c->F, c->gdev.p, x);
  };
  if (c->arnoldi.n <= CN_M) {
    cycle(1, c->arnoldi.n, gmi::control(c->P), st);
    return;
  }
  CCK(cudaMemsetAsync(&c->gdev.p->jend, 0, sizeof(CnDev) - offsetof(CnDev, jend), st));
  cudaStreamCaptureStatus cs;
  cudaGraph_t top;
  CCK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &top, nullptr, nullptr, nullptr));
  cudaGraphConditionalHandle cyc;
  CCK(cudaGraphConditionalHandleCreate(&cyc, top, 1, cudaGraphCondAssignDefault));
  cudaGraph_t body;
  add_cond(st, cyc, cudaGraphCondTypeWhile, &body);
  cudaStream_t sb = gmi::body_stream(c->P, 0);
  CCK(cudaStreamBeginCaptureToGraph(sb, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  const long long c1 = kernel_launch_count();
  cycle(0, CN_M, nullptr, sb);
  counted();
  k_cn_cycle<<<1, 1, 0, sb>>>(c->gdev.p, cyc);
  gr.per_cycle = kernel_launch_count() - c1;
  cudaGraph_t done;
  CCK(cudaStreamEndCapture(sb, &done));
}

// One AB2/CN step (advance_ab2_cn, solver/cut_cell_solver.py:959-1015, with ab2_cn_step,
// solver/time_integration.py:7-145), captured on st.
void step_body(gm_cc* c, double dt, gm_cc::Graph& gr, cudaStream_t st) {
  const double* inl = c->inlet.p;
  auto mark = [&](int k) {
    // inside a capture an event record node needs the external flag (a plain record only
    // orders the captured streams)
    if (c->phase_on) CCK(cudaEventRecordWithFlags(c->pev[k], st, cudaEventRecordExternal));
  };
  mark(0);
  CCK(cudaMemsetAsync(c->diag.p, 0, offsetof(CcDiagDev, forces), st));
  counted();
  k_cc_pack<<<nblk(c->F), CC_TPB, 0, st>>>(c->geo, c->U.p, c->q0.p);
  momentum(c, true, c->q0.p, inl, 0.0, 0, 0.0, c->now.p, nullptr, st);
  mark(1);
  const double* pressure = c->has_history ? c->halfp.p : c->Pst.p;
  CnEval e{};
  e.x = c->q0.p;
  e.p = pressure;
  e.hdt = 0.5 * dt;
  if (!c->has_history) {
    // projected midpoint start-up
    e.a = c->now.p;
    e.dt = 0.5 * dt;
    e.out = c->mid.p;
    cn_eval<CN_MID>(c, e, st);
    project(c, c->mid.p, 0.5 * dt, c->halfq.p, c->phi.p, S_P0, 0, st);
    momentum(c, true, c->halfq.p, inl, 0.0, 0, 0.0, c->expl.p, nullptr, st);
    e.a = c->expl.p;
  } else {
    e.a = c->now.p;
    e.b = c->prev_adv.p;
    e.s = dt / (2 * c->prev_dt);
  }
  e.dt = dt;
  e.out = c->rhs.p;
  e.out2 = c->star.p;
  e.mx = &c->diag.p->rhs_max;
  cn_eval<CN_RHS>(c, e, st);
  mark(2);
  gmres(c, c->rhs.p, c->star.p, dt, gr, st);
  mark(3);
  CnEval r{};
  r.x = c->star.p;
  r.a = c->rhs.p;
  r.hdt = 0.5 * dt;
  r.mx = &c->diag.p->mres;
  cn_eval<CN_CHECK>(c, r, st);
  mark(4);
  project(c, c->star.p, dt, c->result.p, c->phi.p, S_P1, 1, st);
  mark(5);
  r.x = c->result.p;
  r.out = c->action.p;
  r.out2 = c->tmp.p;
  cn_eval<CN_ACTION>(c, r, st);
  mark(6);
  project(c, c->tmp.p, dt, c->w.p, c->inc.p, S_P2, 2, st);
  mark(7);
  CcEnd n{c->result.p, inl, c->now.p, c->action.p, c->rhs.p, pressure, c->inc.p,
          c->has_history ? dt / (dt + c->prev_dt) : 1.0, dt, 1.0 / (c->rho * c->dx), 1.0 / (c->rho * c->dy),
          c->U.p, c->prev_adv.p, c->halfp.p, c->Pst.p, &gmi::control(c->P)->err, c->diag.p};
  counted();
  k_cc_step_end<<<std::min<unsigned>(nblk(c->F), 1216), CC_TPB, 0, st>>>(c->geo, n);
  forces(c, c->U.p, c->Pst.p, c->nu * c->rho, st);
  mark(8);
}

gm_cc::Graph& step_graph(gm_cc* c, double dt) {
  const std::array<int, 5> sweeps = gmi::held_sweeps(c->P);
  for (auto& g : c->graphs)
    if (g.exec && g.dt == dt && g.hist == c->has_history && (!g.hist || g.prev_dt == c->prev_dt) && g.sweeps == sweeps &&
        g.arnoldi == c->arnoldi.n)
      return g;
  gm_cc::Graph& gr = c->graphs[c->next_graph];
  c->next_graph = (c->next_graph + 1) % 3;
  if (gr.exec) { cudaGraphExecDestroy(gr.exec); gr.exec = nullptr; }
  gr.per_cycle = 0;
  cudaStream_t st = c->st;
  const long long c0 = kernel_launch_count();
  gmi::hold_sweeps(c->P, true);
  cudaGraph_t g = nullptr;
  CCK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  try {
    step_body(c, dt, gr, st);
  } catch (...) {
    gmi::hold_sweeps(c->P, false);
    cudaStreamEndCapture(st, &g);
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    throw;
  }
  gmi::hold_sweeps(c->P, false);
  CCK(cudaStreamEndCapture(st, &g));
  const long long captured = kernel_launch_count() - c0;
  kernel_launch_adjust(-captured);
  gr.outer = captured - gr.per_cycle;
  cudaGraphExec_t ex = nullptr;
  cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) throw CcFail(GM_ECUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
  gr.exec = ex;
  gr.dt = dt;
  gr.hist = c->has_history;
  gr.prev_dt = c->prev_dt;
  gr.sweeps = sweeps;
  gr.arnoldi = c->arnoldi.n;
  return gr;
}

// One step of the legacy cut-cell loop (solver/main.py:297-333, boundary='cut_cell',
// time_scheme='legacy'): the predictor on the stored state (its inlet column is the previous
// step's), compute_rhs / solve_pressure / apply_corrector (the projection of the AB2/CN path),
// p = phi, the step maxima and the forces on the true circle.
void legacy_body(gm_cc* c, double dt, bool centered, cudaStream_t st) {
  const int64_t F = c->F;
  CCK(cudaMemsetAsync(c->diag.p, 0, sizeof(CcDiagDev), st));
  momentum(c, true, c->U.p, nullptr, 0.0, 2, 0.0, c->la.p, c->lr.p, st, !centered);
  momentum(c, false, c->U.p, nullptr, c->nu, 2, 0.0, c->ld.p, c->lr.p, st);
  const bool ab2 = centered && c->l_has_prev;
  counted();
  k_cc_legacy_pred<<<nblk(F), CC_TPB, 0, st>>>(c->geo, c->U.p, c->la.p, c->ld.p, c->lprev.p, c->inlet.p, dt,
                                               ab2 ? dt / (2 * c->l_prev_dt) : 0.0, ab2 ? 1 : 0, c->lstar.p);
  project(c, c->lstar.p, dt, c->w.p, c->Pst.p, S_P1, 1, st);
  counted();
  k_cc_resnorm_part<<<CC_RES_BLOCKS, CC_TPB, 0, st>>>(c->geo, gmi::pressure_residual(c->P), c->lres.p);
  counted();
  k_cc_resnorm_fold<<<1, CC_TPB, 0, st>>>(c->lres.p, CC_RES_BLOCKS, &c->diag.p->res_linf, &c->diag.p->res_l2);
  counted();
  k_cc_unpack<<<nblk(F), CC_TPB, 0, st>>>(c->geo, c->w.p, c->inlet.p, c->U.p);
  counted();
  k_cc_stepmax<<<std::min<unsigned>(nblk(F), 1216), CC_TPB, 0, st>>>(c->geo, c->U.p, &c->diag.p->divmax,
                                                                      &c->diag.p->umax, &c->diag.p->vmax);
  forces(c, c->U.p, c->Pst.p, c->nu * c->rho, st);
}

double bits_to_double(unsigned long long b) {
  double d;
  std::memcpy(&d, &b, sizeof d);
  return d;
}

// the initial state of solver/main.py:166-177 and its projection (:236-240)
void initial_state(gm_cc* c, const std::vector<double>& inlet, const int32_t* cell_type, const double* ax,
                   const double* ay) {
  const int nx = c->nx, ny = c->ny;
  std::vector<double> U(c->F, 0.0);
  for (int j = 0; j < ny; ++j)
    for (int i = 0; i <= nx; ++i) U[(size_t)j * (nx + 1) + i] = inlet[j];
  for (int j = 0; j < ny; ++j)
    for (int i = 0; i < nx; ++i)
      if (cell_type[(size_t)j * nx + i] == -1) {
        U[(size_t)j * (nx + 1) + i] = 0.0;
        U[(size_t)j * (nx + 1) + i + 1] = 0.0;
        U[c->usize + (size_t)j * nx + i] = 0.0;
        U[c->usize + (size_t)(j + 1) * nx + i] = 0.0;
      }
  for (int64_t f = 0; f < c->usize; ++f)
    if (ax[f] == 0.0) U[f] = 0.0;
  for (int64_t f = 0; f < c->vsize; ++f)
    if (ay[f] == 0.0) U[c->usize + f] = 0.0;
  cudaStream_t st = c->st;
  CCK(cudaMemcpyAsync(c->U.p, U.data(), U.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  // compute_rhs(u, v, 1, rho); solve; apply_corrector(u, v, u, v, phi, 1, rho, inlet): the
  // corrector reads the unpacked field (inlet column included)
  CCK(cudaMemsetAsync(c->diag.p, 0, sizeof(CcDiagDev), st));
  CCK(cudaMemsetAsync(gmi::control(c->P), 0, sizeof(StepCtl), st));
  counted();
  k_cc_divrhs<<<nblk(c->psize), CC_TPB, 0, st>>>(c->geo, c->U.p, nullptr, c->rho / 1.0, c->B.p);
  gmi::pressure_solve(c->P, c->B.p, c->phi.p, S_P1);
  counted();
  k_cc_pdiv<<<std::min<unsigned>(nblk(c->psize), 1216), CC_TPB, 0, st>>>(c->geo, gmi::pressure_residual(c->P),
                                                                        1.0 / c->rho, &c->diag.p->pdiv[1]);
  counted();
  k_cc_correct<<<nblk(c->F), CC_TPB, 0, st>>>(c->geo, c->U.p, c->phi.p, (1.0 / c->rho) / c->dx, (1.0 / c->rho) / c->dy,
                                             c->tmp.p, nullptr, 0.0, nullptr);
  counted();
  k_cc_unpack<<<nblk(c->F), CC_TPB, 0, st>>>(c->geo, c->tmp.p, c->inlet.p, c->U.p);
  CCK(cudaMemsetAsync(c->Pst.p, 0, c->psize * sizeof(double), st));
  std::string m;
  int rc = gmi::check(c->P, "initial projection", m);
  if (rc != GM_OK) throw CcFail(rc, m);
  CCK(cudaMemcpyAsync(c->host_diag, c->diag.p, sizeof(CcDiagDev), cudaMemcpyDeviceToHost, st));
  CCK(cudaStreamSynchronize(st));
  const double pd = bits_to_double(c->host_diag->pdiv[1]);
  if (!(pd < 1e-10))
    {
      char pbuf[96];
      std::snprintf(pbuf, sizeof pbuf, "Pressure residual exceeds divergence budget: %g", pd);
      throw CcFail(GM_ERUNTIME, pbuf);
    }
}

// Tables of the CN operator (CnOp): the class of every face, and the sparse rows of L = (viscous
// acceleration) of the unknown faces near the body -- those with a curved flux among their four, wall
// shear, covered transfers or a merge -- composed from the same pieces in the order of k_cc_fix and k_cc_rhs.
// Columns that are not unknown hold zero in packed vectors and are left out.
void build_cn(gm_cc* C, const gm_cc_config* cfg, const std::vector<uint8_t>& fl, const std::vector<double>& vr,
              const std::vector<int32_t>& mof, const std::vector<int64_t>& ms, const std::vector<int64_t>& mm,
              const std::vector<double>& mv, const std::vector<int64_t>& tgt, const std::vector<int64_t>& tptr,
              const std::vector<int32_t>& tk, const std::vector<int64_t>& own, const std::vector<int64_t>& optr,
              const std::vector<int64_t>& odon, const std::vector<int64_t>& donors, const std::vector<uint8_t>& dfam,
              const std::vector<int64_t>& dface, const std::vector<int64_t>& dptr, const std::vector<int64_t>& dcol,
              const std::vector<double>& dval) {
  const int nx = C->nx, ny = C->ny, nu1 = nx + 1;
  const int64_t us = C->usize, F = C->F;
  const double dx = C->dx, dy = C->dy, rnu = C->rho * C->nu;
  using Row = std::map<int64_t, double>;
  std::array<std::map<int64_t, int64_t>, 4> over;  // curved faces of each family: row of the tables
  for (size_t r = 0; r < dface.size(); ++r) over[dfam[r]][dface[r]] = (int64_t)r;
  std::map<int64_t, int64_t> tof, oof, don;
  for (size_t t = 0; t < tgt.size(); ++t) tof[tgt[t]] = (int64_t)t;
  for (size_t o = 0; o < own.size(); ++o) oof[own[o]] = (int64_t)o;
  for (int64_t d : donors) don[d] = 1;
  const double dydx = dy / dx, dxdy = dx / dy;
  // flux `idx` of a family (0 F_xx, 1 F_xy, 2 F_yx, 3 F_yy) times s, added to a row
  auto flux = [&](int fam, int64_t idx, double s, Row& row) {
    auto it = over[fam].find(idx);
    if (it != over[fam].end()) {
      for (int64_t e = dptr[it->second]; e < dptr[it->second + 1]; ++e) row[dcol[e]] += s * (rnu * dval[e]);
      return;
    }
    auto u = [&](int j, int i, double w) { row[(int64_t)j * nu1 + i] += s * w; };
    auto v = [&](int j, int i, double w) { row[us + (int64_t)j * nx + i] += s * w; };
    if (fam == 0 || fam == 3) {
      const int j = (int)(idx / nx), i = (int)(idx % nx);
      if (fam == 0) {
        const double w = rnu * (cfg->ax_mid[idx] * dydx);
        u(j, i + 1, w); u(j, i, -w);
      } else {
        const double w = rnu * (cfg->ay_mid[idx] * dxdy);
        v(j + 1, i, w); v(j, i, -w);
      }
      return;
    }
    const int j = (int)(idx / nu1), i = (int)(idx % nu1);
    if (fam == 1) {
      const double w = rnu * (cfg->ay_u[idx] * dxdy);
      if (j == 0) { if (!C->slip) u(0, i, 2.0 * w); }
      else if (j == ny) { if (!C->slip) u(ny - 1, i, -2.0 * w); }
      else { u(j, i, w); u(j - 1, i, -w); }
    } else {
      const double w = rnu * (cfg->ax_v[idx] * dydx);
      if (i == 0) v(j, 0, 2.0 * w);
      else if (i < nx) { v(j, i, w); v(j, i - 1, -w); }
    }
  };
  // the four fluxes of face f (family, index, sign), none on the faces without a flux balance
  struct Part { int fam; int64_t idx; double s; };
  auto parts = [&](int64_t f) {
    std::vector<Part> p;
    if (f < us) {
      const int j = (int)(f / nu1), i = (int)(f % nu1);
      const int64_t c = (int64_t)j * nx + i;
      if (i >= 1 && i < nx) p = {{0, c, 1.0}, {0, c - 1, -1.0}, {1, f + nu1, 1.0}, {1, f, -1.0}};
      else if (i == nx) p = {{0, c - 1, -1.0}, {1, f + nu1, 0.5}, {1, f, -0.5}};
    } else {
      const int64_t c = f - us;
      const int j = (int)(c / nx), i = (int)(c % nx);
      const int64_t t = (int64_t)j * nu1 + i;
      if (j >= 1 && j < ny) p = {{2, t + 1, 1.0}, {2, t, -1.0}, {3, c, 1.0}, {3, c - nx, -1.0}};
    }
    return p;
  };
  auto walled = [&](int64_t f, double s, Row& row) {
    for (const Part& p : parts(f)) flux(p.fam, p.idx, s * p.s, row);
    auto t = tof.find(f);
    if (t == tof.end() || rnu == 0.0) return;
    for (int64_t q = tptr[t->second]; q < tptr[t->second + 1]; ++q) {
      const int k = tk[q];
      const double w = s * (-rnu) * (f < us ? cfg->wall_tx[k] : cfg->wall_ty[k]) * cfg->wall_ds[k];
      for (int64_t e = cfg->wall_rate.ptr[k]; e < cfg->wall_rate.ptr[k + 1]; ++e)
        row[cfg->wall_rate.col[e]] += w * cfg->wall_rate.val[e];
    }
  };
  auto full = [&](int64_t f, double s, Row& row) {
    if (don.count(f)) return;
    walled(f, s, row);
    auto o = oof.find(f);
    if (o != oof.end())
      for (int64_t q = optr[o->second]; q < optr[o->second + 1]; ++q) walled(odon[q], s, row);
  };
  std::vector<uint8_t> cls(F, CN_ZERO);
  std::vector<int32_t> face, col;
  std::vector<int64_t> ptr{0};
  std::vector<double> val;
  const double iv = 1.0 / (C->rho * dx * dy);
  for (int64_t f = 0; f < F; ++f) {
    if (!(fl[f] & F_ACTIVE)) continue;
    const std::vector<Part> ps = parts(f);
    bool row = mof[f] >= 0 || (fl[f] & F_AUX), reg = (fl[f] & F_FLUID) && !(fl[f] & F_SOLID) && ps.size() == 4;
    for (const Part& p : ps) {
      row = row || over[p.fam].count(p.idx);
      const double a = p.fam == 0 ? cfg->ax_mid[p.idx] : p.fam == 1 ? cfg->ay_u[p.idx] : p.fam == 2 ? cfg->ax_v[p.idx] : cfg->ay_mid[p.idx];
      reg = reg && a == 1.0;
    }
    if (row) {
      cls[f] = CN_ROW;
      Row r;
      if (fl[f] & F_SOLID) {}
      else if (mof[f] >= 0) {
        full(ms[mof[f]], mv[mof[f]], r);
        full(mm[mof[f]], mv[mof[f]], r);
      } else if (fl[f] & F_FLUID) full(f, vr[f], r);
      face.push_back((int32_t)f);
      for (const auto& kv : r)
        if (fl[kv.first] & F_ACTIVE) {
          col.push_back((int32_t)kv.first);
          val.push_back(kv.second);
        }
      ptr.push_back((int64_t)col.size());
      continue;
    }
    // regular: full apertures and volume, all four fluxes between two faces of its own grid
    if (f < us) {
      const int j = (int)(f / nu1);
      reg = reg && j >= 1 && j + 1 < ny;
    } else {
      const int i = (int)((f - us) % nx);
      reg = reg && i >= 1 && i + 1 < nx;
    }
    reg = reg && std::fabs(vr[f] / iv - 1.0) <= 1e-15;
    cls[f] = reg ? CN_REGULAR : CN_EDGE;
  }
  cudaStream_t st = C->st;
  C->ncls.upload(cls, st);
  C->nface.upload(face, st);
  C->nptr.upload(ptr, st);
  C->ncol.upload(col, st);
  C->nval.upload(val, st);
  CCK(cudaStreamSynchronize(st));
  C->cn = CnOp{C->ncls.p, (int)face.size(), C->nface.p, C->nptr.p, C->ncol.p, C->nval.p,
               rnu * dydx * iv, rnu * dxdy * iv, rnu, C->slip};
}

template <typename T>
std::vector<T> vec_of(const T* p, size_t n) {
  return p ? std::vector<T>(p, p + n) : std::vector<T>();
}

}  // namespace

// =============================================================================================
// C ABI
// =============================================================================================
extern "C" {

const char* gm_cc_last_error(const gm_cc* c) { return c ? c->err.c_str() : gm_last_error(nullptr); }

int gm_cc_create(const gm_cc_config* cfg, gm_cc** out) {
  if (!cfg || !out) { gm_internal_set_error("null argument"); return GM_EVALUE; }
  *out = nullptr;
  if (!cfg->ax || !cfg->ay || !cfg->ax_mid || !cfg->ay_mid || !cfg->ay_u || !cfg->ax_v || !cfg->cell_type ||
      !cfg->volume_fraction || !cfg->u_volume_fraction || !cfg->v_volume_fraction || !cfg->u_vol || !cfg->v_vol ||
      !cfg->u_vol_eff || !cfg->v_vol_eff) {
    gm_internal_set_error("missing geometry array");
    return GM_EVALUE;
  }
  auto c = std::make_unique<gm_cc>();
  gm_cc* C = c.get();
  const int nx = cfg->nx, ny = cfg->ny;
  gm::Geometry g;
  g.nx = nx; g.ny = ny; g.Lx = cfg->Lx; g.Ly = cfg->Ly; g.D = cfg->D; g.xc = cfg->xc; g.yc = cfg->yc;
  g.nu = cfg->nu; g.rho = cfg->rho; g.U_inf = cfg->U_inf; g.inflow = cfg->inflow; g.U_m = cfg->U_m;
  int ec = 0;
  if (!gm::build_cutcell_geometry(g, cfg->ax, cfg->ay, cfg->cell_type, cfg->volume_fraction, ec)) {
    gm_internal_set_error(g.error.c_str());
    return ec ? ec : GM_EVALUE;
  }
  C->nx = nx; C->ny = ny;
  C->usize = g.usize; C->vsize = g.vsize; C->psize = g.psize; C->F = g.usize + g.vsize;
  C->dx = g.dx; C->dy = g.dy; C->rho = cfg->rho; C->nu = cfg->nu; C->D = cfg->D; C->U_ref = g.U_ref;
  C->slip = cfg->slip_walls ? 1 : 0;
  std::vector<double> inlet = g.u_inlet;
  for (int64_t f : g.ui) C->act_idx.push_back(f);
  for (int64_t f : g.vi) C->act_idx.push_back(g.usize + f);
  C->n_active = (int64_t)C->act_idx.size();
  std::vector<uint8_t> act_u = g.act_u, act_v = g.act_v;
  std::string perr;
  int rc = gmi::pressure_create(std::move(g), &C->P, perr);
  if (rc != GM_OK) {
    gm_internal_set_error(perr.c_str());
    return rc;
  }
  rc = guarded(nullptr, [&] {
    cudaStream_t st = C->st = gmi::stream(C->P);
    const int64_t F = C->F, Pn = C->psize, us = C->usize;
    const int64_t nvert = (int64_t)(ny + 1) * (nx + 1);
    C->ax.upload(vec_of(cfg->ax, us), st);
    C->ay.upload(vec_of(cfg->ay, C->vsize), st);
    C->kappa.upload(vec_of(cfg->volume_fraction, Pn), st);
    {
      // folded factors of the structured kernels (see CcGeo)
      const double dx = C->dx, dy = C->dy, rho = cfg->rho;
      std::vector<double> cxx(Pn), cyy(Pn), axx(Pn), ayy(Pn), cxy(nvert), cyx(nvert), axy(nvert), ayx(nvert), aout(ny),
          ik(Pn);
      for (int64_t c = 0; c < Pn; ++c) {
        cxx[c] = cfg->ax_mid[c] * dy / dx;
        cyy[c] = cfg->ay_mid[c] * dx / dy;
        axx[c] = rho * cfg->ax_mid[c] * dy;
        ayy[c] = rho * cfg->ay_mid[c] * dx;
        ik[c] = cfg->cell_type[c] == 0 ? 1.0 / cfg->volume_fraction[c] : 1.0;
      }
      for (int64_t t = 0; t < nvert; ++t) {
        cxy[t] = cfg->ay_u[t] * dx / dy;
        cyx[t] = cfg->ax_v[t] * dy / dx;
        axy[t] = rho * cfg->ay_u[t] * dx;
        ayx[t] = rho * cfg->ax_v[t] * dy;
      }
      for (int j = 0; j < ny; ++j) aout[j] = rho * cfg->ax[(int64_t)j * (nx + 1) + nx] * dy;
      C->cxx.upload(cxx, st); C->cyy.upload(cyy, st); C->axx.upload(axx, st); C->ayy.upload(ayy, st);
      C->cxy.upload(cxy, st); C->cyx.upload(cyx, st); C->axy.upload(axy, st); C->ayx.upload(ayx, st);
      C->aout.upload(aout, st); C->ikappa.upload(ik, st);
    }
    C->cell_type.upload(vec_of(cfg->cell_type, Pn), st);
    C->inlet.upload(inlet, st);
    // face flags and volumes (fluid: fraction >= 0.3 and open; solid: covered face)
    std::vector<uint8_t> fl(F, 0);
    std::vector<double> vr(F, 1.0);
    for (int64_t f = 0; f < F; ++f) {
      const bool u = f < us;
      const int64_t k = u ? f : f - us;
      const double ap = u ? cfg->ax[k] : cfg->ay[k];
      const double fr = u ? cfg->u_volume_fraction[k] : cfg->v_volume_fraction[k];
      if (u ? act_u[k] : act_v[k]) fl[f] |= F_ACTIVE;
      if (fr >= 0.3 && ap > 0.0) fl[f] |= F_FLUID;
      if (ap == 0.0) fl[f] |= F_SOLID;
      vr[f] = 1.0 / (cfg->rho * (u ? cfg->u_vol[k] : cfg->v_vol[k]));
    }
    C->vol_rho.upload(vr, st);
    // merges in list order; a face written by several keeps the last
    std::vector<int32_t> mof(F, -1);
    std::vector<int64_t> ms, mm;
    std::vector<double> mv;
    auto add_merges = [&](int64_t n, const int64_t* tab, bool u) {
      const int64_t pitch = u ? nx + 1 : nx, off = u ? 0 : us;
      const double* eff = u ? cfg->u_vol_eff : cfg->v_vol_eff;
      for (int64_t k = 0; k < n; ++k) {
        const int64_t s = tab[4 * k] * pitch + tab[4 * k + 1], m = tab[4 * k + 2] * pitch + tab[4 * k + 3];
        const int32_t idx = (int32_t)ms.size();
        ms.push_back(off + s);
        mm.push_back(off + m);
        mv.push_back(1.0 / (cfg->rho * eff[s]));
        mof[off + s] = idx;
        mof[off + m] = idx;
      }
    };
    if (cfg->n_u_merge > 0 && !cfg->u_merge) throw CcFail(GM_EVALUE, "missing merge table");
    if (cfg->n_v_merge > 0 && !cfg->v_merge) throw CcFail(GM_EVALUE, "missing merge table");
    add_merges(cfg->n_u_merge, cfg->u_merge, true);
    add_merges(cfg->n_v_merge, cfg->v_merge, false);
    C->merge_of.upload(mof, st);
    C->ms.upload(ms, st);
    C->mm.upload(mm, st);
    C->mvol_rho.upload(mv, st);
    // covered-volume transfers: owners with their donors in order
    std::map<int64_t, std::vector<int64_t>> owners;
    std::vector<int64_t> donors;
    auto add_cov = [&](int64_t n, const int64_t* d, const int64_t* o, int64_t off) {
      for (int64_t k = 0; k < n; ++k) {
        owners[off + o[k]].push_back(off + d[k]);
        donors.push_back(off + d[k]);
      }
    };
    add_cov(cfg->n_u_covered, cfg->u_covered, cfg->u_owner, 0);
    add_cov(cfg->n_v_covered, cfg->v_covered, cfg->v_owner, us);
    std::vector<int64_t> own, optr{0}, odon;
    for (auto& kv : owners) {
      own.push_back(kv.first);
      odon.insert(odon.end(), kv.second.begin(), kv.second.end());
      optr.push_back((int64_t)odon.size());
    }
    C->own.upload(own, st);
    C->optr.upload(optr, st);
    C->odon.upload(odon, st);
    C->don.upload(donors, st);
    // wall: shear-rate rows, targets with their points in order
    const int64_t nw = cfg->n_wall;
    C->wptr.upload(vec_of(cfg->wall_rate.ptr, nw + 1), st);
    const int64_t wnnz = nw > 0 ? cfg->wall_rate.ptr[nw] : 0;
    C->wcol.upload(vec_of(cfg->wall_rate.col, wnnz), st);
    C->wval.upload(vec_of(cfg->wall_rate.val, wnnz), st);
    C->wtx.upload(vec_of(cfg->wall_tx, nw), st);
    C->wty.upload(vec_of(cfg->wall_ty, nw), st);
    C->wds.upload(vec_of(cfg->wall_ds, nw), st);
    C->tau.alloc(std::max<int64_t>(1, nw));
    std::map<int64_t, std::vector<int32_t>> targets;
    for (int64_t k = 0; k < nw; ++k) targets[cfg->wall_u[k]].push_back((int32_t)k);
    std::map<int64_t, std::vector<int32_t>> vtargets;
    for (int64_t k = 0; k < nw; ++k) vtargets[us + cfg->wall_v[k]].push_back((int32_t)k);
    std::vector<int64_t> tgt, tptr{0};
    std::vector<int32_t> tk;
    for (auto* mp : {&targets, &vtargets})
      for (auto& kv : *mp) {
        tgt.push_back(kv.first);
        tk.insert(tk.end(), kv.second.begin(), kv.second.end());
        tptr.push_back((int64_t)tk.size());
      }
    C->tgt.upload(tgt, st);
    C->tptr.upload(tptr, st);
    C->tk.upload(tk, st);
    // faces with wall shear, owners and donors: the sorted list the fused right-hand side
    // kernel searches (flag F_AUX)
    std::map<int64_t, std::array<int32_t, 3>> aux;  // face -> target entry, owner entry, donor
    for (size_t t = 0; t < tgt.size(); ++t) aux.emplace(tgt[t], std::array<int32_t, 3>{-1, -1, 0})
                                               .first->second[0] = (int32_t)t;
    for (size_t o = 0; o < own.size(); ++o) aux.emplace(own[o], std::array<int32_t, 3>{-1, -1, 0})
                                               .first->second[1] = (int32_t)o;
    for (int64_t d : donors) aux.emplace(d, std::array<int32_t, 3>{-1, -1, 0}).first->second[2] = 1;
    std::vector<int64_t> aux_face;
    std::vector<int32_t> aux_tgt, aux_own;
    std::vector<uint8_t> aux_don;
    for (auto& kv : aux) {
      aux_face.push_back(kv.first);
      aux_tgt.push_back(kv.second[0]);
      aux_own.push_back(kv.second[1]);
      aux_don.push_back((uint8_t)kv.second[2]);
      fl[kv.first] |= F_AUX;
    }
    C->flags.upload(fl, st);
    C->aux_face.upload(aux_face, st);
    C->aux_tgt.upload(aux_tgt, st);
    C->aux_own.upload(aux_own, st);
    C->aux_don.upload(aux_don, st);
    // curved-face overrides of the four families
    std::vector<uint8_t> dfam, afam;
    std::vector<int64_t> dface, dptr{0}, dcol, aface, apptr{0}, uptr{0}, ucol, vptr{0}, vcol;
    std::vector<double> dval, uval, vval, alen;
    for (int fm = 0; fm < 4; ++fm) {
      const gm_cc_faces& fc = cfg->faces[fm];
      for (int64_t r = 0; r < fc.n_dif; ++r) {
        dfam.push_back((uint8_t)fm);
        dface.push_back(fc.dif_face[r]);
        for (int64_t e = fc.dif_grad.ptr[r]; e < fc.dif_grad.ptr[r + 1]; ++e) {
          dcol.push_back(fc.dif_grad.col[e]);
          dval.push_back(fc.dif_grad.val[e]);
        }
        dptr.push_back((int64_t)dcol.size());
      }
      // advective faces: the Gauss points of face r are those with patch == r (contiguous)
      int64_t p = 0;
      for (int64_t r = 0; r < fc.n_adv; ++r) {
        afam.push_back((uint8_t)fm);
        aface.push_back(fc.adv_face[r]);
        while (p < fc.n_adv_points && fc.adv_patch[p] == r) {
          for (int64_t e = fc.adv_u.ptr[p]; e < fc.adv_u.ptr[p + 1]; ++e) {
            ucol.push_back(fc.adv_u.col[e]);
            uval.push_back(fc.adv_u.val[e]);
          }
          uptr.push_back((int64_t)ucol.size());
          for (int64_t e = fc.adv_v.ptr[p]; e < fc.adv_v.ptr[p + 1]; ++e) {
            vcol.push_back(fc.adv_v.col[e]);
            vval.push_back(fc.adv_v.val[e]);
          }
          vptr.push_back((int64_t)vcol.size());
          alen.push_back(fc.adv_len[p]);
          ++p;
        }
        apptr.push_back((int64_t)alen.size());
      }
      if (p != fc.n_adv_points) throw CcFail(GM_EVALUE, "advective face points must be grouped by face in order");
    }
    C->dfam.upload(dfam, st); C->dface.upload(dface, st); C->dptr.upload(dptr, st);
    C->dcol.upload(dcol, st); C->dval.upload(dval, st);
    C->afam.upload(afam, st); C->aface.upload(aface, st); C->apptr.upload(apptr, st);
    C->uptr.upload(uptr, st); C->ucol.upload(ucol, st); C->uval.upload(uval, st);
    C->vptr.upload(vptr, st); C->vcol.upload(vcol, st); C->vval.upload(vval, st);
    C->alen.upload(alen, st);
    // kernel arguments
    CcGeo& G = C->geo;
    G.nx = nx; G.ny = ny; G.usize = us; G.vsize = C->vsize; G.psize = Pn; G.F = F; G.dx = C->dx; G.dy = C->dy;
    G.idx = 1.0 / C->dx; G.idy = 1.0 / C->dy;
    G.ax = C->ax.p; G.ay = C->ay.p;
    G.cxx = C->cxx.p; G.cyy = C->cyy.p; G.cxy = C->cxy.p; G.cyx = C->cyx.p;
    G.axx = C->axx.p; G.ayy = C->ayy.p; G.axy = C->axy.p; G.ayx = C->ayx.p; G.aout = C->aout.p;
    G.flags = C->flags.p; G.cell_type = C->cell_type.p; G.kappa = C->kappa.p; G.ikappa = C->ikappa.p;
    G.ivol_rho = C->vol_rho.p; G.merge_of = C->merge_of.p; G.ms = C->ms.p; G.mm = C->mm.p;
    G.imvol_rho = C->mvol_rho.p;
    CcFix& X = C->fix;
    X.n_dif = (int)dface.size(); X.dfam = C->dfam.p; X.dface = C->dface.p; X.dptr = C->dptr.p; X.dcol = C->dcol.p;
    X.dval = C->dval.p;
    X.n_adv = (int)aface.size(); X.afam = C->afam.p; X.aface = C->aface.p; X.apptr = C->apptr.p;
    X.uptr = C->uptr.p; X.ucol = C->ucol.p; X.uval = C->uval.p; X.vptr = C->vptr.p; X.vcol = C->vcol.p;
    X.vval = C->vval.p; X.alen = C->alen.p;
    CcWall& W = C->wall;
    W.n = (int)nw; W.ptr = C->wptr.p; W.col = C->wcol.p; W.val = C->wval.p; W.tx = C->wtx.p; W.ty = C->wty.p;
    W.ds = C->wds.p; W.n_tgt = (int)tgt.size(); W.tgt = C->tgt.p; W.tptr = C->tptr.p; W.tk = C->tk.p;
    W.n_own = (int)own.size(); W.own = C->own.p; W.optr = C->optr.p; W.odon = C->odon.p;
    W.n_don = (int)donors.size(); W.don = C->don.p; W.tau = C->tau.p;
    W.n_aux = (int)aux_face.size(); W.aux_face = C->aux_face.p; W.aux_tgt = C->aux_tgt.p; W.aux_own = C->aux_own.p;
    W.aux_don = C->aux_don.p;
    // state and work arrays
    for (Buf<double>* b : {&C->U, &C->prev_adv, &C->q0, &C->now, &C->mid, &C->halfq, &C->expl,
                           &C->offset, &C->rhs, &C->star, &C->w, &C->result, &C->action, &C->tmp, &C->zero,
                           &C->la, &C->ld, &C->lr, &C->lprev, &C->lstar}) {
      b->alloc(F);
      b->zero(st);
    }
    for (Buf<double>* b : {&C->Pst, &C->halfp, &C->B, &C->phi, &C->inc}) {
      b->alloc(Pn);
      b->zero(st);
    }
    C->fxx.alloc(Pn); C->fyy.alloc(Pn); C->fxy.alloc(nvert); C->fyx.alloc(nvert);
    C->flux = CcFlux{C->fxx.p, C->fxy.p, C->fyx.p, C->fyy.p};
    C->pb.alloc(std::max(1, gmi::surface(C->P).n));
    C->V.alloc((size_t)(CN_M + 1) * F);
    C->gpart.alloc((size_t)CN_BLOCKS * CN_M);
    C->gpart2.alloc((size_t)CN_BLOCKS * CN_M);
    C->gdev.alloc(1);
    CCK(cudaMemsetAsync(C->gdev.p, 0, sizeof(CnDev), st));
    build_cn(C, cfg, fl, vr, mof, ms, mm, mv, tgt, tptr, tk, own, optr, odon, donors, dfam, dface, dptr, dcol, dval);
    C->lres.alloc(2 * CC_RES_BLOCKS);
    C->ftau.alloc(std::max<int64_t>(1, nw));
    C->diag.alloc(1);
    CCK(cudaMallocHost(&C->host_diag, sizeof(CcDiagDev)));
    C->d_act.upload(C->act_idx, st);
    if (const char* e = std::getenv("GHOSTMAC_PHASE_TIMING")) C->phase_on = e[0] == '1';
    if (C->phase_on)
      for (auto& e : C->pev) CCK(cudaEventCreate(&e));
    initial_state(C, inlet, cfg->cell_type, cfg->ax, cfg->ay);
  });
  if (rc != GM_OK) {
    gm_cc_destroy(c.release());
    return rc;
  }
  *out = c.release();
  return GM_OK;
}

int gm_cc_destroy(gm_cc* c) {
  if (!c) return GM_OK;
  if (c->st) cudaStreamSynchronize(c->st);
  for (auto& g : c->graphs)
    if (g.exec) cudaGraphExecDestroy(g.exec);
  if (c->host_diag) cudaFreeHost(c->host_diag);
  for (auto& e : c->pev)
    if (e) cudaEventDestroy(e);
  gm_handle* P = c->P;
  delete c;  // device buffers first, then the pressure handle and its stream
  if (P) gmi::pressure_destroy(P);
  return GM_OK;
}

int gm_cc_get_sizes(const gm_cc* c, gm_sizes* o) {
  if (!c || !o) return GM_EVALUE;
  std::memset(o, 0, sizeof *o);
  o->nx = c->nx; o->ny = c->ny; o->usize = c->usize; o->vsize = c->vsize; o->psize = c->psize;
  const gm::Geometry& g = gmi::geometry(c->P);
  o->nu_active = (int64_t)g.ui.size(); o->nv_active = (int64_t)g.vi.size(); o->np_active = (int64_t)g.pi.size();
  o->qsize = c->n_active;
  o->n_surface = g.n_surface;
  o->rank_p = gmi::schur_rank(c->P);
  o->dx = c->dx; o->dy = c->dy; o->U_ref = c->U_ref;
  return GM_OK;
}

int gm_cc_get_indices(const gm_cc* c, int64_t* ui, int64_t* vi, int64_t* pi) {
  if (!c) return GM_EVALUE;
  const gm::Geometry& g = gmi::geometry(c->P);
  if (ui) std::copy(g.ui.begin(), g.ui.end(), ui);
  if (vi) std::copy(g.vi.begin(), g.vi.end(), vi);
  if (pi) std::copy(g.pi.begin(), g.pi.end(), pi);
  return GM_OK;
}

int gm_cc_get_surface_points(const gm_cc* c, double* yx) {
  if (!c || !yx) return GM_EVALUE;
  const gm::Geometry& g = gmi::geometry(c->P);
  for (int k = 0; k < g.n_surface; ++k) {
    yx[2 * k] = g.surf_y[k];
    yx[2 * k + 1] = g.surf_x[k];
  }
  return GM_OK;
}

int gm_cc_set_state(gm_cc* c, const double* u, const double* v, const double* p) {
  if (!c) return GM_EVALUE;
  return guarded(c, [&] {
    if (u) copy_in(c->U.p, u, c->usize, c->st);
    if (v) copy_in(c->U.p + c->usize, v, c->vsize, c->st);
    if (p) copy_in(c->Pst.p, p, c->psize, c->st);
    CCK(cudaStreamSynchronize(c->st));
  });
}

int gm_cc_get_state(gm_cc* c, double* u, double* v, double* p) {
  if (!c) return GM_EVALUE;
  return guarded(c, [&] {
    if (u) CCK(cudaMemcpyAsync(u, c->U.p, c->usize * sizeof(double), cudaMemcpyDefault, c->st));
    if (v) CCK(cudaMemcpyAsync(v, c->U.p + c->usize, c->vsize * sizeof(double), cudaMemcpyDefault, c->st));
    if (p) CCK(cudaMemcpyAsync(p, c->Pst.p, c->psize * sizeof(double), cudaMemcpyDefault, c->st));
    CCK(cudaStreamSynchronize(c->st));
  });
}

int gm_cc_set_inlet(gm_cc* c, const double* u_inlet) {
  if (!c || !u_inlet) return GM_EVALUE;
  return guarded(c, [&] {
    copy_in(c->inlet.p, u_inlet, c->ny, c->st);
    c->offset_stale = true;
    CCK(cudaStreamSynchronize(c->st));
  });
}

int gm_cc_set_history(gm_cc* c, int32_t has_history, const double* prev_adv, const double* half_p, double prev_dt) {
  if (!c) return GM_EVALUE;
  return guarded(c, [&] {
    if (has_history) {
      if (!prev_adv || !half_p || !(std::isfinite(prev_dt) && prev_dt > 0))
        throw CcFail(GM_EVALUE, "AB2 history requires a finite positive previous timestep");
      // packed previous advection -> face grid
      std::vector<double> q((size_t)c->n_active), grid((size_t)c->F, 0.0);
      CCK(cudaMemcpy(q.data(), prev_adv, q.size() * sizeof(double), cudaMemcpyDefault));
      for (int64_t k = 0; k < c->n_active; ++k) grid[(size_t)c->act_idx[k]] = q[(size_t)k];
      CCK(cudaMemcpyAsync(c->prev_adv.p, grid.data(), grid.size() * sizeof(double), cudaMemcpyHostToDevice, c->st));
      copy_in(c->halfp.p, half_p, c->psize, c->st);
      c->prev_dt = prev_dt;
    }
    c->has_history = has_history != 0;
    CCK(cudaStreamSynchronize(c->st));
  });
}

int gm_cc_get_history(gm_cc* c, int32_t* has_history, double* prev_adv, double* half_p, double* prev_dt) {
  if (!c) return GM_EVALUE;
  return guarded(c, [&] {
    if (has_history) *has_history = c->has_history ? 1 : 0;
    if (prev_dt) *prev_dt = c->prev_dt;
    if (!c->has_history) return;
    if (prev_adv) {
      std::vector<double> grid((size_t)c->F);
      CCK(cudaMemcpyAsync(grid.data(), c->prev_adv.p, grid.size() * sizeof(double), cudaMemcpyDeviceToHost, c->st));
      CCK(cudaStreamSynchronize(c->st));
      std::vector<double> q((size_t)c->n_active);
      for (int64_t k = 0; k < c->n_active; ++k) q[(size_t)k] = grid[(size_t)c->act_idx[k]];
      CCK(cudaMemcpy(prev_adv, q.data(), q.size() * sizeof(double), cudaMemcpyDefault));
    }
    if (half_p) CCK(cudaMemcpyAsync(half_p, c->halfp.p, c->psize * sizeof(double), cudaMemcpyDefault, c->st));
    CCK(cudaStreamSynchronize(c->st));
  });
}

int gm_cc_step(gm_cc* c, double dt, int32_t n_steps, double start_time, gm_cc_step_diag* diag) {
  if (!c) return GM_EVALUE;
  if (!(std::isfinite(dt) && dt > 0) || n_steps <= 0) {
    c->err = "Finite fields and a positive timestep are required";
    return GM_EVALUE;
  }
  return guarded(c, [&] {
    cudaStream_t st = c->st;
    for (int32_t k = 0; k < n_steps; ++k) {
      refresh_offset(c);
      if (!c->counts_known) {
        for (int s : {S_P0, S_P1, S_P2}) gmi::set_sweeps(c->P, s, gmi::checks(c->P) - 1);
        c->arnoldi.raise(12);
      }
      gm_cc::Graph& gr = step_graph(c, dt);
      CCK(cudaMemsetAsync(gmi::control(c->P), 0, sizeof(StepCtl), st));
      CCK(cudaGraphLaunch(gr.exec, st));
      int r[4];
      CCK(cudaMemcpyAsync(r, &c->gdev.p->jend, sizeof r, cudaMemcpyDeviceToHost, st));
      CCK(cudaMemcpyAsync(c->host_diag, c->diag.p, sizeof(CcDiagDev), cudaMemcpyDeviceToHost, st));
      std::string m;
      const int prc = gmi::check(c->P, "cut-cell step", m);  // synchronises the stream
      const int cycles = r[1], its = r[2], converged = r[3];
      kernel_launch_adjust(gr.outer + (long long)cycles * gr.per_cycle);
      if (prc == ERR_SWEEPS) {
        // a solve needs more than the graph holds; the state is as before the step: once more with more
        const int what = gmi::failed_gate(c->P), n = c->arnoldi.n;
        if (what == CN_SHORT) c->arnoldi.raise(n < CN_M ? std::min(n + 2, CN_M) : CN_M + 1);
        else gmi::add_sweep(c->P, what);
        ++c->repeats;
        --k;
        continue;
      }
      // the first step sets the counts, and those that later steps do not use fall (HeldCount)
      const int used = cycles > 0 ? CN_M + 1 : its;
      if (!c->counts_known) c->arnoldi.n = std::max(used, c->arnoldi.least);
      c->arnoldi.steps(used, 1);
      for (int s : {S_P0, S_P1, S_P2}) {
        const int run = gmi::sweeps_run(c->P, s);
        if (!c->counts_known) gmi::set_sweeps(c->P, s, run);
        if (s != S_P0) gmi::note_sweeps(c->P, s, run, 1);
      }
      c->counts_known = true;
      if (c->phase_on)
        for (int q = 0; q < gm_cc::NPHASE; ++q) {
          float ms = 0.f;
          c->phase_ms[q] = cudaEventElapsedTime(&ms, c->pev[q], c->pev[q + 1]) == cudaSuccess ? ms : 0.0;
        }
      const CcDiagDev& d = *c->host_diag;
      gm_cc_step_diag out{};
      out.time = start_time + (k + 1) * dt;
      out.dt = dt;
      out.momentum_iterations = its;
      out.pressure_residual_linf = out.pressure_residual_l2 = std::nan("");
      out.momentum_residual_linf = bits_to_double(d.mres);
      out.coupled_momentum_residual_linf = bits_to_double(d.coupled);
      out.predicted_divergence = std::max(bits_to_double(d.pdiv[1]), bits_to_double(d.pdiv[2]));
      if (!c->has_history) out.predicted_divergence = std::max(out.predicted_divergence, bits_to_double(d.pdiv[0]));
      out.pressure_solves = c->has_history ? 2 : 3;
      out.max_divergence = bits_to_double(d.divmax);
      out.cfl = dt * (bits_to_double(d.umax) / c->dx + bits_to_double(d.vmax) / c->dy);
      for (int q = 0; q < 6; ++q) out.forces[q] = d.forces[q];
      const double denom = 0.5 * c->rho * (c->U_ref * c->U_ref) * c->D;
      out.cd = d.forces[0] / denom;
      out.cl = d.forces[1] / denom;
      out.cd_pressure = d.forces[2] / denom;
      out.cd_viscous = d.forces[4] / denom;
      out.cl_pressure = d.forces[3] / denom;
      out.cl_viscous = d.forces[5] / denom;
      // the step has replaced the state; history for the next step
      c->has_history = true;
      c->prev_dt = dt;
      int cls = GM_OK, gate = 0;
      std::string msg;
      const double rmax = bits_to_double(d.rhs_max);
      char buf[128];  // messages in the reference's %g form
      if (prc != GM_OK) { cls = prc; gate = GM_GATE_PRESSURE; msg = m; }
      else if (!(out.predicted_divergence < 1e-10)) {
        std::snprintf(buf, sizeof buf, "Pressure residual exceeds divergence budget: %g", out.predicted_divergence);
        cls = GM_ERUNTIME; gate = GM_GATE_PRESSURE; msg = buf;
      } else if (!converged || !(out.momentum_residual_linf <= 1e-10 * std::max(1.0, rmax)) ||
                 !std::isfinite(out.momentum_residual_linf)) {
        std::snprintf(buf, sizeof buf, "CN momentum solve failed: info=%d, residual=%g", converged ? 0 : 1,
                      out.momentum_residual_linf);
        cls = GM_ERUNTIME; gate = GM_GATE_MOMENTUM; msg = buf;
      } else if (!std::isfinite(out.cd) || !std::isfinite(out.cl)) {
        std::snprintf(buf, sizeof buf, "Non-finite force at t=%g; results not saved", out.time);
        cls = GM_EFLOAT; gate = GM_GATE_FORCE; msg = buf;
      } else if (!(out.max_divergence < 1e-10) || !(out.cfl < 0.5)) {
        cls = GM_ERUNTIME; gate = GM_GATE_STEP;
        msg = "Step failed the divergence/CFL acceptance gate";
      }
      out.status = cls;
      out.gate = gate;
      if (diag) diag[k] = out;
      if (cls != GM_OK) throw CcFail(cls, msg);
    }
  });
}

int gm_cc_legacy_step(gm_cc* c, double dt, int32_t n_steps, double start_time, int32_t centered,
                      gm_cc_step_diag* diag) {
  if (!c) return GM_EVALUE;
  if (!(std::isfinite(dt) && dt > 0) || n_steps <= 0) {
    c->err = "Finite fields and a positive timestep are required";
    return GM_EVALUE;
  }
  return guarded(c, [&] {
    cudaStream_t st = c->st;
    for (int32_t k = 0; k < n_steps; ++k) {
      CCK(cudaMemsetAsync(gmi::control(c->P), 0, sizeof(StepCtl), st));
      legacy_body(c, dt, centered != 0, st);
      CCK(cudaGetLastError());
      CCK(cudaMemcpyAsync(c->host_diag, c->diag.p, sizeof(CcDiagDev), cudaMemcpyDeviceToHost, st));
      std::string m;
      const int prc = gmi::check(c->P, "cut-cell legacy step", m);  // synchronises the stream
      // the predictor has replaced its history (solver/cut_cell_solver.py:1029-1031)
      c->l_has_prev = true;
      c->l_prev_dt = dt;
      const CcDiagDev& d = *c->host_diag;
      gm_cc_step_diag out{};
      out.time = start_time + (k + 1) * dt;
      out.dt = dt;
      out.predicted_divergence = bits_to_double(d.pdiv[1]);
      out.pressure_solves = 1;
      out.max_divergence = bits_to_double(d.divmax);
      out.cfl = dt * (bits_to_double(d.umax) / c->dx + bits_to_double(d.vmax) / c->dy);
      for (int q = 0; q < 6; ++q) out.forces[q] = d.forces[q];
      const double denom = 0.5 * c->rho * (c->U_ref * c->U_ref) * c->D;
      out.cd = d.forces[0] / denom;
      out.cl = d.forces[1] / denom;
      out.cd_pressure = d.forces[2] / denom;
      out.cd_viscous = d.forces[4] / denom;
      out.cl_pressure = d.forces[3] / denom;
      out.cl_viscous = d.forces[5] / denom;
      out.pressure_residual_linf = d.res_linf;
      out.pressure_residual_l2 = d.res_l2;
      int cls = GM_OK, gate = 0;
      std::string msg;
      char buf[96];
      if (prc != GM_OK) { cls = prc; gate = GM_GATE_PRESSURE; msg = m; }
      else if (!(out.predicted_divergence < 1e-10)) {
        std::snprintf(buf, sizeof buf, "Pressure residual exceeds divergence budget: %g", out.predicted_divergence);
        cls = GM_ERUNTIME; gate = GM_GATE_PRESSURE; msg = buf;
      } else if (!std::isfinite(out.cd) || !std::isfinite(out.cl)) {
        std::snprintf(buf, sizeof buf, "Non-finite force at t=%g; results not saved", out.time);
        cls = GM_EFLOAT; gate = GM_GATE_FORCE; msg = buf;
      }
      out.status = cls;
      out.gate = gate;
      if (diag) diag[k] = out;
      if (cls != GM_OK) throw CcFail(cls, msg);
    }
  });
}

int gm_cc_set_legacy_history(gm_cc* c, int32_t has_history, const double* prev_accel, double prev_dt) {
  if (!c) return GM_EVALUE;
  if (has_history && (!prev_accel || !(std::isfinite(prev_dt) && prev_dt > 0))) {
    c->err = "Incomplete predictor checkpoint history";
    return GM_EVALUE;
  }
  return guarded(c, [&] {
    if (has_history) copy_in(c->lprev.p, prev_accel, c->F, c->st);
    else CCK(cudaMemsetAsync(c->lprev.p, 0, c->F * sizeof(double), c->st));
    CCK(cudaStreamSynchronize(c->st));
    c->l_has_prev = has_history != 0;
    c->l_prev_dt = has_history ? prev_dt : 0.0;
  });
}

int gm_cc_get_legacy_history(gm_cc* c, int32_t* has_history, double* prev_accel, double* prev_dt) {
  if (!c) return GM_EVALUE;
  return guarded(c, [&] {
    if (has_history) *has_history = c->l_has_prev ? 1 : 0;
    if (prev_dt) *prev_dt = c->l_prev_dt;
    if (prev_accel) {
      CCK(cudaMemcpyAsync(prev_accel, c->lprev.p, c->F * sizeof(double), cudaMemcpyDefault, c->st));
      CCK(cudaStreamSynchronize(c->st));
    }
  });
}

int gm_cc_held_sweeps(const gm_cc* c, int32_t held[6], int64_t* repeats) {
  if (!c) return GM_EVALUE;
  if (held) {
    const std::array<int, 5> n = gmi::held_sweeps(c->P);
    std::copy(n.begin(), n.end(), held);
    held[5] = c->arnoldi.n;
  }
  if (repeats) *repeats = c->repeats;
  return GM_OK;
}

int gm_cc_phase_timing(const gm_cc* c, double out[8]) {
  if (!c || !out) return GM_EVALUE;
  for (int q = 0; q < gm_cc::NPHASE; ++q) out[q] = c->phase_ms[q];
  return GM_OK;
}

int gm_cc_apply(gm_cc* c, int32_t op, double param, const double* x, double* y, double* y2) {
  if (!c || !x || !y) return GM_EVALUE;
  return guarded(c, [&] {
    cudaStream_t st = c->st;
    const int64_t F = c->F, Pn = c->psize;
    auto gather = [&](const double* grid, double* outp) {
      std::vector<double> g((size_t)F), q((size_t)c->n_active);
      CCK(cudaMemcpyAsync(g.data(), grid, F * sizeof(double), cudaMemcpyDeviceToHost, st));
      CCK(cudaStreamSynchronize(st));
      for (int64_t k = 0; k < c->n_active; ++k) q[(size_t)k] = g[(size_t)c->act_idx[k]];
      CCK(cudaMemcpy(outp, q.data(), q.size() * sizeof(double), cudaMemcpyDefault));
    };
    auto scatter = [&](const double* q, double* grid) {
      std::vector<double> h((size_t)c->n_active), g((size_t)F, 0.0);
      CCK(cudaMemcpy(h.data(), q, h.size() * sizeof(double), cudaMemcpyDefault));
      for (int64_t k = 0; k < c->n_active; ++k) g[(size_t)c->act_idx[k]] = h[(size_t)k];
      CCK(cudaMemcpyAsync(grid, g.data(), F * sizeof(double), cudaMemcpyHostToDevice, st));
    };
    switch (op) {
      case GM_CC_OP_MOMENTUM_ADVECTION:
      case GM_CC_OP_MOMENTUM_ADVECTION_UPWIND:
      case GM_CC_OP_MOMENTUM_DIFFUSION: {
        copy_in(c->tmp.p, x, F, st);
        const bool adv = op != GM_CC_OP_MOMENTUM_DIFFUSION;
        momentum(c, adv, c->tmp.p, nullptr, adv ? 0.0 : param, 2, 0.0, c->w.p, c->action.p, st,
                 op == GM_CC_OP_MOMENTUM_ADVECTION_UPWIND);
        CCK(cudaMemcpyAsync(y, c->w.p, F * sizeof(double), cudaMemcpyDefault, st));
        if (y2) CCK(cudaMemcpyAsync(y2, c->action.p, F * sizeof(double), cudaMemcpyDefault, st));
        break;
      }
      case GM_CC_OP_ADVECTION:
      case GM_CC_OP_DIFFUSION: {
        scatter(x, c->tmp.p);
        if (op == GM_CC_OP_ADVECTION) momentum(c, true, c->tmp.p, c->inlet.p, 0.0, 0, 0.0, c->w.p, nullptr, st);
        else {
          refresh_offset(c);
          CnEval e{};
          e.x = c->tmp.p;
          e.out = c->w.p;
          cn_eval<CN_L>(c, e, st);
        }
        gather(c->w.p, y);
        break;
      }
      case GM_CC_OP_H_MATVEC: {
        scatter(x, c->tmp.p);
        CnEval e{};
        e.x = c->tmp.p;
        e.hdt = 0.5 * param;
        e.out = c->w.p;
        cn_eval<CN_H>(c, e, st);
        gather(c->w.p, y);
        break;
      }
      case GM_CC_OP_PROJECT: {
        scatter(x, c->tmp.p);
        CCK(cudaMemsetAsync(gmi::control(c->P), 0, sizeof(StepCtl), st));
        CCK(cudaMemsetAsync(c->diag.p, 0, sizeof(CcDiagDev), st));
        project(c, c->tmp.p, param, c->w.p, c->phi.p, S_P1, 1, st);
        std::string m;
        int rc = gmi::check(c->P, "project", m);
        if (rc != GM_OK) throw CcFail(rc, m);
        gather(c->w.p, y);
        if (y2) CCK(cudaMemcpyAsync(y2, c->phi.p, Pn * sizeof(double), cudaMemcpyDefault, st));
        break;
      }
      case GM_CC_OP_PRESSURE_SOLVE: {
        // solve_pressure(rhs, dt = param, rho): A phi = rhs on the fluid cells, phi = 0 on covered
        copy_in(c->B.p, x, Pn, st);
        counted();
        k_cc_scale_rhs<<<nblk(Pn), CC_TPB, 0, st>>>(c->geo, c->B.p);
        CCK(cudaMemsetAsync(gmi::control(c->P), 0, sizeof(StepCtl), st));
        CCK(cudaMemsetAsync(c->diag.p, 0, sizeof(CcDiagDev), st));
        gmi::pressure_solve(c->P, c->B.p, c->phi.p, S_P1);
        counted();
        k_cc_pdiv<<<std::min<unsigned>(nblk(Pn), 1216), CC_TPB, 0, st>>>(
            c->geo, gmi::pressure_residual(c->P), param / c->rho, &c->diag.p->pdiv[1]);
        std::string m;
        int rc = gmi::check(c->P, "pressure solve", m);
        if (rc != GM_OK) throw CcFail(rc, m);
        CCK(cudaMemcpyAsync(c->host_diag, c->diag.p, sizeof(CcDiagDev), cudaMemcpyDeviceToHost, st));
        CCK(cudaStreamSynchronize(st));
        const double pd = bits_to_double(c->host_diag->pdiv[1]);
        if (!(pd < 1e-10)) {
      char pbuf[96];
      std::snprintf(pbuf, sizeof pbuf, "Pressure residual exceeds divergence budget: %g", pd);
      throw CcFail(GM_ERUNTIME, pbuf);
    }
        CCK(cudaMemcpyAsync(y, c->phi.p, Pn * sizeof(double), cudaMemcpyDefault, st));
        break;
      }
      default:
        throw CcFail(GM_EVALUE, "unknown cut-cell operator");
    }
    CCK(cudaGetLastError());
    CCK(cudaStreamSynchronize(st));
  });
}

int gm_cc_surface_forces(gm_cc* c, const double* u, const double* v, const double* p, double mu, double out[6]) {
  if (!c || !u || !v || !p || !out) return GM_EVALUE;
  return guarded(c, [&] {
    cudaStream_t st = c->st;
    copy_in(c->tmp.p, u, c->usize, st);
    copy_in(c->tmp.p + c->usize, v, c->vsize, st);
    copy_in(c->B.p, p, c->psize, st);
    forces(c, c->tmp.p, c->B.p, mu, st);
    CCK(cudaMemcpyAsync(out, c->diag.p->forces, 6 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CCK(cudaStreamSynchronize(st));
  });
}

int gm_cc_divergence_stats(gm_cc* c, const double* u, const double* v, double out[3]) {
  if (!c || !out) return GM_EVALUE;
  return guarded(c, [&] {
    cudaStream_t st = c->st;
    const double* U = c->U.p;
    if (u || v) {
      copy_in(c->tmp.p, u ? u : c->U.p, c->usize, st);
      copy_in(c->tmp.p + c->usize, v ? v : c->U.p + c->usize, c->vsize, st);
      U = c->tmp.p;
    }
    counted();
    k_cc_divstats<<<1, CC_FORCE_THREADS, 0, st>>>(c->geo, U, c->pb.p);
    double r[4];
    CCK(cudaMemcpyAsync(r, c->pb.p, sizeof r, cudaMemcpyDeviceToHost, st));
    CCK(cudaStreamSynchronize(st));
    out[0] = r[0];
    out[1] = r[2] > 0 ? std::sqrt(r[1] / r[2]) : 0.0;
    out[2] = r[3];
  });
}

}  // extern "C"

// =============================================================================================
// the pressure system alone (the legacy staircase loop's Poisson solve)
// =============================================================================================
struct gm_poisson {
  std::string err;
  gm_handle* P = nullptr;
  int64_t psize = 0;
  Buf<double> b, x;
  Buf<double> ikappa;
  Buf<int32_t> cell_type;
  // the legacy loop's device scratch and per-step records (see gml::forces)
  Buf<double> lscratch, lrec;
  bool counts_known = false;  // a first step of the loop has set the sweeps its solves hold
  long long repeats = 0;      // solves that went on with a refinement sweep more
  cudaEvent_t ev_in = nullptr, ev_out = nullptr;
};

extern "C" {

const char* gm_poisson_last_error(const gm_poisson* p) { return p ? p->err.c_str() : gm_last_error(nullptr); }

int gm_poisson_create(int32_t nx, int32_t ny, double Lx, double Ly, double D, double xc, double yc, const double* ax,
                      const double* ay, const int32_t* cell_type, const double* kappa, gm_poisson** out) {
  if (!out || !ax || !ay || !cell_type || !kappa) { gm_internal_set_error("null argument"); return GM_EVALUE; }
  *out = nullptr;
  auto q = std::make_unique<gm_poisson>();
  gm::Geometry g;
  g.nx = nx; g.ny = ny; g.Lx = Lx; g.Ly = Ly; g.D = D; g.xc = xc; g.yc = yc;
  g.nu = 1.0; g.rho = 1.0; g.U_inf = 1.0; g.inflow = 0; g.U_m = 0.0;
  int ec = 0;
  if (!gm::build_cutcell_geometry(g, ax, ay, cell_type, kappa, ec)) {
    gm_internal_set_error(g.error.c_str());
    return ec ? ec : GM_EVALUE;
  }
  q->psize = g.psize;
  std::string perr;
  int rc = gmi::pressure_create(std::move(g), &q->P, perr);
  if (rc != GM_OK) {
    gm_internal_set_error(perr.c_str());
    return rc;
  }
  rc = guarded(nullptr, [&] {
    cudaStream_t st = gmi::stream(q->P);
    q->b.alloc(q->psize);
    q->x.alloc(q->psize);
    std::vector<double> ik(q->psize);
    for (int64_t c = 0; c < q->psize; ++c) ik[c] = cell_type[c] == 0 ? 1.0 / kappa[c] : 1.0;
    q->ikappa.upload(ik, st);
    q->cell_type.upload(std::vector<int32_t>(cell_type, cell_type + q->psize), st);
    CCK(cudaStreamSynchronize(st));
  });
  if (rc != GM_OK) {
    gm_poisson_destroy(q.release());
    return rc;
  }
  *out = q.release();
  return GM_OK;
}

int gm_poisson_destroy(gm_poisson* p) {
  if (!p) return GM_OK;
  gm_handle* P = p->P;
  if (P) cudaStreamSynchronize(gmi::stream(P));
  if (p->ev_in) cudaEventDestroy(p->ev_in);
  if (p->ev_out) cudaEventDestroy(p->ev_out);
  delete p;
  if (P) gmi::pressure_destroy(P);
  return GM_OK;
}

int gm_poisson_legacy_step(gm_poisson* p, gm_legacy_state* s, double dt, int32_t n_steps, gm_legacy_step_diag* diag,
                           void* stream) {
  if (!p) return GM_EVALUE;
  if (!s || n_steps <= 0 || !(std::isfinite(dt) && dt > 0)) {
    p->err = "a state, a positive step count and a finite positive dt are required";
    return GM_EVALUE;
  }
  if ((int64_t)s->nx * s->ny != p->psize || !s->u || !s->v || !s->p || !s->u_star || !s->v_star || !s->rhs ||
      !s->phi || !s->prev_du || !s->prev_dv || !s->zero_p || !s->mask || !s->inlet ||
      (s->centered && s->has_prev && !(std::isfinite(s->prev_dt) && s->prev_dt > 0))) {
    p->err = "the legacy state does not match the pressure system or is incomplete";
    return GM_EVALUE;
  }
  if (s->ghost)
    for (int k = 0; k < 2; ++k)
      if (s->n_ghost[k] < 0 || (s->n_ghost[k] > 0 && (!s->target[k] || !s->src[k] || !s->snap_of[k] ||
                                                      !s->weights[k] || !s->gamma[k] || !s->level[k]))) {
        p->err = "incomplete ghost tables";
        return GM_EVALUE;
      }
  try {
    cudaStream_t st = gmi::stream(p->P);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    if (!p->ev_in) CCK(cudaEventCreateWithFlags(&p->ev_in, cudaEventDisableTiming));
    if (!p->ev_out) CCK(cudaEventCreateWithFlags(&p->ev_out, cudaEventDisableTiming));
    CCK(cudaEventRecord(p->ev_in, cs));
    CCK(cudaStreamWaitEvent(st, p->ev_in, 0));
    const size_t need = gml::scratch_doubles(*s);
    if (p->lscratch.n < need) p->lscratch.alloc(need);
    constexpr int NR = 6;  // a step's record (gml::forces)
    if (p->lrec.n < (size_t)n_steps * NR) p->lrec.alloc((size_t)n_steps * NR);
    StepCtl* ctl = gmi::control(p->P);
    CCK(cudaMemsetAsync(ctl, 0, sizeof(StepCtl), st));
    CCK(cudaMemsetAsync(p->lrec.p, 0, (size_t)n_steps * NR * sizeof(double), st));
    std::vector<double> rec((size_t)n_steps * NR);
    // All steps queue behind each other: a failed pressure gate stops the kernels behind it, and a solve
    // that needs more refinement sweeps than are held (FP64 starts with none) goes on from there with one
    // more.  With a read-back a step and two idle sweeps a solve a step took 229 us at 350x213, now 154.
    // The loop's first step holds every sweep and sets the count (HeldCount).
    bool predicted = false;
    for (int32_t k = 0; k < n_steps;) {
      if (!p->counts_known) gmi::set_sweeps(p->P, S_P1, gmi::checks(p->P) - 1);
      for (const int32_t end = p->counts_known ? n_steps : 1; k < end; ++k) {
        if (!predicted) {
          gml::predict(*s, dt, p->lscratch.p, p->cell_type.p, p->ikappa.p, &ctl->err, st);
          if (s->centered) {  // the loop keeps the AB2 history before its pressure solve (solver/main.py:320)
            s->has_prev = 1;
            s->prev_dt = dt;
          }
          CCK(cudaMemsetAsync(ctl->solve, 0, sizeof ctl->solve, st));
        }
        predicted = false;
        gmi::hold_sweeps(p->P, true);
        gmi::pressure_solve(p->P, s->rhs, s->phi, S_P1);
        gmi::hold_sweeps(p->P, false);
        gml::correct(*s, dt, p->lscratch.p, &ctl->err, st);
        gml::forces(*s, p->lscratch.p, p->lrec.p + (size_t)k * NR, ctl, S_P1, gmi::checks(p->P), st);
      }
      CCK(cudaMemcpyAsync(rec.data(), p->lrec.p, rec.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
      CCK(cudaGetLastError());
      std::string m;
      const int rc = gmi::check(p->P, "pressure solve", m);  // synchronises the stream
      if (rc == GM_OK) {
        if (!p->counts_known) gmi::set_sweeps(p->P, S_P1, (int)rec[5] - 1);
        p->counts_known = true;
        continue;
      }
      if (rc != ERR_SWEEPS) throw CcFail(rc, m);
      gmi::add_sweep(p->P, gmi::failed_gate(p->P));
      ++p->repeats;
      for (k = 0; k < n_steps && rec[(size_t)k * NR + 5] != 0.0; ++k) {}
      CCK(cudaMemsetAsync(ctl, 0, sizeof(StepCtl), st));
      predicted = true;
    }
    CCK(cudaEventRecord(p->ev_out, st));
    CCK(cudaStreamWaitEvent(cs, p->ev_out, 0));
    for (int32_t k = 0; k < n_steps; ++k) gmi::note_sweeps(p->P, S_P1, (int)rec[(size_t)k * NR + 5] - 1, 1);
    if (diag)
      for (int32_t k = 0; k < n_steps; ++k) {
        for (int q = 0; q < 4; ++q) diag[k].forces[q] = rec[(size_t)k * NR + q];
        diag[k].pressure_residual_linf = rec[(size_t)k * NR + 4];
      }
  } catch (const CcFail& e) {
    p->err = e.msg;
    return e.cls;
  } catch (const std::exception& e) {
    p->err = e.what();
    return GM_ECUDA;
  }
  return GM_OK;
}

int gm_poisson_held_sweeps(const gm_poisson* p, int32_t* held, int64_t* repeats) {
  if (!p) return GM_EVALUE;
  if (held) *held = gmi::held_sweeps(p->P)[S_P1];
  if (repeats) *repeats = p->repeats;
  return GM_OK;
}

int gm_poisson_solve(gm_poisson* p, const double* rhs, double* phi, double* residual_linf) {
  if (!p || !rhs || !phi) return GM_EVALUE;
  int rc = GM_OK;
  try {
    cudaStream_t st = gmi::stream(p->P);
    copy_in(p->b.p, rhs, p->psize, st);
    CcGeo g{};
    g.psize = p->psize;
    g.cell_type = p->cell_type.p;
    g.ikappa = p->ikappa.p;
    counted();
    k_cc_scale_rhs<<<nblk(p->psize), CC_TPB, 0, st>>>(g, p->b.p);
    CCK(cudaMemsetAsync(gmi::control(p->P), 0, sizeof(StepCtl), st));
    gmi::pressure_solve(p->P, p->b.p, p->x.p, S_P1);
    std::string m;
    rc = gmi::check(p->P, "pressure solve", m);
    if (rc != GM_OK) throw CcFail(rc, m);
    if (residual_linf) {
      unsigned long long* bits = nullptr;
      CCK(cudaMallocAsync(reinterpret_cast<void**>(&bits), sizeof(unsigned long long), st));
      CCK(cudaMemsetAsync(bits, 0, sizeof(unsigned long long), st));
      counted();
      k_cc_maxdiff<<<std::min<unsigned>(nblk(p->psize), 1216), CC_TPB, 0, st>>>(
          p->psize, gmi::pressure_residual(p->P), nullptr, nullptr, 0.0, bits);
      unsigned long long hb = 0;
      CCK(cudaMemcpyAsync(&hb, bits, sizeof hb, cudaMemcpyDeviceToHost, st));
      CCK(cudaFreeAsync(bits, st));
      CCK(cudaStreamSynchronize(st));
      *residual_linf = bits_to_double(hb);
    }
    CCK(cudaMemcpyAsync(phi, p->x.p, p->psize * sizeof(double), cudaMemcpyDefault, st));
    CCK(cudaStreamSynchronize(st));
  } catch (const CcFail& e) {
    p->err = e.msg;
    return e.cls;
  } catch (const std::exception& e) {
    p->err = e.what();
    return GM_ECUDA;
  }
  return GM_OK;
}

}  // extern "C"
