// Periodic Taylor-Green case on the GPU (verification/taylor_green.py:14-59): the AB2/CN
// step of solver/time_integration.py:7-145 with the periodic staggered operators of
// periodic_momentum_operator (solver/cut_cell_solver.py:108-130, the full-fluid flux form of
// compute_momentum_rhs :790-957) and Fourier-space pressure and CN solves.
//
// Grid: u[j][i] at (i h, (j + 1/2) h), v[j][i] at ((i + 1/2) h, j h), p at cell centres,
// h = 2 pi / n; the velocity buffer holds u (n x n) then v (n x n), float64.
//
// Precision 0 runs everything in FP64.  Precision 1 runs the stencils of the momentum
// right-hand side and the Fourier solves in FP32 and refines both solves against the FP64
// operators (the CN system to the reference's residual gate, the pressure until the
// projected divergence is below 1e-11).
//
// A Fourier solve is three kernels: rows forward, columns (forward, symbol, inverse, in place),
// rows inverse.  In FP64 the real fields share complex transforms: the two velocity components as
// u + i v (the CN operator is real and the same for both), two rows of the divergence for the
// pressure, whose spectrum then has n / 2 + 1 columns.  A step decides nothing on the host: the
// launches of up to 64 steps are queued, the FP32 mode's with a held number of refinement sweeps
// gated on the device, and the failed-gate word is read once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>
#include <string>
#include <vector>

#include "../../include/ghostmac.h"
#include "exactdiv.cuh"
#include "fftplan.hpp"
#include "heldcount.hpp"
#include "transforms.cuh"

namespace gmk {
void kernel_launch_adjust(long long delta);  // the library's launch counter (kernels.cu)
int pdl_mode_ext();
}

namespace {
using namespace gmk;

constexpr int PT = 256;

struct TgError : std::exception {
  int cls;
  std::string msg;
  TgError(int c, std::string m) : cls(c), msg(std::move(m)) {}
  const char* what() const noexcept override { return msg.c_str(); }
};
#define TG_CK(call)                                                                              \
  do {                                                                                            \
    cudaError_t e_ = (call);                                                                      \
    if (e_ != cudaSuccess) throw TgError(GM_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
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
    if (count) TG_CK(cudaMalloc(&p, count * sizeof(T)));
  }
};

__device__ __forceinline__ int wrapi(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
__device__ __forceinline__ unsigned long long dbits_(double v) { return (unsigned long long)__double_as_longlong(v); }
// |v| as bits, on the integer pipe: the mask is PTX because the compiler turns fabs, or a C++
// mask of the sign bit, into an FP64 instruction
__device__ __forceinline__ unsigned long long absbits_(double v) {
  unsigned long long r;
  asm("and.b64 %0, %1, 0x7fffffffffffffff;" : "=l"(r) : "l"(dbits_(v)));
  return r;
}

__device__ void commit_max(unsigned long long v, unsigned long long* dst) {
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  if ((threadIdx.x & 31) == 0 && v) atomicMax(dst, v);
}

// ---- periodic flux-form operators (T arithmetic, S storage) -----------------------------
// -N(u) at u[j][i]: east/west face fluxes -uE^2 h, north/south corner fluxes -vN uN h, / h^2
template <typename T, typename S>
__device__ __forceinline__ T adv_u_p(const S* u, const S* v, int n, int j, int i, T h) {
  const int ip = wrapi(i + 1, n), im = wrapi(i - 1, n), jp = wrapi(j + 1, n), jm = wrapi(j - 1, n);
  const T uc = (T)u[j * n + i];
  const T uE = (T)0.5 * (uc + (T)u[j * n + ip]), uW = (T)0.5 * ((T)u[j * n + im] + uc);
  const T vN = (T)0.5 * ((T)v[jp * n + im] + (T)v[jp * n + i]), uN = (T)0.5 * (uc + (T)u[jp * n + i]);
  const T vS = (T)0.5 * ((T)v[j * n + im] + (T)v[j * n + i]), uS = (T)0.5 * ((T)u[jm * n + i] + uc);
  const T fE = -(uE * uE * h), fW = -(uW * uW * h), fN = -(vN * uN * h), fS = -(vS * uS * h);
  return ((fE - fW) + (fN - fS)) / (h * h);
}
template <typename T, typename S>
__device__ __forceinline__ T adv_v_p(const S* u, const S* v, int n, int j, int i, T h) {
  const int ip = wrapi(i + 1, n), im = wrapi(i - 1, n), jp = wrapi(j + 1, n), jm = wrapi(j - 1, n);
  const T vc = (T)v[j * n + i];
  const T vN = (T)0.5 * (vc + (T)v[jp * n + i]), vS = (T)0.5 * ((T)v[jm * n + i] + vc);
  const T uE = (T)0.5 * ((T)u[jm * n + ip] + (T)u[j * n + ip]), vE = (T)0.5 * (vc + (T)v[j * n + ip]);
  const T uW = (T)0.5 * ((T)u[jm * n + i] + (T)u[j * n + i]), vW = (T)0.5 * ((T)v[j * n + im] + vc);
  const T fN = -(vN * vN * h), fS = -(vS * vS * h), fE = -(uE * vE * h), fW = -(uW * vW * h);
  return ((fE - fW) + (fN - fS)) / (h * h);
}
// nu L at a point of one component (5-point, the face fluxes nu (f_next - f) / h * h)
template <typename T, typename S>
__device__ __forceinline__ T lap_p(const S* f, int n, int j, int i, T h, T nu) {
  const int ip = wrapi(i + 1, n), im = wrapi(i - 1, n), jp = wrapi(j + 1, n), jm = wrapi(j - 1, n);
  const T c = (T)f[j * n + i];
  const T fE = nu * ((T)f[j * n + ip] - c) / h * h, fW = nu * (c - (T)f[j * n + im]) / h * h;
  const T fN = nu * ((T)f[jp * n + i] - c) / h * h, fS = nu * (c - (T)f[jm * n + i]) / h * h;
  return ((fE - fW) + (fN - fS)) / (h * h);
}

// ---- a step's control words -----------------------------------------------------------------
// Reductions (bits of non-negative doubles), the step whose gate failed (RED_ERR, from 1) and, when it
// failed because a solve needed more refinement sweeps than were queued, that solve's slot + 1
// (RED_SHORT); then, of every refined solve (FP32 mode), the most sweeps that it ran in a step since the words
// were read (RED_USED) and this step's residual at every check.
enum : int { RED_CN = 0, RED_RHS = 1, RED_DIV = 2, RED_COUPLED = 3, RED_SHORT = 4, RED_ERR = 5, RED_USED = 6, NSLOT = 4, RED_W = RED_USED + NSLOT };
enum : int { SLOT_START = 0, SLOT_CN = 1, SLOT_P1 = 2, SLOT_P2 = 3, SLOT_CHECKS = 9, RED_N = RED_W + NSLOT * SLOT_CHECKS };
// Whether an earlier gate of this call failed: the state writers of the steps queued behind it return.
__device__ __forceinline__ bool tg_failed(const unsigned long long* red) {
  return *(const volatile unsigned long long*)(red + RED_ERR) != 0;
}
// A kernel launched as a programmatic dependent starts before its predecessor ends; every kernel of this
// file waits for it here before it reads anything.
__device__ __forceinline__ void tg_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Whether check k of a refined solve is above its target: max |r| <= 32 eps max(1, max |b|) for the CN
// solve, max |r| step <= 1e-11 for a pressure.  A check that did not run holds zero.
__device__ __forceinline__ bool tg_above(const unsigned long long* red, int slot, int k, double step) {
  const double r = __longlong_as_double((long long)*(const volatile unsigned long long*)(red + RED_W + slot * SLOT_CHECKS + k));
  if (slot != SLOT_CN) return !(r * step <= 1e-11);
  const double b = __longlong_as_double((long long)*(const volatile unsigned long long*)(red + RED_RHS));
  return !(r <= 32 * 2.220446049250313e-16 * (b > 1.0 ? b : 1.0));
}
// The FP32 mode queues a fixed number of refinement sweeps for each solve; the kernels of a sweep run
// while the check `k` before it (k < 0: none) is above the target.
struct TgGate {
  const unsigned long long* red;  // null: always open
  int slot, k;
  double step;
};
__device__ __forceinline__ bool tg_open(const TgGate& g) {
  tg_wait();
  if (!g.red) return true;
  return !tg_failed(g.red) && (g.k < 0 || tg_above(g.red, g.slot, g.k, g.step));
}
// The solve's residual is still above the target after all sweeps that were queued (`held`; the largest
// number that the mode takes, `most`, never falls short): the step fails and the host repeats it.
struct TgHeld {
  int slot, held, most;  // slot < 0: none
  double step;
};
__device__ __forceinline__ bool tg_short(unsigned long long* red, const TgHeld& h, int step_index) {
  if (h.slot < 0) return false;
  if (blockIdx.x == 0 && (int)threadIdx.x < h.held && tg_above(red, h.slot, threadIdx.x, h.step))
    atomicMax(red + RED_USED + h.slot, (unsigned long long)threadIdx.x + 1);  // a sweep ran behind this check
  if (h.held >= h.most || !tg_above(red, h.slot, h.held, h.step)) return false;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    red[RED_SHORT] = (unsigned long long)h.slot + 1;
    red[RED_ERR] = (unsigned long long)step_index;
  }
  return true;
}

// ---- kernels ------------------------------------------------------------------------------
// AB2/CN right-hand sides (solver/time_integration.py:20-67): mode 0 AB2, mode 1 start-up
// midpoint, mode 2 start-up CN right-hand side from the half-step velocity
// (the FP32 mode's; FP64: k_tg_rhs64)
template <typename T>
__global__ void k_tg_rhs(int n, double h, double nu, int mode, double dt, double alpha, const double* __restrict__ q,
                         const double* __restrict__ qh, const double* __restrict__ p, const double* __restrict__ prev,
                         double* __restrict__ now, double* __restrict__ out, unsigned long long* red, TgHeld start,
                         int step_index) {
  tg_wait();
  if (tg_failed(red) || (mode == 2 && tg_short(red, start, step_index))) return;
  const int nn = n * n;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  // this step's words; the previous step's kernels have read theirs (mode 2 follows the start-up solve)
  if (mode != 2 && t < NSLOT * SLOT_CHECKS) red[RED_W + t] = 0;
  if (mode != 2 && t == 0) red[RED_RHS] = 0;
  if (t >= 2 * nn) return;
  const int comp = t >= nn, k = t - comp * nn, j = k / n, i = k - j * n;
  const double* u = q;
  const double* v = q + nn;
  const T hh = (T)h, nuu = (T)nu, ddt = (T)dt;
  T lq, gp, a = 0;
  if (comp == 0) {
    lq = lap_p<T>(u, n, j, i, hh, nuu);
    gp = ((T)p[j * n + i] - (T)p[j * n + wrapi(i - 1, n)]) / hh;
    if (mode != 2) a = adv_u_p<T>(u, v, n, j, i, hh);
  } else {
    lq = lap_p<T>(v, n, j, i, hh, nuu);
    gp = ((T)p[j * n + i] - (T)p[wrapi(j - 1, n) * n + i]) / hh;
    if (mode != 2) a = adv_v_p<T>(u, v, n, j, i, hh);
  }
  const double qv = q[t];
  if (mode == 1) {
    now[t] = (double)a;
    out[t] = qv + (double)((T)0.5 * ddt * ((a + lq) - gp));
    return;
  }
  T expl;
  if (mode == 0) {
    expl = ((T)1 + (T)alpha) * a - (T)alpha * (T)prev[t];
    now[t] = (double)a;
  } else {
    expl = comp == 0 ? adv_u_p<T>(qh, qh + nn, n, j, i, hh) : adv_v_p<T>(qh, qh + nn, n, j, i, hh);
  }
  out[t] = qv + (double)(ddt * (expl + (T)0.5 * lq - gp));
}

// ---- FP64 stencils: 1/h and the products of the step formed on the host (GB300 issues FP64 at
// 1/64 of the FP32 rate and a divide costs about seven instructions) --------------------------
__device__ __forceinline__ double lap4(const double* __restrict__ f, int n, int j, int i, int k, double c) {
  const double e = f[i + 1 < n ? k + 1 : k + 1 - n], w = f[i > 0 ? k - 1 : k - 1 + n];
  const double u = f[j + 1 < n ? k + n : k + n - n * n], d = f[j > 0 ? k - n : k - n + n * n];
  return fma(-4.0, c, (e + w) + (u + d));
}

// FP64 right-hand sides (modes as k_tg_rhs), one thread per cell for its u and v face: the corner
// products u v are formed once for both, sums stay unhalved (ka = -1/(4h)), and the constants
// multiply last: about 45 FP64 instructions a cell.  The form with its divides took 369 us at
// 1024^2.
struct TgRhsC {
  double ka, kl, kg, c1, c2;  // -1/(4h); for the step e: nu e/(2 h^2) (mode 1: nu e/h^2), e/h, e (1 + alpha), e alpha
};
template <int MODE>
__global__ void k_tg_rhs64(int n, TgRhsC c, const double* __restrict__ q, const double* __restrict__ qh,
                           const double* __restrict__ p, const double* __restrict__ prev, double* __restrict__ now,
                           double* __restrict__ out, unsigned long long* red) {
  tg_wait();
  if (tg_failed(red)) return;
  const int nn = n * n, k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) red[RED_CN] = red[RED_RHS] = 0;  // this step's; the previous step's were read by its gate
  if (k >= nn) return;
  const int j = k / n, i = k - j * n;
  const int jp = j + 1 < n ? k + n : k + n - nn, jm = j > 0 ? k - n : k - n + nn;  // (j + 1, i), (j - 1, i)
  const int dp = i + 1 < n ? 1 : 1 - n, dm = i > 0 ? -1 : n - 1;                     // to i + 1, i - 1
  const double* u = q;
  const double* v = q + nn;
  const double uc = u[k], ue = u[k + dp], uw = u[k + dm], un = u[jp], us = u[jm];
  const double vc = v[k], ve = v[k + dp], vw = v[k + dm], vn = v[jp], vs = v[jm];
  double au, av;
  {
    const double* a = MODE == 2 ? qh : q;
    const double* b = a + nn;
    const double Uc = MODE == 2 ? a[k] : uc, Ue = MODE == 2 ? a[k + dp] : ue, Uw = MODE == 2 ? a[k + dm] : uw;
    const double Un = MODE == 2 ? a[jp] : un, Us = MODE == 2 ? a[jm] : us, Use = a[jm + dp];
    const double Vc = MODE == 2 ? b[k] : vc, Ve = MODE == 2 ? b[k + dp] : ve, Vw = MODE == 2 ? b[k + dm] : vw;
    const double Vn = MODE == 2 ? b[jp] : vn, Vs = MODE == 2 ? b[jm] : vs, Vnw = b[jp + dm];
    // corner products at (j, i), (j + 1, i), (j, i + 1), times 4
    const double c00 = (Vw + Vc) * (Us + Uc), c10 = (Vnw + Vn) * (Uc + Un), c01 = (Vc + Ve) * (Use + Ue);
    const double e = Uc + Ue, w = Uw + Uc, nn_ = Vc + Vn, ss = Vs + Vc;
    au = fma(e, e, -(w * w)) + (c10 - c00);
    av = fma(nn_, nn_, -(ss * ss)) + (c01 - c00);
  }
  const double lu = fma(-4.0, uc, (ue + uw) + (un + us)), lv = fma(-4.0, vc, (ve + vw) + (vn + vs));
  const double pc = p[k], gu = pc - p[k + dm], gv = pc - p[jm];
  au *= c.ka;
  av *= c.ka;
  if (MODE != 2) {
    now[k] = au;
    now[nn + k] = av;
  }
  double xu = c.c1 * au, xv = c.c1 * av;
  if (MODE == 0) {
    xu = fma(-c.c2, prev[k], xu);
    xv = fma(-c.c2, prev[nn + k], xv);
  }
  out[k] = uc + fma(c.kl, lu, fma(-c.kg, gu, xu));
  out[nn + k] = vc + fma(c.kl, lv, fma(-c.kg, gv, xv));
}

// The stencils that both precisions share, in two forms.  P64: as above, reciprocals on the host.
// Otherwise with the divides: the FP32 mode's pressure holds the FP32 rounding of its state, which
// another last bit of these stencils moves by 4e-8 in 20 steps, and its small grids gain little.
struct TgC {
  double h, nu, hdt;     // with divides: spacing, viscosity, dt / 2
  double hh, ihh;        // h^2 and its reciprocal
  double ih, kh;         // 1 / h; P64: dt nu / (2 h^2)
};
// nu L at a point (lap_p in FP64) with div_by for its divides
__device__ __forceinline__ double lap_d(const TgC& g, const double* f, int n, int j, int i) {
  const int ip = wrapi(i + 1, n), im = wrapi(i - 1, n), jp = wrapi(j + 1, n), jm = wrapi(j - 1, n);
  const double c = f[j * n + i], h = g.h, nu = g.nu;
  const double fE = div_by(nu * (f[j * n + ip] - c), h, g.ih) * h, fW = div_by(nu * (c - f[j * n + im]), h, g.ih) * h;
  const double fN = div_by(nu * (f[jp * n + i] - c), h, g.ih) * h, fS = div_by(nu * (c - f[jm * n + i]), h, g.ih) * h;
  return div_by((fE - fW) + (fN - fS), g.hh, g.ihh);
}
template <bool P64>
__device__ __forceinline__ double helm_p(const TgC& c, const double* __restrict__ f, int n, int j, int i, int k, double x) {
  if (P64) return fma(-c.kh, lap4(f, n, j, i, k, x), x);
  return x - c.hdt * lap_d(c, f, n, j, i);
}
__device__ __forceinline__ double div_sum(const double* __restrict__ q, int n, int j, int i, int k) {
  const int nn = n * n;
  return q[i + 1 < n ? k + 1 : k + 1 - n] - q[k] + q[nn + (j + 1 < n ? k + n : k + n - nn)] - q[nn + k];
}

// max |b - H x| (H = I - dt/2 nu L) and max |b|
template <bool P64>
__global__ void k_tg_hres(int n, TgC c, const double* __restrict__ b, const double* __restrict__ x,
                          unsigned long long* rmax, unsigned long long* bmax, TgGate gate) {
  if (!tg_open(gate)) return;
  const int nn = n * n;
  unsigned long long rm = 0, bm = 0;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 2 * nn; t += gridDim.x * blockDim.x) {
    const int comp = t >= nn, k = t - comp * nn, j = k / n, i = k - j * n;
    const double bv = b[t], rv = bv - helm_p<P64>(c, x + comp * nn, n, j, i, k, x[t]);
    rm = max(rm, absbits_(rv));
    bm = max(bm, absbits_(bv));
  }
  commit_max(rm, rmax);
  if (bmax) commit_max(bm, bmax);
}

// FP32 mode: (A phi)(k) with A = div grad (periodic 5-point / h^2)
__device__ __forceinline__ double pres_p(const TgC& c, const double* __restrict__ x, int n, int j, int i, int k) {
  return div_by(((x[j * n + wrapi(i + 1, n)] - x[k]) - (x[k] - x[j * n + wrapi(i - 1, n)]) +
                 (x[wrapi(j + 1, n) * n + i] - x[k]) - (x[k] - x[wrapi(j - 1, n) * n + i])), c.hh, c.ihh);
}
// max |b - A phi|
__global__ void k_tg_pres(int n, TgC c, const double* __restrict__ b, const double* __restrict__ x,
                          unsigned long long* rmax, TgGate gate) {
  if (!tg_open(gate)) return;
  const int nn = n * n;
  unsigned long long rm = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const int j = k / n, i = k - j * n;
    rm = max(rm, absbits_(b[k] - pres_p(c, x, n, j, i, k)));
  }
  commit_max(rm, rmax);
}

// out = q - step grad(phi), one thread per cell.  With gate_step > 0 (the projection of the CN
// velocity) it first applies the CN gate max |H star - rhs| <= 1e-10 max(1, max |rhs|)
// (solver/time_integration.py:100-104): every block reads the same two words, a failed gate records
// the step and leaves the state alone.
template <bool P64>
__global__ void k_tg_update(int n, TgC c, double step, double kg, const double* __restrict__ q,
                            const double* __restrict__ phi, double* __restrict__ out, unsigned long long* red,
                            int gate_step, TgHeld cn) {
  tg_wait();
  if (gate_step > 0) {
    if (tg_failed(red) || (!P64 && tg_short(red, cn, gate_step))) return;
    int last = 0;  // FP32 mode: the last check that ran
    if (!P64)
      while (last < cn.held && tg_above(red, SLOT_CN, last, 0.0)) ++last;
    const double r = __longlong_as_double((long long)red[P64 ? RED_CN : RED_W + SLOT_CN * SLOT_CHECKS + last]);
    const double b = __longlong_as_double((long long)red[RED_RHS]);
    if (!(r <= 1e-10 * (b > 1.0 ? b : 1.0)) || !isfinite(r)) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (!P64) red[RED_CN] = dbits_(r);
        red[RED_ERR] = (unsigned long long)gate_step;
      }
      return;
    }
  }
  const int nn = n * n, k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nn) return;
  const int j = k / n, i = k - j * n;
  const double f = phi[k];
  const double gu = f - phi[i > 0 ? k - 1 : k - 1 + n], gv = f - phi[j > 0 ? k - n : k - n + nn];
  out[k] = P64 ? fma(-kg, gu, q[k]) : q[k] - step * div_by(gu, c.h, c.ih);
  out[nn + k] = P64 ? fma(-kg, gv, q[nn + k]) : q[nn + k] - step * div_by(gv, c.h, c.ih);
}

// action = H result, proj = result + (rhs - action)   (solver/time_integration.py:107-113), and
// the largest |div result|
template <bool P64>
__global__ void k_tg_defect(int n, TgC c, const double* __restrict__ res, const double* __restrict__ rhs,
                            double* __restrict__ action, double* __restrict__ proj, unsigned long long* red, TgHeld p1,
                            int step_index) {
  tg_wait();
  if (tg_failed(red) || (!P64 && tg_short(red, p1, step_index))) return;
  const int nn = n * n;
  unsigned long long m = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const int j = k / n, i = k - j * n;
#pragma unroll
    for (int comp = 0; comp < 2; ++comp) {
      const int t = comp * nn + k;
      const double x = res[t], a = helm_p<P64>(c, res + comp * nn, n, j, i, k, x);
      action[t] = a;
      proj[t] = x + (rhs[t] - a);
    }
    const double d = div_sum(res, n, j, i, k);
    m = max(m, absbits_(P64 ? d * c.ih : div_by(d, c.h, c.ih)));
  }
  commit_max(m, red + RED_DIV);
}

// half = p + inc, out = half + factor inc, max |action - rhs + dt grad inc| (kg = dt / h)
template <bool P64>
__global__ void k_tg_pout(int n, TgC c, double dt, double kg, double factor, const double* __restrict__ p,
                          const double* __restrict__ inc, const double* __restrict__ action,
                          const double* __restrict__ rhs, double* __restrict__ half, double* __restrict__ pout,
                          unsigned long long* red, TgHeld p2, int step_index) {
  tg_wait();
  if (tg_failed(red) || (!P64 && tg_short(red, p2, step_index))) return;
  const int nn = n * n;
  unsigned long long m = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const int j = k / n, i = k - j * n;
    const double f = inc[k];
    const double gu = f - inc[i > 0 ? k - 1 : k - 1 + n], gv = f - inc[j > 0 ? k - n : k - n + nn];
    const double au = action[k] - rhs[k], av = action[nn + k] - rhs[nn + k];
    m = max(m, absbits_(P64 ? fma(kg, gu, au) : au + dt * div_by(gu, c.h, c.ih)));
    m = max(m, absbits_(P64 ? fma(kg, gv, av) : av + dt * div_by(gv, c.h, c.ih)));
    const double hv = p[k] + f;
    half[k] = hv;
    pout[k] = hv + factor * f;
  }
  commit_max(m, red + RED_COUPLED);
}

// ---- Fourier solves: rows (x) forward -> columns (y) forward, symbol, inverse -> rows inverse ----
// The symbol of the periodic 5-point Laplacian is lam(k, l) = -4 (s_k + s_l) / h^2 with
// s_k = sin^2(pi k / n).  kind 0: phi = F^-1[F b / lam] with the mean mode set to zero
// (verification/taylor_green.py:41-45); kind 1: x = F^-1[F b / (1 - c lam)].
//
// How a real field goes through the complex transforms:
//   LINE_REAL  one real row per transform (FP32: its rounding is kept as it is)
//   LINE_PAIR  two rows of s div(q) as real and imaginary part (FP64 pressure): the spectra of both
//              rows separate by their symmetry, n / 2 + 1 modes each, so the column pass runs
//              half the columns.  2 A and 2 B are stored, the halves are in the final scale
//   LINE_UV    u + i v (FP64 CN solve): the operator is real, so both parts solve at once
// FP64 transforms are bound by the FP64 pipe (about 33 instructions a complex point and pass): with
// these a pressure solve takes half and a CN solve half of the one-row form's work.  At 1024^2
// (8 8 8 2) the column pass takes 150 us for u + i v and 77 for a pressure (0.80 and 0.77 of the pipe's
// rate), row passes 82-87 and 47-54; a solve of seven kernels with transposes took 366 us a field,
// 186 a pressure and 319 both components with four transforms a block (3 % less with one, see gm_tg_create)
// and, forward in the FP32 mode (one real row each):
//   LINE_DIV   div(q) / step, stored on the way (the right-hand side of a pressure)
//   LINE_PRES  the residual b - A x of a pressure, its maximum on the way: a check of the refinement and
//   LINE_HRES  the first pass of the sweep behind it in one kernel; of the CN solve
enum : int { LINE_REAL = 0, LINE_PAIR = 1, LINE_UV = 2, LINE_DIV = 3, LINE_PRES = 4, LINE_HRES = 5 };
struct TgRow {
  TgC c;
  double s;              // LINE_DIV: 1 / step
  double* d;             // LINE_DIV: the stored right-hand side
  const double* x;       // LINE_PRES, LINE_HRES: the iterate
  unsigned long long *rmax, *bmax;
};

// A block holds gpb groups of gt threads, each with two length-n buffers (pad entries apart, so that
// a quarter warp's column loads touch distinct banks), behind the plan's twiddles.
template <typename T>
__host__ __device__ inline int tg_pad(int gpb) { return gpb > 1 ? (sizeof(T) == 8 ? 2 : 4) : 0; }
template <typename T>
__host__ __device__ inline size_t tg_smem(int n, int tw, int gpb) {
  return ((size_t)tw * sizeof(cplx<T>) + 15) / 16 * 16 + (size_t)gpb * (2 * (size_t)n + tg_pad<T>(gpb)) * sizeof(cplx<T>);
}
template <typename T>
__device__ __forceinline__ const cplx<T>* tw_of(const unsigned char* smem) { return reinterpret_cast<const cplx<T>*>(smem); }
template <typename T>
__device__ __forceinline__ cplx<T>* tg_stage(const FftPlan& plan, const cplx<T>* __restrict__ tw_g, unsigned char* smem) {
  cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem);
  for (int q = threadIdx.x; q < plan.tw_len; q += blockDim.x) tw[q] = tw_g[q];
  __syncthreads();
  return reinterpret_cast<cplx<T>*>(smem + ((size_t)plan.tw_len * sizeof(cplx<T>) + 15) / 16 * 16);
}

// Rows forward.  in: the real field (LINE_REAL; field blockIdx.y of n n values), q (LINE_PAIR), the
// two components (LINE_UV).
template <typename T, int LINE>
__global__ void k_tg_rows_fwd(int n, FftPlan plan, const cplx<T>* __restrict__ tw_g, const double* __restrict__ in,
                              cplx<T>* __restrict__ S, int pitch, double s, int gt, int gpb, TgRow rw, TgGate gate) {
  if (!tg_open(gate)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* base = tg_stage<T>(plan, tw_g, smem_raw);
  const int grp = threadIdx.x / gt, tid = threadIdx.x - grp * gt, nn = n * n;
  const int line = blockIdx.x * gpb + grp, row = LINE == LINE_PAIR ? 2 * line : line;
  if (row >= n) return;
  cplx<T>* a = base + (size_t)grp * (2 * n + tg_pad<T>(gpb));
  cplx<T>* b = a + n;
  const Grp G{tid, gt, grp + 1};
  if (LINE == LINE_REAL) {
    const double* src = in + (size_t)blockIdx.y * nn + (size_t)row * n;
    for (int e = tid; e < n; e += gt) a[e] = {(T)src[e], (T)0};
  } else if (LINE == LINE_UV) {
    const double* src = in + (size_t)row * n;
    for (int e = tid; e < n; e += gt) a[e] = {(T)src[e], (T)src[nn + e]};
  } else if (LINE == LINE_DIV) {
    for (int e = tid; e < n; e += gt) {
      const int k = row * n + e;
      const double d = div_by(div_sum(in, n, row, e, k), rw.c.h, rw.c.ih) * rw.s;
      rw.d[k] = d;
      a[e] = {(T)d, (T)0};
    }
  } else if (LINE == LINE_PRES || LINE == LINE_HRES) {
    const double* src = in + (size_t)blockIdx.y * nn;
    const double* x = rw.x + (size_t)blockIdx.y * nn;
    unsigned long long rm = 0, bm = 0;
    for (int e = tid; e < n; e += gt) {
      const int k = row * n + e;
      const double bv = src[k], r = bv - (LINE == LINE_PRES ? pres_p(rw.c, x, n, row, e, k) : helm_p<false>(rw.c, x, n, row, e, k, x[k]));
      a[e] = {(T)r, (T)0};
      rm = max(rm, absbits_(r));
      bm = max(bm, absbits_(bv));
    }
    commit_max(rm, rw.rmax);
    if (LINE == LINE_HRES && rw.bmax) commit_max(bm, rw.bmax);
  } else {
    const bool two = row + 1 < n;
    for (int e = tid; e < n; e += gt) {
      const double d0 = div_sum(in, n, row, e, row * n + e) * s;
      const double d1 = two ? div_sum(in, n, row + 1, e, (row + 1) * n + e) * s : 0.0;
      a[e] = {(T)d0, (T)d1};
    }
  }
  G.sync();
  const cplx<T>* r = fft_run<T>(a, b, plan, 1, tw_of<T>(smem_raw), -1, G);
  cplx<T>* dst = S + (size_t)blockIdx.y * nn + (size_t)row * pitch;
  if (LINE == LINE_PAIR) {
    const bool two = row + 1 < n;
    for (int k = tid; k <= n / 2; k += gt) {
      const cplx<T> z = r[k], c = r[k ? n - k : 0];
      dst[k] = {z.x + c.x, z.y - c.y};
      if (two) dst[pitch + k] = {z.y + c.y, c.x - z.x};
    }
  } else {
    for (int e = tid; e < n; e += gt) dst[e] = r[e];
  }
}

// Columns forward, symbol, columns inverse, in place: a block's groups take gpb neighbouring
// columns, loaded and stored by the whole block along the rows (64-byte pieces for FP64).  f: the
// FP64 symbol table (n x (n / 2 + 1), lam(k, n - l) = lam(k, l)); FP32 forms the symbol as it goes.
template <typename T>
__global__ void k_tg_cols(int n, FftPlan plan, const cplx<T>* __restrict__ tw_g, cplx<T>* __restrict__ S, int pitch,
                          int ncols, const double* __restrict__ f, const T* __restrict__ s2, int kind, T hh2, T coef,
                          int gt, int gpb, TgGate gate) {
  if (!tg_open(gate)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* base = tg_stage<T>(plan, tw_g, smem_raw);
  const int stride = 2 * n + tg_pad<T>(gpb), c0 = blockIdx.x * gpb;
  cplx<T>* field = S + (size_t)blockIdx.y * n * n;
  const int lc = threadIdx.x % gpb, lr = threadIdx.x / gpb, ls = blockDim.x / gpb;
  if (c0 + lc < ncols)
    for (int e = lr; e < n; e += ls) base[lc * stride + e] = field[(size_t)e * pitch + c0 + lc];
  __syncthreads();
  const int grp = threadIdx.x / gt, tid = threadIdx.x - grp * gt, col = c0 + grp;
  cplx<T>* r = base + grp * stride;  // where the column ends up (group-uniform)
  if (col < ncols) {
    cplx<T>* a = r;
    cplx<T>* b = a + n;
    const Grp G{tid, gt, grp + 1};
    const cplx<T>* tw = tw_of<T>(smem_raw);
    r = fft_run<T>(a, b, plan, 1, tw, -1, G);
    cplx<T>* o = r == a ? b : a;
    if (sizeof(T) == 8) {
      const int nh = n / 2 + 1, kc = col < nh ? col : n - col;
      for (int e = tid; e < n; e += gt) {
        const T g = (T)f[(size_t)e * nh + kc];
        r[e] = {r[e].x * g, r[e].y * g};
      }
    } else {
      for (int e = tid; e < n; e += gt) {
        const T lam = (T)-4 * (s2[col] + s2[e]) / hh2;
        T g;
        if (kind == 0) g = (col == 0 && e == 0) ? (T)0 : (T)1 / lam;
        else g = (T)1 / ((T)1 - coef * lam);
        r[e] = {r[e].x * g, r[e].y * g};
      }
    }
    G.sync();
    r = fft_run<T>(r, o, plan, 1, tw, +1, G);
  }
  // two transforms of equal length end in the buffer they began in: column c is at base + c stride
  __syncthreads();
  if (c0 + lc < ncols)
    for (int e = lr; e < n; e += ls) field[(size_t)e * pitch + c0 + lc] = base[lc * stride + e];
}

// Rows inverse: the real parts (LINE_PAIR: two rows, LINE_UV: both components) times scale, FP64.
template <typename T, int LINE>
__global__ void k_tg_rows_inv(int n, FftPlan plan, const cplx<T>* __restrict__ tw_g, const cplx<T>* __restrict__ S,
                              int pitch, double* __restrict__ out, T scale, int accumulate, int gt, int gpb, TgGate gate) {
  if (!tg_open(gate)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* base = tg_stage<T>(plan, tw_g, smem_raw);
  const int grp = threadIdx.x / gt, tid = threadIdx.x - grp * gt, nn = n * n;
  const int line = blockIdx.x * gpb + grp, row = LINE == LINE_PAIR ? 2 * line : line;
  if (row >= n) return;
  cplx<T>* a = base + (size_t)grp * (2 * n + tg_pad<T>(gpb));
  cplx<T>* b = a + n;
  const Grp G{tid, gt, grp + 1};
  const cplx<T>* src = S + (size_t)blockIdx.y * nn + (size_t)row * pitch;
  const bool two = LINE == LINE_PAIR && row + 1 < n;
  if (LINE == LINE_PAIR) {
    for (int k = tid; k <= n / 2; k += gt) {
      const cplx<T> A = src[k], B = two ? src[pitch + k] : cplx<T>{(T)0, (T)0};
      a[k] = {A.x - B.y, A.y + B.x};
      if (k && n - k != k) a[n - k] = {A.x + B.y, B.x - A.y};
    }
  } else {
    for (int e = tid; e < n; e += gt) a[e] = src[e];
  }
  G.sync();
  const cplx<T>* r = fft_run<T>(a, b, plan, 1, tw_of<T>(smem_raw), +1, G);
  double* dst = out + (size_t)blockIdx.y * nn + (size_t)row * n;
  for (int e = tid; e < n; e += gt) {
    const double re = (double)(r[e].x * scale);
    if (LINE == LINE_REAL) {
      dst[e] = accumulate ? dst[e] + re : re;
    } else {
      const double im = (double)(r[e].y * scale);
      dst[e] = re;
      if (LINE == LINE_UV) dst[nn + e] = im;
      else if (two) dst[n + e] = im;
    }
  }
}

// FP64 symbol tables (n x (n / 2 + 1)): the factor of each mode
__global__ void k_tg_symbol(int n, const double* __restrict__ s2, int kind, double hh2, double coef, double* __restrict__ f) {
  tg_wait();
  const int nh = n / 2 + 1;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n * nh; t += gridDim.x * blockDim.x) {
    const int l = t / nh, k = t - l * nh;
    const double lam = -4 * (s2[l] + s2[k]) / hh2;
    f[t] = kind == 0 ? (t == 0 ? 0.0 : 1 / lam) : 1 / (1 - coef * lam);
  }
}

unsigned grid_for(int64_t n) { return (unsigned)std::min<int64_t>((n + PT - 1) / PT, 152 * 8); }

}  // namespace

struct gm_tg {
  int n = 0, precision = 0;
  double nu = 0, h = 0;
  std::string err;
  cudaStream_t st = nullptr;
  FftPlan plan{};
  int gt[2] = {32, 32}, gpb[2] = {1, 1};  // threads per transform, transforms per block (FP32, FP64)
  size_t smem[2] = {0, 0};
  Buf<double> q, qn, hist, now, rhs, star, mid, half_q, action, proj, phalf, phalf_n, pout, phi, inc, div;
  Buf<double> tw64, s2_64, sym_p, sym_h;  // FP64 symbol tables of the pressure and the CN operator (for sym_dt)
  Buf<float> tw32, s2_32;
  double sym_dt = 0;
  Buf<unsigned char> spec;            // the spectrum: n x n complex FP64, or two of FP32
  Buf<unsigned long long> red;        // RED_*
  unsigned long long* host_red = nullptr;  // its page-locked copy
  // FP32 mode: refinement sweeps queued for each solve.  A read-back per check held the stream for some
  // 20 us, six to eight times a step; now the steps of a call queue behind each other, a step that needs
  // one sweep more than is held leaves its state alone, and the host repeats it with the sweep.  The
  // first step holds as many as the mode takes and sets the counts, which fall when unused (HeldCount).
  HeldCount held[NSLOT];
  bool held_known = false;
  long long repeats = 0;  // steps repeated for a sweep more
  ~gm_tg() { if (host_red) cudaFreeHost(host_red); }
  bool has_history = false;
  double prev_dt = 0;
};

namespace {

template <typename... K, typename... A>
void tg_launch(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = gmk::pdl_mode_ext();
  cfg.attrs = at;
  cfg.numAttrs = 1;
  gmk::kernel_launch_adjust(1);
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

unsigned blocks_of(int64_t n) { return (unsigned)((n + PT - 1) / PT); }
TgC stencil_consts(const gm_tg* t, double dt) {
  const double hh = t->h * t->h;
  return TgC{t->h, t->nu, 0.5 * dt, hh, 1.0 / hh, 1.0 / t->h, 0.5 * dt * t->nu / hh};
}
// refinement sweeps at most: CN 6 (then a last check), pressure 8 (none behind the last)
int most_of(int slot) { return slot == SLOT_CN ? 6 : 8; }
TgHeld held_of(const gm_tg* t, int slot, double step) {
  return t->precision ? TgHeld{slot, t->held[slot].n, most_of(slot), step} : TgHeld{-1, 0, 0, 0.0};
}

// One application of a solve: kind 0 Poisson, 1 Helmholtz (coef = dt nu / 2), the forward rows as LINE:
//   FP32: x (+)= S^-1 of `fields` cell grids of n n values.
//   FP64: kind 0 takes the velocity b and solves for s div(b); kind 1 takes both components.
// first gates the forward rows, rest the other two kernels.
template <typename T, int LINE>
void fourier_solve(gm_tg* t, int kind, double coef, const double* b, double* x, bool accumulate, int fields, double s,
                   const TgRow& rw, const TgGate& first, const TgGate& rest) {
  constexpr bool D = sizeof(T) == 8;
  constexpr int INV = D ? LINE : LINE_REAL;
  const int n = t->n, gt = t->gt[D], gpb = t->gpb[D];
  const dim3 thr((unsigned)(gt * gpb));
  const size_t sm = t->smem[D];
  cudaStream_t st = t->st;
  const cplx<T>* tw = D ? (const cplx<T>*)t->tw64.p : (const cplx<T>*)t->tw32.p;
  const T* s2 = D ? (const T*)t->s2_64.p : (const T*)t->s2_32.p;
  cplx<T>* S = reinterpret_cast<cplx<T>*>(t->spec.p);
  const T scale = (T)((LINE == LINE_PAIR ? 0.5 : 1.0) / ((double)n * n));
  const int ncols = LINE == LINE_PAIR ? n / 2 + 1 : n, lines = LINE == LINE_PAIR ? (n + 1) / 2 : n;
  const dim3 gr((unsigned)((lines + gpb - 1) / gpb), (unsigned)fields), gc((unsigned)((ncols + gpb - 1) / gpb), (unsigned)fields);
  const double* f = kind == 0 ? t->sym_p.p : t->sym_h.p;
  tg_launch(k_tg_rows_fwd<T, LINE>, gr, thr, sm, st, n, t->plan, tw, b, S, ncols, s, gt, gpb, rw, first);
  tg_launch(k_tg_cols<T>, gc, thr, sm, st, n, t->plan, tw, S, ncols, ncols, f, s2, kind, (T)(t->h * t->h), (T)coef, gt, gpb, rest);
  tg_launch(k_tg_rows_inv<T, INV>, gr, thr, sm, st, n, t->plan, tw, (const cplx<T>*)S, ncols, x, scale, accumulate ? 1 : 0, gt, gpb, rest);
  TG_CK(cudaGetLastError());
}

const unsigned long long* read_red(gm_tg* t) {
  TG_CK(cudaMemcpyAsync(t->host_red, t->red.p, RED_W * sizeof(unsigned long long), cudaMemcpyDeviceToHost, t->st));
  TG_CK(cudaStreamSynchronize(t->st));
  return t->host_red;
}
double bitsd(unsigned long long b) {
  double d;
  std::memcpy(&d, &b, sizeof d);
  return d;
}

// The FP32 solve of a slot with its held refinement sweeps: the residual that sweep k transforms is check
// k - 1, so a sweep is three kernels; a last check follows the last sweep.
template <int FIRST, int RES>
void refined_solve(gm_tg* t, int slot, double coef, const double* b, const double* rhs, double* x, double dt, double step) {
  const int fields = slot == SLOT_CN ? 2 : 1, kind = slot == SLOT_CN ? 1 : 0, held = std::min(t->held[slot].n, most_of(slot));
  unsigned long long* w = t->red.p + RED_W + slot * SLOT_CHECKS;
  unsigned long long* bmax = slot == SLOT_CN ? t->red.p + RED_RHS : nullptr;
  const TgC c = stencil_consts(t, dt);
  auto gate = [&](int k) { return TgGate{t->red.p, slot, k, step}; };
  TgRow rw{c, 1.0 / step, t->div.p, x, nullptr, nullptr};
  fourier_solve<float, FIRST>(t, kind, coef, b, x, false, fields, 0.0, rw, gate(-1), gate(-1));
  for (int k = 1; k <= held; ++k) {
    rw.rmax = w + k - 1;
    rw.bmax = k == 1 ? bmax : nullptr;
    fourier_solve<float, RES>(t, kind, coef, rhs, x, true, fields, 0.0, rw, gate(k - 2), gate(k - 1));
  }
  if (slot != SLOT_CN && held >= most_of(slot)) return;
  const int64_t nn = (int64_t)t->n * t->n;
  if (slot == SLOT_CN)
    tg_launch(k_tg_hres<false>, dim3(grid_for(2 * nn)), dim3(PT), 0, t->st, t->n, c, rhs, (const double*)x, w + held,
              held == 0 ? bmax : nullptr, gate(held - 1));
  else
    tg_launch(k_tg_pres, dim3(grid_for(nn)), dim3(PT), 0, t->st, t->n, c, rhs, (const double*)x, w + held, gate(held - 1));
}

// project(q, step): phi = A^-1 (div q / step), out = q - step grad phi (refined in FP32 mode
// until the projected divergence max |step (b - A phi)| is below 1e-11)
void tg_project(gm_tg* t, const double* q, double step, double* out, double* phi, int slot, int gate_step) {
  if (t->precision == 0)
    fourier_solve<double, LINE_PAIR>(t, 0, 0.0, q, phi, false, 1, 1.0 / (t->h * step), TgRow{}, TgGate{}, TgGate{});
  else
    refined_solve<LINE_DIV, LINE_PRES>(t, slot, 0.0, q, t->div.p, phi, 0.0, step);
  if (!out) return;
  tg_launch(t->precision ? k_tg_update<false> : k_tg_update<true>, dim3(blocks_of((int64_t)t->n * t->n)), dim3(PT), 0, t->st, t->n,
            stencil_consts(t, 0.0), step, step / t->h, q, (const double*)phi, out, t->red.p, gate_step, held_of(t, SLOT_CN, 0.0));
}

// star = H^-1 rhs (two components), refined in FP32 mode to the CN gate
void tg_helmholtz(gm_tg* t, double dt, const double* rhs, double* star) {
  const int n = t->n;
  const int64_t nn = (int64_t)n * n;
  const double c = 0.5 * dt * t->nu;
  if (t->precision) {
    refined_solve<LINE_REAL, LINE_HRES>(t, SLOT_CN, c, rhs, rhs, star, dt, 1.0);
    return;
  }
  if (t->sym_dt != dt) {
    tg_launch(k_tg_symbol, dim3(grid_for((int64_t)n * (n / 2 + 1))), dim3(PT), 0, t->st, n, (const double*)t->s2_64.p, 1,
              t->h * t->h, c, t->sym_h.p);
    t->sym_dt = dt;
  }
  fourier_solve<double, LINE_UV>(t, 1, c, rhs, star, false, 1, 0.0, TgRow{}, TgGate{}, TgGate{});
  tg_launch(k_tg_hres<true>, dim3(grid_for(2 * nn)), dim3(PT), 0, t->st, n, stencil_consts(t, dt), rhs, (const double*)star,
            t->red.p + RED_CN, t->red.p + RED_RHS, TgGate{});
}

// ab2_cn_step (solver/time_integration.py:7-145) with the periodic operators, queued on the
// stream; `step` counts from 1 in the call.  The steps behind a failed gate leave the state alone
// (see k_tg_update).
void tg_step(gm_tg* t, double dt, int step) {
  const int n = t->n;
  const int64_t nn = (int64_t)n * n;
  cudaStream_t st = t->st;
  const double h = t->h;
  auto rhs_kernel = [&](int mode, double alpha, const double* qh, double* out) {
    if (t->precision == 1) {
      tg_launch(k_tg_rhs<float>, dim3(blocks_of(2 * nn)), dim3(PT), 0, st, n, h, t->nu, mode, dt, alpha, (const double*)t->q.p, qh,
                (const double*)t->phalf.p, (const double*)t->hist.p, t->now.p, out, t->red.p, held_of(t, SLOT_START, 0.5 * dt), step);
      return;
    }
    const double e = mode == 1 ? 0.5 * dt : dt;  // the start-up midpoint goes half a step with the full L q
    const TgRhsC c{-0.25 / h, (mode == 1 ? 1.0 : 0.5) * e * t->nu / (h * h), e / h, e * (1 + alpha), e * alpha};
    auto* k = mode == 0 ? k_tg_rhs64<0> : mode == 1 ? k_tg_rhs64<1> : k_tg_rhs64<2>;
    tg_launch(k, dim3(blocks_of(nn)), dim3(PT), 0, st, n, c, (const double*)t->q.p, qh, (const double*)t->phalf.p,
              (const double*)t->hist.p, t->now.p, out, t->red.p);
  };
  const bool first = !t->has_history;
  if (first) {
    rhs_kernel(1, 0.0, nullptr, t->mid.p);
    tg_project(t, t->mid.p, 0.5 * dt, t->half_q.p, t->phi.p, SLOT_START, 0);
    rhs_kernel(2, 0.0, t->half_q.p, t->rhs.p);
  } else {
    rhs_kernel(0, dt / (2 * t->prev_dt), nullptr, t->rhs.p);
  }
  tg_helmholtz(t, dt, t->rhs.p, t->star.p);
  tg_project(t, t->star.p, dt, t->qn.p, t->phi.p, SLOT_P1, step);
  const bool f32 = t->precision != 0;
  tg_launch(f32 ? k_tg_defect<false> : k_tg_defect<true>, dim3(grid_for(nn)), dim3(PT), 0, st, n, stencil_consts(t, dt),
            (const double*)t->qn.p, (const double*)t->rhs.p, t->action.p, t->proj.p, t->red.p, held_of(t, SLOT_P1, dt), step);
  tg_project(t, t->proj.p, dt, nullptr, t->inc.p, SLOT_P2, 0);
  const double factor = first ? 1.0 : dt / (dt + t->prev_dt);
  tg_launch(f32 ? k_tg_pout<false> : k_tg_pout<true>, dim3(grid_for(nn)), dim3(PT), 0, st, n, stencil_consts(t, dt), dt, dt / h,
            factor, (const double*)t->phalf.p, (const double*)t->inc.p, (const double*)t->action.p, (const double*)t->rhs.p,
            t->phalf_n.p, t->pout.p, t->red.p, held_of(t, SLOT_P2, dt), step);
  TG_CK(cudaGetLastError());
}

void tg_swap(gm_tg* t) {
  std::swap(t->q.p, t->qn.p);
  std::swap(t->phalf.p, t->phalf_n.p);
  std::swap(t->hist.p, t->now.p);
}

// n_steps steps; the largest divergence of any of them raises *max_div.  A failed CN gate leaves the
// state after the last good step.
void tg_steps(gm_tg* t, double dt, int n_steps, double* max_div) {
  const bool had = t->has_history;
  const double prev = t->prev_dt;
  TG_CK(cudaMemsetAsync(t->red.p, 0, RED_N * sizeof(unsigned long long), t->st));
  const unsigned long long* r = t->host_red;
  const bool f32 = t->precision != 0;
  for (int done = 0, read = 0; done < n_steps;) {
    if (f32 && !t->held_known)
      for (int s = 0; s < NSLOT; ++s) t->held[s].n = most_of(s);
    tg_step(t, dt, done + 1);
    tg_swap(t);
    t->has_history = true;
    t->prev_dt = dt;
    ++done;
    if (done != n_steps && done - read < 64 && (!f32 || t->held_known)) continue;
    const int err = (int)read_red(t)[RED_ERR];
    if (!err) {
      for (int s = 0; f32 && s < NSLOT; ++s) {
        const int used = (int)r[RED_USED + s];
        if (!t->held_known) t->held[s].n = used;
        else if (s != SLOT_START) t->held[s].steps(used, done - read);
      }
      t->held_known = f32;
      if (f32) TG_CK(cudaMemsetAsync(t->red.p + RED_USED, 0, NSLOT * sizeof(unsigned long long), t->st));
      read = done;
      continue;
    }
    if ((done - (err - 1)) % 2) tg_swap(t);  // step err failed: the state is that after err - 1 steps
    if (err == 1) { t->has_history = had; t->prev_dt = prev; }
    const int slot = (int)r[RED_SHORT] - 1;
    if (slot < 0) throw TgError(GM_ERUNTIME, "CN momentum solve failed: residual=" + std::to_string(bitsd(r[RED_CN])));
    t->held[slot].raise(t->held[slot].n + 1);
    ++t->repeats;
    done = read = err - 1;
    TG_CK(cudaMemsetAsync(t->red.p + RED_SHORT, 0, 2 * sizeof(unsigned long long), t->st));
  }
  *max_div = std::max(*max_div, bitsd(r[RED_DIV]));
}

int tg_guard(gm_tg* t, const std::function<void()>& f) {
  try {
    f();
    return GM_OK;
  } catch (const TgError& e) {
    if (t) t->err = e.msg;
    return e.cls;
  } catch (const std::exception& e) {
    if (t) t->err = e.what();
    return GM_ECUDA;
  }
}

std::string g_tg_create_error;

}  // namespace

extern "C" {

int gm_tg_create(int32_t n, double nu, int32_t precision, gm_tg** out) {
  if (!out) return GM_EVALUE;
  *out = nullptr;
  if (n < 8 || !(std::isfinite(nu) && nu > 0)) { g_tg_create_error = "Require n>=8 and finite positive nu"; return GM_EVALUE; }
  if (precision != 0 && precision != 1) { g_tg_create_error = "precision must be 0 or 1"; return GM_EVALUE; }
  auto t = std::make_unique<gm_tg>();
  t->n = n;
  t->nu = nu;
  t->h = 2 * 3.141592653589793 / n;
  t->precision = precision;
  int rc = tg_guard(t.get(), [&] {
    TG_CK(cudaStreamCreateWithFlags(&t->st, cudaStreamNonBlocking));
    t->plan = make_plan(n, precision == 0);
    std::vector<double> tw = plan_twiddles(t->plan);
    t->tw64.alloc(tw.size());
    TG_CK(cudaMemcpy(t->tw64.p, tw.data(), tw.size() * sizeof(double), cudaMemcpyHostToDevice));
    std::vector<float> tw32(tw.begin(), tw.end());
    t->tw32.alloc(tw32.size());
    TG_CK(cudaMemcpy(t->tw32.p, tw32.data(), tw32.size() * sizeof(float), cudaMemcpyHostToDevice));
    std::vector<double> s2(n);
    for (int k = 0; k < n; ++k) s2[k] = std::pow(std::sin(3.141592653589793 * k / n), 2);
    t->s2_64.alloc(n);
    TG_CK(cudaMemcpy(t->s2_64.p, s2.data(), n * sizeof(double), cudaMemcpyHostToDevice));
    std::vector<float> s2f(s2.begin(), s2.end());
    t->s2_32.alloc(n);
    TG_CK(cudaMemcpy(t->s2_32.p, s2f.data(), n * sizeof(float), cudaMemcpyHostToDevice));
    int optin = 0;
    TG_CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, 0));
    int dyn = optin;
    // the limit is a process-wide attribute of the kernel shared by every handle: the device
    // maximum, so that a smaller handle created later cannot lower it below a larger one's need
    for (auto f : {(const void*)k_tg_rows_fwd<float, LINE_REAL>, (const void*)k_tg_rows_fwd<float, LINE_DIV>,
                   (const void*)k_tg_rows_fwd<float, LINE_PRES>, (const void*)k_tg_rows_fwd<float, LINE_HRES>,
                   (const void*)k_tg_rows_fwd<double, LINE_PAIR>,
                   (const void*)k_tg_rows_fwd<double, LINE_UV>, (const void*)k_tg_rows_inv<float, LINE_REAL>,
                   (const void*)k_tg_rows_inv<double, LINE_PAIR>, (const void*)k_tg_rows_inv<double, LINE_UV>,
                   (const void*)k_tg_cols<float>, (const void*)k_tg_cols<double>}) {
      cudaFuncAttributes fa;
      TG_CK(cudaFuncGetAttributes(&fa, f));
      const int d = optin - (int)fa.sharedSizeBytes;
      dyn = std::min(dyn, d);
      TG_CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, d));
    }
    if (tg_smem<double>(n, t->plan.tw_len, 1) > (size_t)dyn) throw TgError(GM_EVALUE, "grid too large for the row transforms");
    // Threads of a transform and transforms of a block, by sweeps of both over n = 128..4096 (us a step).
    // FP64: one transform a block (smaller blocks spread evenly over the SMs; column accesses of 16 bytes
    // cost less than that gains: n = 512 328 -> 257, 700 1074 -> 796, 1024 884 -> 853, 2048 3550 -> 3272
    // against four or two) with a thread per radix-4 butterfly, 128 to 256 but no more than n / 2
    // (n = 250: 32 threads 232, 64 147, 128 135; 2048: 256 3272, 512 3452).
    // FP32: powers of two from 512 a thread per radix-8 butterfly and four transforms (512: 417 against
    // 430 with 128 x 2); else some 128 threads, as one warp a transform leaves the chip idle (250:
    // 32 x 4 248, 128 x 2 191) or a thread per radix-5 butterfly (700: 96 x 4 1062, 192 x 2 946), two a block.
    auto r32 = [](int v) { return std::max(32, (v + 31) / 32 * 32); };
    const bool octal = n >= 512 && (n & (n - 1)) == 0;
    t->gt[1] = std::max(r32(n / 8), std::min(r32(n / 2), std::max(128, std::min(256, r32(n / 4)))));
    t->gt[0] = octal ? r32(n / 8) : std::min(r32(n / 2), std::max(128, r32(n / 5)));
    for (int d = 0; d < 2; ++d) {
      t->gt[d] = std::min(512, t->gt[d]);
      auto need = [&](int g) { return d ? tg_smem<double>(n, t->plan.tw_len, g) : tg_smem<float>(n, t->plan.tw_len, g); };
      for (int g = 2; d == 0 && g <= (octal ? 4 : 2); g *= 2)
        if (t->gt[d] * g <= 512 && need(g) <= (size_t)dyn) t->gpb[d] = g;
      t->smem[d] = need(t->gpb[d]);
    }
    const int64_t nn = (int64_t)n * n;
    for (Buf<double>* b : {&t->q, &t->qn, &t->hist, &t->now, &t->rhs, &t->star, &t->mid, &t->half_q, &t->action,
                           &t->proj}) {
      b->alloc(2 * nn);
      TG_CK(cudaMemset(b->p, 0, 2 * nn * sizeof(double)));
    }
    for (Buf<double>* b : {&t->phalf, &t->phalf_n, &t->pout, &t->phi, &t->inc, &t->div}) {
      b->alloc(nn);
      TG_CK(cudaMemset(b->p, 0, nn * sizeof(double)));
    }
    t->spec.alloc((size_t)nn * 16);
    if (precision == 0) {
      t->sym_p.alloc((size_t)n * (n / 2 + 1));
      t->sym_h.alloc((size_t)n * (n / 2 + 1));
      k_tg_symbol<<<grid_for((int64_t)n * (n / 2 + 1)), PT, 0, t->st>>>(n, t->s2_64.p, 0, t->h * t->h, 0.0, t->sym_p.p);
      gmk::kernel_launch_adjust(1);
      TG_CK(cudaGetLastError());
    }
    t->red.alloc(RED_N);
    TG_CK(cudaMallocHost(&t->host_red, RED_W * sizeof(unsigned long long)));
    TG_CK(cudaMemset(t->red.p, 0, RED_N * sizeof(unsigned long long)));
  });
  if (rc != GM_OK) { g_tg_create_error = t->err; return rc; }
  *out = t.release();
  return GM_OK;
}

int gm_tg_destroy(gm_tg* t) {
  if (!t) return GM_OK;
  if (t->st) {
    cudaStreamSynchronize(t->st);
    cudaStreamDestroy(t->st);
  }
  delete t;
  return GM_OK;
}

const char* gm_tg_last_error(const gm_tg* t) { return t ? t->err.c_str() : g_tg_create_error.c_str(); }

int gm_tg_set_state(gm_tg* t, const double* q, const double* p) {
  if (!t || !q || !p) return GM_EVALUE;
  return tg_guard(t, [&] {
    const int64_t nn = (int64_t)t->n * t->n;
    TG_CK(cudaMemcpyAsync(t->q.p, q, 2 * nn * sizeof(double), cudaMemcpyDefault, t->st));
    TG_CK(cudaMemcpyAsync(t->phalf.p, p, nn * sizeof(double), cudaMemcpyDefault, t->st));
    TG_CK(cudaMemcpyAsync(t->pout.p, t->phalf.p, nn * sizeof(double), cudaMemcpyDeviceToDevice, t->st));
    TG_CK(cudaStreamSynchronize(t->st));
    t->has_history = false;
    t->prev_dt = 0;
  });
}

int gm_tg_get_state(gm_tg* t, double* q, double* p_half, double* p_out) {
  if (!t) return GM_EVALUE;
  return tg_guard(t, [&] {
    const int64_t nn = (int64_t)t->n * t->n;
    if (q) TG_CK(cudaMemcpyAsync(q, t->q.p, 2 * nn * sizeof(double), cudaMemcpyDefault, t->st));
    if (p_half) TG_CK(cudaMemcpyAsync(p_half, t->phalf.p, nn * sizeof(double), cudaMemcpyDefault, t->st));
    if (p_out) TG_CK(cudaMemcpyAsync(p_out, t->pout.p, nn * sizeof(double), cudaMemcpyDefault, t->st));
    TG_CK(cudaStreamSynchronize(t->st));
  });
}

int gm_tg_held_sweeps(const gm_tg* t, int32_t held[4], int64_t* repeats) {
  if (!t) return GM_EVALUE;
  for (int s = 0; held && s < NSLOT; ++s) held[s] = t->held[s].n;
  if (repeats) *repeats = t->repeats;
  return GM_OK;
}

int gm_tg_step(gm_tg* t, double dt, int32_t n_steps, double* max_divergence) {
  if (!t || n_steps <= 0 || !(std::isfinite(dt) && dt > 0)) {
    if (t) t->err = "Finite fields and a positive timestep are required";
    return GM_EVALUE;
  }
  return tg_guard(t, [&] {
    double md = max_divergence ? *max_divergence : 0.0;
    tg_steps(t, dt, n_steps, &md);
    if (max_divergence) *max_divergence = md;
  });
}

}  // extern "C"
