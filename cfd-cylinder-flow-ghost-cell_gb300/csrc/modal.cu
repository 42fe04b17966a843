// Snapshot POD (method of snapshots, postprocessing/modal_analysis.py:17-98) on the GPU.
//
// For M snapshots of N points (rows of X):
//   mean       the time average of every point, summed over the snapshots in order (the order
//              numpy's mean along axis 0 adds them), so it equals the reference bit for bit;
//   X'         X - mean, kept on the device;
//   C          X' X'^T / M, an M x M Gram matrix: 16 x 16 output tiles of the upper triangle, the
//              point range split over blocks (each block accumulates its slice in FP64 from
//              shared-memory tiles), the slices then summed in a fixed order;
// the host takes the eigen-decomposition of C (M is small), and the device forms
//   phi_i      = X'^T v_i / sigma_i, one thread per point for a group of modes;
//   a_i        = X' phi_i, dot products over the points (per-slice partials, fixed-order sums).
// All arithmetic is FP64.  Input snapshots may be host or device memory.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/ghostmac.h"

namespace gmk {
void kernel_launch_adjust(long long delta);
}

struct gm_pod {
  int M = 0;
  int64_t N = 0;
  double* X = nullptr;       // M x N fluctuations
  double* mean = nullptr;    // N
  double* part = nullptr;    // Gram / coefficient partial sums
  size_t part_n = 0;
  double* C = nullptr;       // M x M
  double* V = nullptr;       // M x k eigenvector columns (row s: snapshot s)
  double* modes = nullptr;   // k x N
  double* coef = nullptr;    // k x M
  int kcap = 0;
  std::string err;
};

namespace {

constexpr int MAXM = 4096;

__global__ void k_pod_mean(const double* __restrict__ X, int M, int64_t N, double* __restrict__ mean,
                           double* __restrict__ Xp) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= N) return;
  double s = 0.0;
  for (int i = 0; i < M; ++i) s += X[(int64_t)i * N + p];
  const double m = s / (double)M;
  mean[p] = m;
  for (int i = 0; i < M; ++i) Xp[(int64_t)i * N + p] = X[(int64_t)i * N + p] - m;
}

// The Gram matrix is bound by the FP64 pipe (M (M + 1) / 2 fused multiply-adds a point).  One
// block forms a 16 x 16 tile of the upper triangle over one slice of the points: 16-wide tiles
// waste little on the diagonal (5,376 products a point for M = 96, of 4,656 needed; 32-wide tiles
// 6,144), and the slice count fills the GPU whatever M and N are (GRAM_BLOCKS blocks, slices of at
// least GRAM_MIN points), where a fixed slice of 16,384 points left 110 of 152 SMs idle on
// 96 x 80,000 values (5.32 ms, now 0.72 ms: 0.60 T products/s, the FP64 pipe's rate).  Four groups of 64 threads take a quarter of every staged chunk
// each, four outputs a thread, and add their sums in group order.
constexpr int T = 16, KCHUNK = 64, GROUPS = 4;
constexpr int GRAM_BLOCKS = 152 * 8, GRAM_MIN = 512;
__device__ __forceinline__ void tri_tile(int e, int nt, int& bi, int& bj) {  // row-major upper triangle
  bi = 0;
  while (e >= nt - bi) { e -= nt - bi; ++bi; }
  bj = bi + e;
}
__global__ void __launch_bounds__(64 * GROUPS) k_pod_gram(const double* __restrict__ Xp, int M, int64_t N,
                                                          int64_t slice, double* __restrict__ part) {
  __shared__ double a[T][KCHUNK + 1];
  __shared__ double b[T][KCHUNK + 1];
  __shared__ double red[GROUPS - 1][T * T];
  const int nt = (M + T - 1) / T;
  int bi, bj;
  tri_tile(blockIdx.x, nt, bi, bj);
  const int g = threadIdx.x >> 6, t = threadIdx.x & 63, tx = t & 15, ty = t >> 4;  // outputs (ty + 4 q, tx)
  const int64_t p0 = (int64_t)blockIdx.y * slice, p1 = min(N, p0 + slice);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t k0 = p0; k0 < p1; k0 += KCHUNK) {
    const int64_t k = k0 + t;
#pragma unroll
    for (int r = 0; r < T; r += GROUPS) {
      const int gi = bi * T + r + g, gj = bj * T + r + g;
      a[r + g][t] = (gi < M && k < p1) ? Xp[(int64_t)gi * N + k] : 0.0;
      b[r + g][t] = (gj < M && k < p1) ? Xp[(int64_t)gj * N + k] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < KCHUNK / GROUPS; ++kk) {
      const int c = g * (KCHUNK / GROUPS) + kk;
      const double bv = b[tx][c];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = fma(a[ty + 4 * q][c], bv, acc[q]);
    }
    __syncthreads();
  }
  if (g > 0)
#pragma unroll
    for (int q = 0; q < 4; ++q) red[g - 1][(ty + 4 * q) * T + tx] = acc[q];
  __syncthreads();
  if (g == 0) {
    double* o = part + ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * T * T;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = (ty + 4 * q) * T + tx;
      double v = acc[q];
      for (int w = 0; w < GROUPS - 1; ++w) v += red[w][e];
      o[e] = v;
    }
  }
}

// C[i][j] = C[j][i] = (sum over slices in order) / M; block e: tile e of the upper triangle
__global__ void __launch_bounds__(T * T) k_pod_gram_fold(const double* __restrict__ part, int M, int nslice,
                                                         double* __restrict__ C) {
  const int nt = (M + T - 1) / T;
  int bi, bj;
  tri_tile(blockIdx.x, nt, bi, bj);
  const int i = bi * T + threadIdx.x / T, j = bj * T + threadIdx.x % T;
  if (i >= M || j >= M || j < i) return;
  double s = 0.0;
#pragma unroll 8
  for (int sl = 0; sl < nslice; ++sl) s += part[((int64_t)sl * gridDim.x + blockIdx.x) * T * T + threadIdx.x];
  const double c = s / (double)M;
  C[(int64_t)i * M + j] = c;
  C[(int64_t)j * M + i] = c;
}

// Modes and coefficients are FP64-bound as well (M k fused multiply-adds a point each).  Both take
// the k modes in groups of QB <= 8, k split evenly (10 modes: 5 + 5), so that a value of X' is
// loaded once for QB products held in registers and no product is padding.
constexpr int QMAX = 8;
int mode_groups(int k) { return (k + QMAX - 1) / QMAX; }
int mode_width(int k) { return (k + mode_groups(k) - 1) / mode_groups(k); }

// modes[q][p] = sum_s X'[s][p] V[s][q] / sigma[q] (zero where sigma <= 1e-12), one thread a point
// (one mode at a time re-read X' for every mode: 192 us on 96 x 80,000 values and 10 modes, now 158).
template <int QB>
__global__ void k_pod_modes(const double* __restrict__ Xp, int M, int64_t N, const double* __restrict__ V, int k,
                            const double* __restrict__ inv_sigma, double* __restrict__ modes) {
  __shared__ double vs[64][QB];
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int q0 = blockIdx.y * QB;
  double acc[QB];
#pragma unroll
  for (int u = 0; u < QB; ++u) acc[u] = 0.0;
  for (int i0 = 0; i0 < M; i0 += 64) {
    const int ni = min(64, M - i0);
    __syncthreads();
    for (int e = threadIdx.x; e < ni * QB; e += blockDim.x) {
      const int i = e / QB, u = e - i * QB;
      vs[i][u] = q0 + u < k ? V[(int64_t)(i0 + i) * k + q0 + u] : 0.0;
    }
    __syncthreads();
    if (p < N)
#pragma unroll 8
      for (int i = 0; i < ni; ++i) {
        const double x = Xp[(int64_t)(i0 + i) * N + p];
#pragma unroll
        for (int u = 0; u < QB; ++u) acc[u] += x * vs[i][u];
      }
  }
  if (p >= N) return;
#pragma unroll
  for (int u = 0; u < QB; ++u)
    if (q0 + u < k) modes[(int64_t)(q0 + u) * N + p] = inv_sigma[q0 + u] > 0 ? acc[u] * inv_sigma[q0 + u] : 0.0;
}

// part[slice][s][q] = sum over the slice's points of X'[s][p] modes[q][p]: a block takes 32 snapshots
// (its lanes) x QB modes, its eight warps an eighth of every staged chunk each, added in warp order
// (one output at a time with a block reduction each took 1.33 ms on the sizes above, now 0.16 ms).
constexpr int CR = 32, CK = 64, CW = 8;
template <int QB>
__global__ void __launch_bounds__(32 * CW) k_pod_coef_part(const double* __restrict__ Xp, int M, int64_t N,
                                                           const double* __restrict__ modes, int k, int64_t slice,
                                                           double* __restrict__ part) {
  __shared__ double a[CR][CK + 1];
  __shared__ double b[QB][CK];
  __shared__ double red[CW][QB][CR];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int s0 = blockIdx.x * CR, q0 = blockIdx.y * QB;
  const int64_t p0 = (int64_t)blockIdx.z * slice, p1 = min(N, p0 + slice);
  double acc[QB];
#pragma unroll
  for (int u = 0; u < QB; ++u) acc[u] = 0.0;
  for (int64_t k0 = p0; k0 < p1; k0 += CK) {
#pragma unroll
    for (int e = 0; e < CR * CK / (32 * CW); ++e) {
      const int f = e * 32 * CW + threadIdx.x, r = f / CK, c = f % CK;
      a[r][c] = (s0 + r < M && k0 + c < p1) ? Xp[(int64_t)(s0 + r) * N + k0 + c] : 0.0;
    }
    for (int f = threadIdx.x; f < QB * CK; f += 32 * CW) {
      const int r = f / CK, c = f % CK;
      b[r][c] = (q0 + r < k && k0 + c < p1) ? modes[(int64_t)(q0 + r) * N + k0 + c] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < CK / CW; ++kk) {
      const int c = w * (CK / CW) + kk;
      const double x = a[lane][c];
#pragma unroll
      for (int u = 0; u < QB; ++u) acc[u] += x * b[u][c];
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < QB; ++u) red[w][u][lane] = acc[u];
  __syncthreads();
  for (int e = threadIdx.x; e < QB * CR; e += 32 * CW) {
    const int u = e / CR, r = e % CR;
    if (s0 + r >= M || q0 + u >= k) continue;
    double t = 0.0;
    for (int v = 0; v < CW; ++v) t += red[v][u][r];
    part[((int64_t)blockIdx.z * M + s0 + r) * k + q0 + u] = t;
  }
}
// coef[q][s]: the slices' sums, one warp an output (lanes over slices, fixed butterfly)
__global__ void k_pod_coef_fold(const double* __restrict__ part, int nb, int M, int k, double* __restrict__ coef) {
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (e >= M * k) return;
  const int s = e / k, q = e - s * k;
  double t = 0.0;
  for (int b = lane; b < nb; b += 32) t += part[((int64_t)b * M + s) * k + q];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) coef[(int64_t)q * M + s] = t;
}

template <int QB>
void launch_modes(const double* Xp, int M, int64_t N, const double* V, int k, const double* inv_sigma, double* modes,
                  int64_t slice, int nslice, double* part, cudaStream_t st) {
  const unsigned ng = (unsigned)mode_groups(k);
  k_pod_modes<QB><<<dim3((unsigned)((N + 255) / 256), ng), 256, 0, st>>>(Xp, M, N, V, k, inv_sigma, modes);
  k_pod_coef_part<QB><<<dim3((unsigned)((M + CR - 1) / CR), ng, (unsigned)nslice), 32 * CW, 0, st>>>(Xp, M, N, modes, k,
                                                                                                    slice, part);
}

// slices of the point range that give about GRAM_BLOCKS blocks over `tiles` tiles, of at least
// GRAM_MIN points (a multiple of the staged chunk)
int64_t slice_points(int64_t N, int64_t tiles) {
  const int64_t want = std::max<int64_t>(1, GRAM_BLOCKS / tiles);
  int64_t s = std::max<int64_t>((N + want - 1) / want, GRAM_MIN);
  s = std::max<int64_t>(s, (N + 65534) / 65535);
  return (s + KCHUNK - 1) / KCHUNK * KCHUNK;
}

bool is_device(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

int fail(gm_pod* p, int code, const std::string& msg) {
  p->err = msg;
  return code;
}
int cuda_fail(gm_pod* p, cudaError_t e) {
  cudaGetLastError();
  return fail(p, GM_ECUDA, cudaGetErrorString(e));
}
template <typename Tp>
cudaError_t grow(Tp** ptr, size_t& have, size_t need) {
  if (have >= need && *ptr) return cudaSuccess;
  if (*ptr) cudaFree(*ptr);
  *ptr = nullptr;
  have = 0;
  cudaError_t e = cudaMalloc(ptr, need * sizeof(Tp));
  if (e == cudaSuccess) have = need;
  return e;
}

}  // namespace

extern "C" {

int gm_pod_create(int32_t n_snapshots, int64_t n_points, gm_pod** out) {
  if (!out) return GM_EVALUE;
  *out = nullptr;
  if (n_snapshots < 1 || n_snapshots > MAXM || n_points < 1) return GM_EVALUE;
  gm_pod* p = new gm_pod();
  p->M = n_snapshots;
  p->N = n_points;
  cudaError_t e = cudaMalloc(&p->X, (size_t)p->M * p->N * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&p->mean, (size_t)p->N * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&p->C, (size_t)p->M * p->M * sizeof(double));
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (p->X) cudaFree(p->X);
    if (p->mean) cudaFree(p->mean);
    if (p->C) cudaFree(p->C);
    delete p;
    return GM_ECUDA;
  }
  *out = p;
  return GM_OK;
}

int gm_pod_destroy(gm_pod* p) {
  if (!p) return GM_OK;
  for (double* q : {p->X, p->mean, p->part, p->C, p->V, p->modes, p->coef})
    if (q) cudaFree(q);
  delete p;
  return GM_OK;
}

const char* gm_pod_last_error(const gm_pod* p) { return p ? p->err.c_str() : "null handle"; }

int gm_pod_gram(gm_pod* p, const double* snapshots, double* mean, double* gram, void* stream) {
  if (!p || !snapshots || !mean || !gram) return p ? fail(p, GM_EVALUE, "null argument") : GM_EVALUE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int M = p->M;
  const int64_t N = p->N;
  const size_t bytes = (size_t)M * N * sizeof(double);
  // the snapshots go through the fluctuation buffer: staged there first when they are host data
  const double* X = snapshots;
  if (!is_device(snapshots)) {
    if (cudaError_t e = cudaMemcpyAsync(p->X, snapshots, bytes, cudaMemcpyHostToDevice, st)) return cuda_fail(p, e);
    X = p->X;
  }
  k_pod_mean<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(X, M, N, p->mean, p->X);
  const int64_t nt = (M + T - 1) / T, tiles = nt * (nt + 1) / 2;
  const int64_t slice = slice_points(N, tiles), nslice = (N + slice - 1) / slice;
  if (cudaError_t e = grow(&p->part, p->part_n, (size_t)(nslice * tiles * T * T))) return cuda_fail(p, e);
  k_pod_gram<<<dim3((unsigned)tiles, (unsigned)nslice), 64 * GROUPS, 0, st>>>(p->X, M, N, slice, p->part);
  k_pod_gram_fold<<<(unsigned)tiles, T * T, 0, st>>>(p->part, M, (int)nslice, p->C);
  gmk::kernel_launch_adjust(3);
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(p, e);
  cudaError_t e = cudaMemcpyAsync(mean, p->mean, N * sizeof(double), cudaMemcpyDefault, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(gram, p->C, (size_t)M * M * sizeof(double), cudaMemcpyDefault, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(p, e);
  return GM_OK;
}

int gm_pod_modes(gm_pod* p, const double* eigvecs, const double* sigma, int32_t k, double* modes, double* coeffs,
                 void* stream) {
  if (!p || !eigvecs || !sigma || !modes || !coeffs) return p ? fail(p, GM_EVALUE, "null argument") : GM_EVALUE;
  if (k < 1 || k > p->M) return fail(p, GM_EVALUE, "mode count must be between 1 and the snapshot count");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int M = p->M;
  const int64_t N = p->N;
  if (k > p->kcap) {
    for (double** q : {&p->V, &p->modes, &p->coef})
      if (*q) { cudaFree(*q); *q = nullptr; }
    cudaError_t e = cudaMalloc(&p->V, ((size_t)M * k + k) * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&p->modes, (size_t)k * N * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&p->coef, (size_t)k * M * sizeof(double));
    if (e != cudaSuccess) return cuda_fail(p, e);
    p->kcap = k;
  }
  std::vector<double> host((size_t)M * k + k);
  std::memcpy(host.data(), eigvecs, (size_t)M * k * sizeof(double));
  for (int q = 0; q < k; ++q) host[(size_t)M * k + q] = sigma[q] > 1e-12 ? 1.0 / sigma[q] : 0.0;
  if (cudaError_t e = cudaMemcpyAsync(p->V, host.data(), host.size() * sizeof(double), cudaMemcpyHostToDevice, st))
    return cuda_fail(p, e);
  const int64_t slice = slice_points(N, (int64_t)((M + CR - 1) / CR) * mode_groups(k)), nslice = (N + slice - 1) / slice;
  if (cudaError_t e = grow(&p->part, p->part_n, (size_t)(nslice * M * k))) return cuda_fail(p, e);
  auto* launch = launch_modes<1>;
  switch (mode_width(k)) {
    case 1: break;
    case 2: launch = launch_modes<2>; break;
    case 3: launch = launch_modes<3>; break;
    case 4: launch = launch_modes<4>; break;
    case 5: launch = launch_modes<5>; break;
    case 6: launch = launch_modes<6>; break;
    case 7: launch = launch_modes<7>; break;
    default: launch = launch_modes<8>; break;
  }
  launch(p->X, M, N, p->V, k, p->V + (size_t)M * k, p->modes, slice, (int)nslice, p->part, st);
  k_pod_coef_fold<<<(unsigned)(((int64_t)M * k * 32 + 255) / 256), 256, 0, st>>>(p->part, (int)nslice, M, k, p->coef);
  gmk::kernel_launch_adjust(3);
  if (cudaError_t e = cudaGetLastError()) return cuda_fail(p, e);
  cudaError_t e = cudaMemcpyAsync(modes, p->modes, (size_t)k * N * sizeof(double), cudaMemcpyDefault, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(coeffs, p->coef, (size_t)k * M * sizeof(double), cudaMemcpyDefault, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(p, e);
  return GM_OK;
}

}  // extern "C"
