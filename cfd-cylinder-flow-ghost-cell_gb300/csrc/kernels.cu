// Kernels of the ghost-cell AB2/CN step (sm_103a).  See kernels.cuh for the layout.
#include <algorithm>
#include <atomic>
#include <vector>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <utility>

#include "kernels.cuh"
#include "momentum.cuh"

namespace gmk {

static constexpr int TPB = 256;
static constexpr double EPS64 = 2.220446049250313e-16;

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Block-wide max of non-negative doubles (as bits) and optional sum; thread 0 commits atomically.
__device__ void block_commit_max(unsigned long long v, unsigned long long* dst) {
  __shared__ unsigned long long sm[32];
  v = warp_max_u64(v);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sm[wid] = v;
  __syncthreads();
  if (wid == 0) {
    int nw = (blockDim.x + 31) >> 5;
    v = lane < nw ? sm[lane] : 0ull;
    v = warp_max_u64(v);
    if (lane == 0 && v) atomicMax(dst, v);
  }
}
__device__ void block_commit_sum(double v, double* dst) {
  __shared__ double sm[32];
  v = warp_sum(v);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sm[wid] = v;
  __syncthreads();
  if (wid == 0) {
    int nw = (blockDim.x + 31) >> 5;
    v = lane < nw ? sm[lane] : 0.0;
    v = warp_sum(v);
    if (lane == 0 && v != 0.0) atomicAdd(dst, v);
  }
}
// FP32 variant for diagnostics sums of the FP32 mode (FP64 adds issue at 1/64 of the FP32 rate)
__device__ void block_commit_sum_f32(float v, double* dst) {
  __shared__ float smf[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) smf[wid] = v;
  __syncthreads();
  if (wid == 0) {
    int nw = (blockDim.x + 31) >> 5;
    v = lane < nw ? smf[lane] : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0 && v != 0.0f) atomicAdd(dst, f32_to_f64i(v));
  }
}
// |v| as bits with the sign bit cleared, on the integer pipe.  Written as PTX, like the
// exponent test below, so that the compiler cannot turn either back into FP64 instructions
// (fabs, a compare).  With both in PTX the residual kernels measured 8-9 % faster on a GB300.
__device__ __forceinline__ unsigned long long absbits(double v) {
  unsigned long long r;
  asm("and.b64 %0, %1, 0x7fffffffffffffff;" : "=l"(r) : "l"(dbits(v)));
  return r;
}
// |v| (the same value as fabs) on the integer pipe
__device__ __forceinline__ double absd(double v) { return bits2d(absbits(v)); }
// Inf or NaN, by the exponent bits (integer pipe, for the same reason)
__device__ __forceinline__ bool nonfinite_bits(double v) {
  unsigned long long r;
  asm("and.b64 %0, %1, 0x7ff0000000000000;" : "=l"(r) : "l"(dbits(v)));
  return r == 0x7ff0000000000000ull;
}

// Launch as a programmatic dependent of the previous kernel on the stream (its launch overlaps
// that kernel's end; the kernel's gate_open waits for it with griddepcontrol.wait before any
// read).  Used for every step kernel that begins with gate_open: the solve sweeps, the
// momentum right-hand side, the ghost rows, the projection, the defect, the pressure output,
// the maxima and the forces.
// GHOSTMAC_NO_PDL=1 launches them as ordinary stream successors.
static int pdl_mode() {
  static int mode = -1;
  if (mode < 0) {
    const char* e = std::getenv("GHOSTMAC_NO_PDL");
    mode = (e && e[0] == '1') ? 0 : 1;
  }
  return mode;
}
// A kernel behind a conditional node or a join of two streams is launched plainly.
template <typename... KArgs, typename... Args>
static void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                       Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl_mode();
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

static inline unsigned blocks_for(int64_t n, int tpb = TPB) { return (unsigned)((n + tpb - 1) / tpb); }
// Grid of the reduction kernels: grid-stride loops over at most 4 blocks per SM of a GB300,
// so each block commits its partial max/sum with one atomic per quantity.
static inline unsigned reduce_blocks(int64_t n) {
  unsigned b = blocks_for(n);
  return b < 608u ? b : 608u;
}
// Blocks of the residual kernels.  Each block ends with its reductions (a warp-shuffle sum
// costs five adds per thread), so fewer, longer-striding blocks spend less on them.  Measured
// on the 800x820 case: the FP64 residual (sums in FP64) was fastest at 304 blocks, the
// FP32-mode residual (sums in FP32, and the FP64 stencil its only FP64 work) at 608.
static inline unsigned residual_blocks(int64_t n, bool res_f32) {
  const unsigned b = blocks_for(n), cap = res_f32 ? 608u : 304u;
  return b < cap ? b : cap;
}
__device__ __forceinline__ unsigned long long umax64(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

// Host-side count of kernel launches issued by this library (all launchers call note_launch).
static std::atomic<long long> g_launches{0};
static inline void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
long long kernel_launch_count() { return g_launches.load(); }
// Graph capture records launches that have not run yet; the host corrects the count by the
// captured nodes and adds the nodes a graph replay executed.
void kernel_launch_adjust(long long delta) { g_launches.fetch_add(delta, std::memory_order_relaxed); }

// Optional CUDA-event timing of every launch, summed per kernel class (used by the
// benchmark for its per-class breakdown and the dominant kernel's launch time).  Classes:
// 1 x pass, 2 column solves, 3 momentum, 4 residual, 5 boundary chain / Schur GEMV, 6 projection pieces,
// 7 defect / pressure output, 8 ghost rows, 9 forces / maxima, 10 gates and loop control,
// 11 FP32 Jacobi sweeps of the Helmholtz systems, 12 row transforms on the tensor cores.
namespace {
struct KTimer {
  bool on = false;
  std::vector<cudaEvent_t> ev;
  std::vector<int> cls;
  int used = 0;
  std::vector<double> bytes;
  double total_ms[KT_CLASSES] = {};
  double total_bytes[KT_CLASSES] = {};
  long long count[KT_CLASSES] = {};
};
KTimer g_kt;
}  // namespace
// begin and end marks of one launch; the end mark carries the launch's algorithmic bytes
static inline void kt_mark(int cls, cudaStream_t st, double bytes = 0.0) {
  if (!g_kt.on || g_kt.used >= (int)g_kt.ev.size()) return;
  g_kt.cls[g_kt.used] = cls;
  g_kt.bytes[g_kt.used] = bytes;
  cudaEventRecord(g_kt.ev[g_kt.used++], st);
}
void ktimer_enable(int on) {
  if (g_kt.ev.empty()) {
    g_kt.ev.resize(4096);
    g_kt.cls.resize(4096);
    g_kt.bytes.resize(4096);
    for (auto& e : g_kt.ev) cudaEventCreate(&e);
  }
  g_kt.on = on != 0;
  g_kt.used = 0;
  for (int k = 0; k < KT_CLASSES; ++k) { g_kt.total_ms[k] = 0; g_kt.total_bytes[k] = 0; g_kt.count[k] = 0; }
}
// Folds the recorded pairs (begin and end of one launch are consecutive) into the totals;
// the streams must be synchronised.
void ktimer_collect() {
  for (int i = 0; i + 1 < g_kt.used; i += 2) {
    float ms = 0;
    if (cudaEventElapsedTime(&ms, g_kt.ev[i], g_kt.ev[i + 1]) == cudaSuccess) {
      const int c = g_kt.cls[i];
      if (c >= 0 && c < KT_CLASSES) {
        g_kt.total_ms[c] += ms;
        g_kt.total_bytes[c] += g_kt.bytes[i + 1];
        g_kt.count[c] += 1;
      }
    }
  }
  cudaGetLastError();
  g_kt.used = 0;
}
bool ktimer_active() { return g_kt.on; }
void note_launch_ext() { note_launch(); }
void kt_mark_ext(int cls, cudaStream_t st, double bytes) { kt_mark(cls, st, bytes); }
int pdl_mode_ext() { return pdl_mode(); }
void ktimer_read(int cls, double* total_ms, long long* count, double* bytes) {
  const bool ok = cls >= 0 && cls < KT_CLASSES;
  *total_ms = ok ? g_kt.total_ms[cls] : 0.0;
  *count = ok ? g_kt.count[cls] : 0;
  *bytes = ok ? g_kt.total_bytes[cls] : 0.0;
}

// ---------------------------------------------------------------------------
// separable inverse: x pass (rows) and y pass (columns with eigenvalue scaling)
// ---------------------------------------------------------------------------
// Row transforms.  A group of `gthreads` threads (one warp, or whole warps on a named
// barrier) transforms one line group -- two paired lines for the Makhoul and DST-I
// transforms, one line or two (TransformTables::xg_two) for the type-IV transforms -- and a block holds
// `gpb` groups.
// Rows r0 .. r0+nr-1 are transformed.  Masked load with the optional spectral correction
// of the boundary term (YCorr); masked store with the optional epilogue out = add + v.
// shared memory of one line group: the two FFT buffers (the real results go to the buffer the
// FFT does not end in)
template <typename T>
__host__ __device__ inline size_t xpass_group_smem(int type, int n, int lpw) {
  return 2 * (size_t)r2r_buffer_elems(type, n, lpw) * sizeof(cplx<T>);
}
// lengths (complex entries) of the plan's twiddles, the pre- and the post-twiddles of a transform
__host__ __device__ inline int xpass_tw_len(int type, int n, int which, int plan_tw) {
  const int fam = r2r_family(type);
  if (which == 0) return plan_tw;
  if (which == 1) return fam == 2 ? n / 2 : 1;
  return fam == 2 ? n / 2 : (fam == 3 ? 1 : n);
}
template <typename T>
__host__ __device__ inline size_t xpass_tw_bytes(int type, int n, int plan_tw) {
  return ((size_t)(xpass_tw_len(type, n, 0, plan_tw) + xpass_tw_len(type, n, 1, plan_tw) +
                   xpass_tw_len(type, n, 2, plan_tw)) * sizeof(cplx<T>) + 15) / 16 * 16;
}
int xpass_lines(int type, int two) { return r2r_paired(type) || two ? 2 : 1; }
size_t xpass_smem_per_group(int type, int n, bool fp32, int two) {
  const int lpw = xpass_lines(type, two);
  return fp32 ? xpass_group_smem<float>(type, n, lpw) : xpass_group_smem<double>(type, n, lpw);
}
size_t xpass_smem_tables(int type, int n, int plan_tw, bool fp32) {
  return fp32 ? xpass_tw_bytes<float>(type, n, plan_tw) : xpass_tw_bytes<double>(type, n, plan_tw);
}

static constexpr int XB = 4;  // loads batched per thread in the row passes
static constexpr int XT = 8;  // table loads in flight per thread while the tables are staged
// Twiddle tables of one transform type staged into the block's shared memory (read by every
// stage of every group: a global load per stage would put an L2 round trip on each stage's
// critical path).  Each thread has XT loads in flight before its first store, so a table of
// up to XT * blockDim.x entries costs one round trip.  The tables are written once at set-up,
// never by a kernel, so the kernels stage them before waiting on the previous kernel of the
// stream.  Called by all threads of the block; ends with a block barrier.
template <typename T>
__device__ __forceinline__ R2RTables<T> xpass_stage_tables(int type, int n, const FftPlan& plan,
                                                           const R2RTables<T>& tb, unsigned char* smem_raw) {
  const int n0 = xpass_tw_len(type, n, 0, plan.tw_len), n1 = xpass_tw_len(type, n, 1, plan.tw_len);
  const int tot = n0 + n1 + xpass_tw_len(type, n, 2, plan.tw_len);
  cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem_raw);
  for (int q0 = threadIdx.x; q0 < tot; q0 += XT * blockDim.x) {
    cplx<T> v[XT];
#pragma unroll
    for (int u = 0; u < XT; ++u) {
      const int q = q0 + u * blockDim.x;
      if (q < tot) v[u] = q < n0 ? tb.W[q] : (q < n0 + n1 ? tb.pre[q - n0] : tb.post[q - n0 - n1]);
    }
#pragma unroll
    for (int u = 0; u < XT; ++u) {
      const int q = q0 + u * blockDim.x;
      if (q < tot) tw[q] = v[u];
    }
  }
  __syncthreads();
  return R2RTables<T>{tw, tw + n0, tw + n0 + n1};
}

// The line groups of (virtual) block bi: group grp of the block transforms lines
// (bi * gpb + grp) * lpw ... of rows r0 .. r0+nr-1.  Groups past the end return at once; every
// group synchronises on its own named barrier only, so a block may run this for several bi in turn.
template <typename T, typename TI, typename TO, bool TWO>
__device__ __forceinline__ void xpass_block(int bi, int n, int r0, int nr, int type, const FftPlan& plan,
                                            const R2RTables<T>& ts, const TI* __restrict__ in, int64_t ibase,
                                            int64_t ipitch, const uint8_t* __restrict__ icls, TO* __restrict__ out,
                                            int64_t obase, int64_t opitch, const uint8_t* __restrict__ ocls,
                                            const double* __restrict__ add, const YCorr<T>& corr, int gthreads,
                                            int gpb, unsigned char* smem_raw) {
  const int lpw = r2r_paired(type) || TWO ? 2 : 1;
  const int grp = threadIdx.x / gthreads, tid = threadIdx.x - grp * gthreads;
  const int l0 = (bi * gpb + grp) * lpw;
  if (grp >= gpb || l0 >= nr) return;
  const int nl = min(lpw, nr - l0);
  unsigned char* mine = smem_raw + xpass_tw_bytes<T>(type, n, plan.tw_len) + (size_t)grp * xpass_group_smem<T>(type, n, lpw);
  cplx<T>* a = reinterpret_cast<cplx<T>*>(mine);
  cplx<T>* b = a + r2r_buffer_elems(type, n, lpw);
  const Grp G{tid, gthreads, grp + 1};
  // per line (at most two): input row offset and the band correction (band row that scales or
  // is the correction, decay factors of this row: nullptr inside the band); scalars selected by
  // the line index, not an indexed array (that would go to local memory)
  int64_t irow0 = 0, irow1 = 0;
  const T *cb0 = nullptr, *cb1 = nullptr, *cf0 = nullptr, *cf1 = nullptr;
  for (int l = 0; l < nl; ++l) {
    const int r = r0 + l0 + l;
    const int64_t ir = ibase + (int64_t)r * ipitch;
    const T* cb = nullptr;
    const T* cf = nullptr;
    if (corr.band) {
      if (r < corr.j0) {
        cb = corr.band;
        cf = corr.phi + (int64_t)r * n;
      } else if (r > corr.j1) {
        cb = corr.band + (int64_t)(corr.j1 - corr.j0) * n;
        cf = corr.psi + (int64_t)(r - corr.j1 - 1) * n;
      } else {
        cb = corr.band + (int64_t)(r - corr.j0) * n;
      }
    }
    if (l == 0) { irow0 = ir; cb0 = cb; cf0 = cf; }
    else { irow1 = ir; cb1 = cb; cf1 = cf; }
  }
  // element e of line l: masked input minus the correction
  auto x = [&](int l, int e) -> T {
    const int64_t o = (l == 0 ? irow0 : irow1) + e;
    const T* cb = l == 0 ? cb0 : cb1;
    const T* cf = l == 0 ? cf0 : cf1;
    const TI v = in[o];
    const uint8_t mk = icls ? icls[o] : (uint8_t)CLS_ACTIVE;
    const T cv = cb ? (cf ? cf[e] * cb[e] : cb[e]) : (T)0;
    return ((mk & CLS_ACTIVE) ? cvt_to<T>(v) : (T)0) - cv;
  };
  const T* stage = r2r_lines<T, TWO>(type, n, nl, a, b, plan, ts, G, x);
  for (int l = 0; l < nl; ++l) {
    const int64_t row = obase + (int64_t)(r0 + l0 + l) * opitch;
    for (int e0 = tid; e0 < n; e0 += XB * gthreads) {
      uint8_t mk[XB];
      double ad[XB];
#pragma unroll
      for (int u = 0; u < XB; ++u) {
        const int64_t fo = row + e0 + u * gthreads;
        if (e0 + u * gthreads < n) {
          mk[u] = ocls ? ocls[fo] : (uint8_t)CLS_ACTIVE;
          ad[u] = add ? add[fo] : 0.0;
        }
      }
#pragma unroll
      for (int u = 0; u < XB; ++u) {
        const int e = e0 + u * gthreads;
        if (e >= n) continue;
        const int64_t fo = row + e;
        if (!(mk[u] & CLS_ACTIVE)) {
          out[fo] = (TO)0;
        } else {
          const T v = stage[l * n + e];
          out[fo] = add ? cvt_to<TO>(ad[u] + cvt_to<double>(v)) : cvt_to<TO>(v);
        }
      }
    }
  }
}

template <typename T, typename TI, typename TO, bool TWO>
__global__ void k_xpass(int n, int r0, int nr, int type, FftPlan plan, R2RTables<T> tb, const TI* __restrict__ in,
                        int64_t ibase, int64_t ipitch, const uint8_t* __restrict__ icls, TO* __restrict__ out,
                        int64_t obase, int64_t opitch, const uint8_t* __restrict__ ocls, const double* __restrict__ add,
                        YCorr<T> corr, int gthreads, int gpb, Gate gate) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const R2RTables<T> ts = xpass_stage_tables<T>(type, n, plan, tb, smem_raw);
  if (!gate_open(gate)) return;
  xpass_block<T, TI, TO, TWO>(blockIdx.x, n, r0, nr, type, plan, ts, in, ibase, ipitch, icls, out, obase, opitch, ocls,
                         add, corr, gthreads, gpb, smem_raw);
}

template <typename T, typename TI, typename TO>
void launch_xpass(const TransformTables& tt, bool inverse, int r0, int nr, const TI* in, int64_t ibase,
                  int64_t ipitch, const uint8_t* icls, TO* out, int64_t obase, int64_t opitch, const uint8_t* ocls,
                  const double* add, const YCorr<T>& corr, const Gate& gate, cudaStream_t st) {
  if (nr <= 0) return;
  using C = cplx<T>;
  const int type = inverse ? tt.tx_inv : tt.tx_fwd;
  R2RTables<T> tb{(const C*)tt.Wx, (const C*)(inverse ? tt.prex_inv : tt.prex),
                  (const C*)(inverse ? tt.postx_inv : tt.postx)};
  const int lpw = xpass_lines(type, tt.xg_two);
  const int per_block = tt.xg_pb * lpw;
  const unsigned grid = (unsigned)((nr + per_block - 1) / per_block);
  note_launch();
  kt_mark(1, st);
  auto* kernel = k_xpass<T, TI, TO, false>;
  if constexpr (sizeof(T) == 8)
    if (lpw == 2 && !r2r_paired(type)) kernel = k_xpass<T, TI, TO, true>;
  launch_pdl(kernel, dim3(grid), dim3(tt.xg_threads * tt.xg_pb), tt.smem_x, st, tt.n, r0, nr, type, tt.plan_x, tb, in, ibase,
             ipitch, icls, out, obase, opitch, ocls, add, corr, tt.xg_threads, tt.xg_pb, gate);
  // algorithmic bytes: one read and one write per point, class maps, the added field and the
  // correction band (tables of the decay factors once per point)
  kt_mark(1, st, (double)nr * tt.n * (sizeof(TI) + sizeof(TO) + (icls ? 1 : 0) + (ocls ? 1 : 0) + (add ? 8 : 0) +
                                      (corr.band ? sizeof(T) : 0)));
}
template void launch_xpass<double, double, double>(const TransformTables&, bool, int, int, const double*, int64_t,
                                                   int64_t, const uint8_t*, double*, int64_t, int64_t,
                                                   const uint8_t*, const double*, const YCorr<double>&, const Gate&,
                                                   cudaStream_t);
template void launch_xpass<float, double, float>(const TransformTables&, bool, int, int, const double*, int64_t,
                                                 int64_t, const uint8_t*, float*, int64_t, int64_t, const uint8_t*,
                                                 const double*, const YCorr<float>&, const Gate&, cudaStream_t);
template void launch_xpass<float, float, float>(const TransformTables&, bool, int, int, const float*, int64_t,
                                                int64_t, const uint8_t*, float*, int64_t, int64_t, const uint8_t*,
                                                const double*, const YCorr<float>&, const Gate&, cudaStream_t);
template void launch_xpass<float, float, double>(const TransformTables&, bool, int, int, const float*, int64_t,
                                                 int64_t, const uint8_t*, double*, int64_t, int64_t, const uint8_t*,
                                                 const double*, const YCorr<float>&, const Gate&, cudaStream_t);

// ---------------------------------------------------------------------------
// y direction of the separable inverse: for every x-mode kx the column system
// (L_y + lambda_x(kx)) z = s / (2 nx) (pressure) or ((1 - c lambda_x) - c L_y) z = s / (2 nx)
// (Helmholtz) is tridiagonal with a constant off-diagonal.  It is solved by a
// partition method: P chunks of inner rows separated by interface rows; each
// thread runs Thomas on one chunk with precomputed pivots, one thread per column
// solves the interface system, and the chunk solutions take the spike
// corrections.  Tables (rows x cols, same layout as the spectral array):
//   inner rows:     t0 = 1/pivot, t1 = left spike v, t2 = right spike w
//   interface rows: t0 = 1/pivot, t1 = sub-diagonal, t2 = sup/pivot of the interface system
// The data and every coefficient of the two recurrences are staged in shared memory
// first, so the dependent chains wait on shared-memory latency only.
// ---------------------------------------------------------------------------
template <typename T, int L>
__device__ __forceinline__ void ysolve_body(int n /*rows*/, int cols, const YChunks& ch, T gamma, T scale,
                                            const T* __restrict__ t0, const T* __restrict__ t1,
                                            const T* __restrict__ t2, T* __restrict__ S, int bid) {
  // L consecutive columns per block (L a power of two: thread -> (column, row/chunk) by shifts)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ns = n | 1;                                  // odd stride between the columns
  T* col = reinterpret_cast<T*>(smem_raw);              // L x ns values
  T* piv = col + (size_t)L * ns;                         // L x ns reciprocal pivots
  T* s1 = piv + (size_t)L * ns;                          // spikes at the interface rows: L x YCHUNK_MAX left (t1),
  T* s2 = s1 + L * YCHUNK_MAX;                           // right (t2)
  uint8_t* chunk_of = reinterpret_cast<uint8_t*>(s2 + L * YCHUNK_MAX);  // of each row; 255 at an interface row
  const int c0 = bid * L;
  const int P = ch.P;
  const int l = threadIdx.x & (L - 1);                   // column of this thread
  const int rsub = threadIdx.x / L;                      // row offset (load/store), chunk (solve)
  const int rstep = blockDim.x / L;
  const bool colok = c0 + l < cols;
  const int64_t cc = c0 + l;
  // load the column values and pivots in one phase, 2 x 8 loads in flight per thread, so that the
  // recurrences wait on shared memory only.  The spikes of the inner rows are read where they are used,
  // once, in the store phase: staged here as well they doubled a block's shared memory, and at 800x820
  // eight FP64 columns were one block an SM whose loads, recurrences and stores did not overlap
  // (35 us a solve, now 31; the 400x200 step 277 -> 271 us)
  for (int e0 = rsub; e0 < n; e0 += 8 * rstep) {
    T sv[8], pvv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * rstep;
      if (colok && e < n) {
        const int64_t o = (int64_t)e * cols + cc;
        sv[u] = S[o];
        pvv[u] = t0[o];
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * rstep;
      if (colok && e < n) {
        col[l * ns + e] = sv[u] * scale;
        piv[l * ns + e] = pvv[u];
      }
    }
  }
  if (colok && rsub < P - 1) {
    const int64_t o = (int64_t)(ch.end[rsub] + 1) * cols + cc;
    s1[l * YCHUNK_MAX + rsub] = t1[o];
    s2[l * YCHUNK_MAX + rsub] = t2[o];
  }
  if (l == 0 && rsub < P) {
    for (int j = ch.start[rsub]; j <= ch.end[rsub]; ++j) chunk_of[j] = (uint8_t)rsub;
    if (rsub < P - 1) chunk_of[ch.end[rsub] + 1] = 255;
  }
  __syncthreads();
  const int p = rsub;
  const bool work = colok && p < P;
  int a = 0, b = -1;
  if (work) { a = ch.start[p]; b = ch.end[p]; }
  T* x = col + l * ns;
  const T* pv = piv + l * ns;
  // phase 1: chunk-local Thomas
  if (work) {
    T prev = 0;
    for (int j = a; j <= b; ++j) {
      prev = (x[j] - gamma * prev) * pv[j];
      x[j] = prev;
    }
    T next = x[b];
    for (int j = b - 1; j >= a; --j) {
      next = x[j] - (gamma * pv[j]) * next;
      x[j] = next;
    }
  }
  __syncthreads();
  // phase 2: interface system, one thread per column (its coefficients are the spike tables at
  // the interface rows)
  if (p == 0 && colok && P > 1) {
    T z = 0;
    for (int q = 0; q < P - 1; ++q) {
      const int e = ch.end[q] + 1;
      const T rhs = x[e] - gamma * x[e - 1] - gamma * x[e + 1];
      z = (rhs - s1[l * YCHUNK_MAX + q] * z) * pv[e];
      x[e] = z;
    }
    T y = 0;
    for (int q = P - 2; q >= 0; --q) {
      const int e = ch.end[q] + 1;
      y = x[e] - s2[l * YCHUNK_MAX + q] * y;
      x[e] = y;
    }
  }
  __syncthreads();
  // phase 3: spike corrections of the inner rows, on the way out
  if (!colok) return;
  for (int e0 = rsub; e0 < n; e0 += 4 * rstep) {
    T v1[4], v2[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * rstep;
      if (P > 1 && e < n) {
        const int64_t o = (int64_t)e * cols + cc;
        v1[u] = t1[o];
        v2[u] = t2[o];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * rstep;
      if (e >= n) continue;
      T v = x[e];
      const int q = P > 1 ? chunk_of[e] : 255;
      if (q != 255) {
        const T yl = q > 0 ? x[ch.end[q - 1] + 1] : (T)0;
        const T yr = q < P - 1 ? x[ch.end[q] + 1] : (T)0;
        v = v - yl * v1[u] - yr * v2[u];
      }
      S[(int64_t)e * cols + cc] = v;
    }
  }
}
template <typename T, int L>
__global__ void k_ysolve(int n /*rows*/, int cols, YChunks ch, T gamma, T scale, const T* __restrict__ t0,
                         const T* __restrict__ t1, const T* __restrict__ t2, T* __restrict__ S, Gate gate) {
  if (!gate_open(gate)) return;
  ysolve_body<T, L>(n, cols, ch, gamma, scale, t0, t1, t2, S, blockIdx.x);
}
size_t ysolve_smem(int rows, int lpb, bool fp32) {
  const size_t esz = fp32 ? 4 : 8;
  // values and pivots, the interface rows' spikes, the rows' chunks
  return (size_t)lpb * ((rows | 1) * 2 + 2 * YCHUNK_MAX) * esz + (size_t)(rows + 15) / 16 * 16;
}

template <typename T>
void launch_ysolve(const TransformTables& tt, int cols, int rows, T* S, const Gate& gate, cudaStream_t st) {
  const unsigned gy = (unsigned)((cols + tt.lpb_y - 1) / tt.lpb_y);
  note_launch();
  kt_mark(2, st);
#define GM_YSOLVE(LL)                                                                                        \
  launch_pdl(k_ysolve<T, LL>, dim3(gy), dim3(tt.threads_y), tt.smem_y, st, rows, cols, tt.ych, (T)tt.gamma,     \
             (T)tt.yscale, (const T*)tt.t0, (const T*)tt.t1, (const T*)tt.t2, S, gate)
  switch (tt.lpb_y) {
    case 2: GM_YSOLVE(2); break;
    case 4: GM_YSOLVE(4); break;
    case 8: GM_YSOLVE(8); break;
    default: GM_YSOLVE(16); break;
  }
#undef GM_YSOLVE
  kt_mark(2, st, (double)rows * cols * sizeof(T) * 5);  // data in and out, three table entries per point
}
template void launch_ysolve<double>(const TransformTables&, int, int, double*, const Gate&, cudaStream_t);
template void launch_ysolve<float>(const TransformTables&, int, int, float*, const Gate&, cudaStream_t);

// Band solve of the boundary term: the x-transformed U c occupies rows j0..j1 only, so per
// x-mode its column solution is the band system (end pivots carry the elimination of the
// rows outside) followed by geometric decay outside the band (phi / psi tables, applied in
// the final x pass).  One thread per column; B holds nb x cols values in place.
template <typename T>
__global__ void k_yband(int nb, int cols, T gamma, T scale, const T* __restrict__ bpiv, T* __restrict__ B,
                        Gate gate) {
  if (!gate_open(gate)) return;
  // the block's columns of B and of the pivots are staged in shared memory first
  // (independent coalesced loads); then one thread per column runs the recurrences
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nc = blockDim.x;
  T* xb = reinterpret_cast<T*>(smem_raw);  // nb x nc
  T* pb = xb + (size_t)nb * nc;
  const int k0 = blockIdx.x * nc;
  const int kk = threadIdx.x;
  if (k0 + kk < cols) {
    for (int j0 = 0; j0 < nb; j0 += 8) {  // 8 rows in flight per thread
      T bv[8], pv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (j0 + u < nb) {
          const int64_t o = (int64_t)(j0 + u) * cols + k0 + kk;
          bv[u] = B[o];
          pv[u] = bpiv[o];
        }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (j0 + u < nb) {
          xb[(j0 + u) * nc + kk] = bv[u] * scale;
          pb[(j0 + u) * nc + kk] = pv[u];
        }
    }
  }
  __syncthreads();
  if (k0 + kk < cols) {
    T z = 0;
    for (int j = 0; j < nb; ++j) {
      z = (xb[j * nc + kk] - gamma * z) * pb[j * nc + kk];
      xb[j * nc + kk] = z;
    }
    T y = z;
    for (int j = nb - 2; j >= 0; --j) {
      y = xb[j * nc + kk] - (gamma * pb[j * nc + kk]) * y;
      xb[j * nc + kk] = y;
    }
  }
  if (k0 + kk < cols)
    for (int j = 0; j < nb; ++j) B[(int64_t)j * cols + k0 + kk] = xb[j * nc + kk];
}
template <typename T>
void launch_yband(const TransformTables& tt, int cols, T* B, const Gate& gate, cudaStream_t st) {
  const int nb = tt.bj1 - tt.bj0 + 1;
  if (nb <= 0) return;
  note_launch();
  kt_mark(2, st);
  // up to 32 columns per block (whole 128/256-byte row segments), shared memory 2 nb x nc values
  const int nc = (int)std::max<size_t>(1, std::min<size_t>(32, (48 * 1024) / (2 * (size_t)nb * sizeof(T))));
  k_yband<T><<<blocks_for(cols, nc), nc, (size_t)2 * nb * nc * sizeof(T), st>>>(nb, cols, (T)tt.gamma, (T)tt.yscale,
                                                                              (const T*)tt.bpiv, B, gate);
  kt_mark(2, st, (double)nb * cols * sizeof(T) * 3);
}
template void launch_yband<double>(const TransformTables&, int, double*, const Gate&, cudaStream_t);
template void launch_yband<float>(const TransformTables&, int, float*, const Gate&, cudaStream_t);

template <typename T, typename TI, typename TO>
__global__ void k_xpass_multi(const __grid_constant__ ArgPack<XpassArgs<T, TI, TO>> p);
template <typename T, int L>
__global__ void k_ysolve_multi(const __grid_constant__ ArgPack<YsolveArgs<T>> p);
__global__ void k_cg_cycle(CompactGmres g, const double* __restrict__ v0, const double* __restrict__ z0,
                           const double* __restrict__ part, int npart, GmresDev* gd, cudaGraphConditionalHandle cycle,
                           double* __restrict__ out);

// Opts the transform kernels into the large dynamic shared memory carve-out; returns the
// dynamic bytes every one of them may use (the opt-in limit minus their static shared memory).
template <typename K>
static int allow_dynamic_smem(K kernel, int optin) {
  cudaFuncAttributes a;
  if (cudaFuncGetAttributes(&a, kernel) != cudaSuccess) return 0;
  int dyn = optin - (int)a.sharedSizeBytes;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess) return 0;
  return dyn;
}
int configure_kernels(int smem_optin) {
  int d = smem_optin;
  d = std::min(d, allow_dynamic_smem(k_xpass<double, double, double, false>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_xpass<double, double, double, true>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_xpass<float, double, float, false>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_xpass<float, float, float, false>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_xpass<float, float, double, false>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve<double, 2>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve<double, 4>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve<double, 8>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve<double, 16>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve<float, 2>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve<float, 4>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve<float, 8>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve<float, 16>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_xpass_multi<double, double, double>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_xpass_multi<float, double, float>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_xpass_multi<float, float, float>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_xpass_multi<float, float, double>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve_multi<double, 2>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve_multi<double, 4>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve_multi<double, 8>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve_multi<double, 16>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve_multi<float, 2>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve_multi<float, 4>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve_multi<float, 8>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_ysolve_multi<float, 16>, smem_optin));
  d = std::min(d, allow_dynamic_smem(k_cg_cycle, smem_optin));
  return d;
}

// ---------------------------------------------------------------------------
// boundary Schur correction: c = S^{-1} (C first), scattered into w2
// ---------------------------------------------------------------------------
static constexpr int SCHUR_ROWS = 4;
// c = M first[mcols] with M = S^{-1} C (rank x m, FP64), scattered to w2 at the boundary rows.
// Every block gathers the m points into shared memory (independent loads), then its warps
// take SCHUR_ROWS rows of the GEMV (lanes over the row, FP64 accumulation).
template <typename TF>
__global__ void k_schur(const TF* __restrict__ first, int rank, int m, const int64_t* __restrict__ mcols,
                        const double* __restrict__ M, const int64_t* __restrict__ rows, double* __restrict__ w2,
                        Gate gate) {
  if (!gate_open(gate)) return;
  extern __shared__ double gsh[];
  for (int q0 = threadIdx.x; q0 < m; q0 += 4 * blockDim.x) {
    int64_t ix[4];
    TF fv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q0 + u * (int)blockDim.x < m) ix[u] = mcols[q0 + u * blockDim.x];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q0 + u * (int)blockDim.x < m) fv[u] = first[ix[u]];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q0 + u * (int)blockDim.x < m) gsh[q0 + u * blockDim.x] = cvt_to<double>(fv[u]);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int r0 = blockIdx.x * SCHUR_ROWS;
  for (int r = r0 + warp; r < min(rank, r0 + SCHUR_ROWS); r += nw) {
    const double* mr = M + (int64_t)r * m;
    double acc = 0.0;
#pragma unroll 8
    for (int q = lane; q < m; q += 32) acc += mr[q] * gsh[q];
    acc = warp_sum(acc);
    if (lane == 0) w2[rows[r]] = acc;
  }
}

template <typename TF>
void launch_schur(const TF* first, int rank, int m, const int64_t* mcols, const double* M, const int64_t* rows,
                  double* w2, const Gate& gate, cudaStream_t st) {
  if (rank <= 0) return;
  const unsigned g = (unsigned)((rank + SCHUR_ROWS - 1) / SCHUR_ROWS);
  note_launch();
  kt_mark(5, st);
  k_schur<TF><<<g, 32 * SCHUR_ROWS, (size_t)m * sizeof(double), st>>>(first, rank, m, mcols, M, rows, w2, gate);
  kt_mark(5, st, (double)m * (sizeof(TF) + 8) + (double)rank * m * 8 + rank * 16.0);
}
template void launch_schur<double>(const double*, int, int, const int64_t*, const double*, const int64_t*, double*,
                                   const Gate&, cudaStream_t);
template void launch_schur<float>(const float*, int, int, const int64_t*, const double*, const int64_t*, double*,
                                  const Gate&, cudaStream_t);

// ---------------------------------------------------------------------------
// boundary term by direct sums
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T warp_sum_t(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

static constexpr int BAND_TPB = 128;   // threads per output of the direct sums
static constexpr int BAND_ITEMS = 16;  // loads in flight per thread (n <= BAND_TPB * BAND_ITEMS per pass)

// Canonical order of the direct sums (every kernel that forms them uses it, so the single-case,
// fused and case-indexed paths agree bitwise): BAND_TPB threads per output, thread t adds its
// products at t, t + BAND_TPB, ... in order, then the warp sums, then the BAND_TPB / 32 warp
// partials in warp order.
template <typename TA, typename TB, typename TS>
__device__ __forceinline__ TS band_partial(const TA* __restrict__ a, const TB* __restrict__ b, int n, int t) {
  TS acc = 0;
  for (int k0 = t; k0 < n; k0 += BAND_TPB * BAND_ITEMS) {
    TA av[BAND_ITEMS];
    TB bv[BAND_ITEMS];
#pragma unroll
    for (int u = 0; u < BAND_ITEMS; ++u) {
      const int k = k0 + u * BAND_TPB;
      av[u] = k < n ? a[k] : (TA)0;
      bv[u] = k < n ? b[k] : (TB)0;
    }
#pragma unroll
    for (int u = 0; u < BAND_ITEMS; ++u) acc += cvt_to<TS>(av[u]) * cvt_to<TS>(bv[u]);
  }
  return acc;
}
// sum of a BAND_TPB-thread group's partials (part: BAND_TPB / 32 shared slots of this group);
// every thread of the block must call it (it holds block barriers)
template <typename T>
__device__ __forceinline__ T band_group_sum(T v, T* part, int t) {
  v = warp_sum_t<T>(v);
  __syncthreads();
  if ((t & 31) == 0) part[t >> 5] = v;
  __syncthreads();
  T s = 0;
#pragma unroll
  for (int w = 0; w < BAND_TPB / 32; ++w) s += part[w];
  return s;
}

// One block per point: the inverse row transform of its spectrum row evaluated at its column
// (coefficients in binv), all of a thread's products loaded before they are summed.
template <typename T>
__device__ __forceinline__ void band_first_body(int n, const int32_t* __restrict__ mrow, const T* __restrict__ binv,
                                                const T* __restrict__ spec, T* __restrict__ firstm, int q) {
  __shared__ T part[BAND_TPB / 32];
  const T v = band_group_sum<T>(
      band_partial<T, T, T>(binv + (int64_t)q * n, spec + (int64_t)mrow[q] * n, n, threadIdx.x), part, threadIdx.x);
  if (threadIdx.x == 0) firstm[q] = v;
}
template <typename T>
__global__ void __launch_bounds__(BAND_TPB) k_band_first(int m, int n, const int32_t* __restrict__ mrow,
                                                         const T* __restrict__ binv, const T* __restrict__ spec,
                                                         T* __restrict__ firstm, Gate gate) {
  if (!gate_open(gate)) return;
  band_first_body<T>(n, mrow, binv, spec, firstm, blockIdx.x);
}

// One block per row of M: c[r] = M[r] . firstm (FP64 accumulation).
template <typename T>
__device__ __forceinline__ void band_gemv_body(int m, const double* __restrict__ M, const T* __restrict__ firstm,
                                               double* __restrict__ c, int r) {
  __shared__ double part[BAND_TPB / 32];
  const double v = band_group_sum<double>(band_partial<double, T, double>(M + (int64_t)r * m, firstm, m, threadIdx.x),
                                          part, threadIdx.x);
  if (threadIdx.x == 0) c[r] = v;
}
template <typename T>
__global__ void __launch_bounds__(BAND_TPB) k_band_gemv(int rank, int m, const double* __restrict__ M,
                                                        const T* __restrict__ firstm, double* __restrict__ c,
                                                        Gate gate) {
  if (!gate_open(gate)) return;
  band_gemv_body<T>(m, M, firstm, c, blockIdx.x);
}

// The boundary term's Schur values in one sum per value: c[r] = G[r] . S[cj0 .. cj1 rows], with
// G = M binv folded on the host (G[r][(j - cj0) n + k] = sum over the points q of spectrum row j
// of M[r][q] binv[q][k]), so that the point values "first" are never formed.  Block (r, s) sums
// slice s of BAND_SPLIT slices (per-thread partials in T, the block's sum in FP64) and writes
// part[r BAND_SPLIT + s]; the band solve adds the slices in a fixed order.
template <typename T>
__device__ __forceinline__ void band_direct_body(int L, const T* __restrict__ G, const T* __restrict__ S,
                                                 double* __restrict__ part, int r, int sl) {
  __shared__ double dpart[BAND_TPB / 32];
  const int len = (L + BAND_SPLIT - 1) / BAND_SPLIT;
  const int i0 = sl * len, i1 = min(L, i0 + len);
  const T v = i1 > i0 ? band_partial<T, T, T>(G + (int64_t)r * L + i0, S + i0, i1 - i0, threadIdx.x) : (T)0;
  const double tot = band_group_sum<double>(cvt_to<double>(v), dpart, threadIdx.x);
  if (threadIdx.x == 0) part[r * BAND_SPLIT + sl] = tot;
}
template <typename T>
__global__ void __launch_bounds__(BAND_TPB) k_band_direct(int L, const T* __restrict__ G, const T* __restrict__ S,
                                                          double* __restrict__ part, Gate gate) {
  if (!gate_open(gate)) return;
  band_direct_body<T>(L, G, S, part, blockIdx.x / BAND_SPLIT, blockIdx.x % BAND_SPLIT);
}

// Blocks of BAND_COLS columns x BAND_ROWT row threads.  Thread (kk, jt) forms the forward
// row transform of U c on band rows jt, jt + BAND_ROWT, ... of column k (a sum over that row's
// boundary values, c staged in shared memory), scaled; then one thread per column runs the band
// system (as k_yband) in shared memory, and all threads write the band back.
static constexpr int BAND_COLS = 16, BAND_ROWT = 16;
template <typename T>
__device__ __forceinline__ void band_fwd_solve_body(int nb, int n, int rank, const int32_t* __restrict__ bptr,
                                                    const double* __restrict__ c,
                                                    const T* __restrict__ bfwd, T gamma, T scale,
                                                    const T* __restrict__ bpiv, T* __restrict__ band, int bid,
                                                    int nsplit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* cs = reinterpret_cast<T*>(smem_raw);   // rank values c (band-row order, as the GEMV writes them)
  T* xb = cs + ((rank + 3) & ~3);           // nb x BAND_COLS
  T* pb = xb + (size_t)nb * BAND_COLS;      // nb x BAND_COLS
  int* ps = reinterpret_cast<int*>(pb + (size_t)nb * BAND_COLS);  // nb + 1 row pointers
  const int tid = threadIdx.x, kk = tid % BAND_COLS, jt = tid / BAND_COLS;
  // c[e], or the sum of its nsplit slices in slice order (k_band_direct)
  for (int e = tid; e < rank; e += blockDim.x) {
    double v = c[(int64_t)e * nsplit];
    for (int sl = 1; sl < nsplit; ++sl) v += c[(int64_t)e * nsplit + sl];
    cs[e] = cvt_to<T>(v);
  }
  for (int j = tid; j <= nb; j += blockDim.x) ps[j] = bptr[j];
  __syncthreads();
  const int k = bid * BAND_COLS + kk;
  if (k < n) {
    for (int j = jt; j < nb; j += BAND_ROWT) {
      const int e0 = ps[j], e1 = ps[j + 1];
      T z = 0;
      for (int e = e0; e < e1; e += 8) {
        T bv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) bv[u] = e + u < e1 ? bfwd[(int64_t)(e + u) * n + k] : (T)0;
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (e + u < e1) z += cs[e + u] * bv[u];
      }
      xb[j * BAND_COLS + kk] = z * scale;
      pb[j * BAND_COLS + kk] = bpiv[(int64_t)j * n + k];
    }
  }
  __syncthreads();
  if (jt == 0 && k < n) {
    T z = 0;
    for (int j = 0; j < nb; ++j) {
      z = (xb[j * BAND_COLS + kk] - gamma * z) * pb[j * BAND_COLS + kk];
      xb[j * BAND_COLS + kk] = z;
    }
    T y = z;
    for (int j = nb - 2; j >= 0; --j) {
      y = xb[j * BAND_COLS + kk] - (gamma * pb[j * BAND_COLS + kk]) * y;
      xb[j * BAND_COLS + kk] = y;
    }
  }
  __syncthreads();
  if (k < n)
    for (int j = jt; j < nb; j += BAND_ROWT) band[(int64_t)j * n + k] = xb[j * BAND_COLS + kk];
}
template <typename T>
__global__ void __launch_bounds__(BAND_COLS * BAND_ROWT) k_band_fwd_solve(
    int nb, int n, int rank, const int32_t* __restrict__ bptr,
    const double* __restrict__ c, const T* __restrict__ bfwd, T gamma, T scale, const T* __restrict__ bpiv,
    T* __restrict__ band, Gate gate, int nsplit) {
  if (!gate_open(gate)) return;
  band_fwd_solve_body<T>(nb, n, rank, bptr, c, bfwd, gamma, scale, bpiv, band, blockIdx.x, nsplit);
}

int band_fwd_blocks(int n) { return (n + BAND_COLS - 1) / BAND_COLS; }
size_t band_fwd_smem(int nb, int rank, bool fp32) {
  const size_t esz = fp32 ? 4 : 8;
  return (size_t)((rank + 3) & ~3) * esz + (size_t)2 * nb * BAND_COLS * esz + (size_t)(nb + 1) * sizeof(int);
}

template <typename T>
void launch_band_first(int m, int n, const int32_t* mrow, const T* binv, const T* spec, T* firstm, const Gate& gate,
                       cudaStream_t st) {
  if (m <= 0) return;
  note_launch();
  kt_mark(5, st);
  launch_pdl(k_band_first<T>, dim3((unsigned)m), dim3(BAND_TPB), 0, st, m, n, mrow, binv, spec, firstm, gate);
  kt_mark(5, st, (double)m * n * 2 * sizeof(T));
}
template <typename T>
void launch_band_gemv(int rank, int m, const double* M, const T* firstm, double* c, const Gate& gate,
                      cudaStream_t st) {
  if (rank <= 0) return;
  note_launch();
  kt_mark(5, st);
  launch_pdl(k_band_gemv<T>, dim3((unsigned)rank), dim3(BAND_TPB), 0, st, rank, m, M, firstm, c, gate);
  kt_mark(5, st, (double)rank * m * 8 + (double)m * sizeof(T) + rank * 8.0);
}
template <typename T>
void launch_band_direct(int rank, int L, const T* G, const T* S, double* part, const Gate& gate, cudaStream_t st) {
  if (rank <= 0) return;
  note_launch();
  kt_mark(5, st);
  launch_pdl(k_band_direct<T>, dim3((unsigned)(rank * BAND_SPLIT)), dim3(BAND_TPB), 0, st, L, G, S, part, gate);
  // G read once, the spectrum rows once per value (L2), the slices written
  kt_mark(5, st, (double)rank * L * sizeof(T) + (double)L * sizeof(T) + rank * BAND_SPLIT * 8.0);
}
template <typename T>
void launch_band_fwd_solve(const TransformTables& tt, int n, int rank, const int32_t* bptr, const double* c,
                           const T* bfwd, T* band, const Gate& gate, cudaStream_t st, int nsplit) {
  const int nb = tt.bj1 - tt.bj0 + 1;
  if (nb <= 0) return;
  note_launch();
  kt_mark(5, st);
  launch_pdl(k_band_fwd_solve<T>, dim3((unsigned)((n + BAND_COLS - 1) / BAND_COLS)), dim3(BAND_COLS * BAND_ROWT),
             band_fwd_smem(nb, rank, sizeof(T) == 4), st, nb, n, rank, bptr, c, bfwd, (T)tt.gamma,
             (T)tt.yscale, (const T*)tt.bpiv, band, gate, nsplit);
  // the forward coefficients, the values c, the pivots and the band written once
  kt_mark(5, st, (double)rank * n * sizeof(T) + rank * 8.0 + (double)nb * n * 2 * sizeof(T));
}
template void launch_band_first<double>(int, int, const int32_t*, const double*, const double*, double*, const Gate&,
                                        cudaStream_t);
template void launch_band_first<float>(int, int, const int32_t*, const float*, const float*, float*, const Gate&,
                                       cudaStream_t);
template void launch_band_gemv<double>(int, int, const double*, const double*, double*, const Gate&, cudaStream_t);
template void launch_band_gemv<float>(int, int, const double*, const float*, double*, const Gate&, cudaStream_t);
template void launch_band_fwd_solve<double>(const TransformTables&, int, int, const int32_t*, const double*,
                                            const double*, double*, const Gate&, cudaStream_t, int);
template void launch_band_fwd_solve<float>(const TransformTables&, int, int, const int32_t*, const double*,
                                           const float*, float*, const Gate&, cudaStream_t, int);
template void launch_band_direct<double>(int, int, const double*, const double*, double*, const Gate&, cudaStream_t);
template void launch_band_direct<float>(int, int, const float*, const float*, double*, const Gate&, cudaStream_t);

// ---------------------------------------------------------------------------
// sparse rows with their loads batched: the column indices and values of up to CSR_B entries
// are loaded together, then the x values they point at, then the products are summed in entry
// order (the same sum as the one-entry-at-a-time loop, without an L2 round trip per entry)
// ---------------------------------------------------------------------------
template <int CSR_B = 8, typename F>
__device__ __forceinline__ void csr_row(const int64_t* __restrict__ col, const double* __restrict__ val, int64_t e0,
                                        int64_t e1, const double* __restrict__ x, int64_t xoff, F&& f) {
  for (int64_t e = e0; e < e1; e += CSR_B) {
    int64_t ci[CSR_B];
    double v[CSR_B], xv[CSR_B];
#pragma unroll
    for (int u = 0; u < CSR_B; ++u)
      if (e + u < e1) {
        ci[u] = col[e + u];
        v[u] = val[e + u];
      }
#pragma unroll
    for (int u = 0; u < CSR_B; ++u)
      if (e + u < e1) xv[u] = x[xoff + ci[u]];
#pragma unroll
    for (int u = 0; u < CSR_B; ++u)
      if (e + u < e1) f(v[u], xv[u]);
  }
}

// ---- the gates of a step (each raises the sticky error word; none clears it) ----
// whether the solve's checks ended within the sweeps that were launched for it
__device__ __forceinline__ bool sweeps_done(StepCtl* ctl, int slot, int nchk, int sweeps) {
  if (sweeps >= nchk - 1 || last_check(&ctl->solve[slot], nchk) <= sweeps) return true;
  raise_gate(ctl, ERR_SWEEPS, slot);
  return false;
}
__device__ void check_momentum(StepCtl* ctl, int nchk, int sweeps_u, int sweeps_v) {
  if (!sweeps_done(ctl, S_HELM_U, nchk, sweeps_u) || !sweeps_done(ctl, S_HELM_V, nchk, sweeps_v)) return;
  double r = 0, bm = 0;
  bool bad = false;
  for (int s = 0; s < 2; ++s) {
    const SolveCtl* sc = &ctl->solve[s];
    double rr = bits2d(sc->rmax[last_check(sc, nchk)]);
    double bb = bits2d(sc->bmax);
    if (!(rr <= r)) r = rr;  // propagates NaN
    if (bb > bm) bm = bb;
    if (sc->xbad) bad = true;
  }
  double thr = 1e-10 * (bm > 1.0 ? bm : 1.0);
  if (bad || !(r <= thr)) raise_gate(ctl, 2, 2);
}
__device__ void check_pressure(StepCtl* ctl, int slot, int nchk, int sweeps) {
  if (!sweeps_done(ctl, slot, nchk, sweeps)) return;
  const SolveCtl* sc = &ctl->solve[slot];
  int k = last_check(sc, nchk);
  double linf = bits2d(sc->rmax[k]), bound = bits2d(sc->bound[k]), bm = bits2d(sc->bmax);
  if (!isfinite(bm)) { raise_gate(ctl, 1, 4); return; }  // solver/pressure_schur.py:33-34
  double t = 64 * EPS64 * (bm > 1.0 ? bm : 1.0);
  t = t > 1e-10 ? t : 1e-10;
  t = bound > t ? bound : t;
  if (sc->xbad || !(linf <= t)) raise_gate(ctl, 2, 3);
}
__device__ __forceinline__ bool projection_ok(const StepCtl* ctl, int k) { return bits2d(ctl->div_max[k]) <= 1e-10; }
__device__ void check_projection(StepCtl* ctl, int k) {
  if (!projection_ok(ctl, k)) raise_gate(ctl, 2, 1);
}
// CFL screen of solver/main.py:273-278 (screen != 0; < 0: every 100th step by the counter) and the
// finite-field check of solver/time_integration.py:15-17 on the velocity maxima of the current state
__device__ void check_cfl(StepCtl* ctl, const unsigned long long* umax, const unsigned long long* vmax, double dt,
                          double dx, double dy, int screen, const long long* counter) {
  if (screen < 0) screen = (*counter % 100) == 0;
  double rate = bits2d(*umax) / dx + bits2d(*vmax) / dy;
  if (screen && (!isfinite(rate) || dt * rate > 0.5)) raise_gate(ctl, 2, 7);
  else if (!isfinite(rate)) raise_gate(ctl, 1, 8);
}

// ---------------------------------------------------------------------------
// ghost extension rows
// ---------------------------------------------------------------------------
// Each ghost value is its row of interior values (the stencils read no ghost point).  A row's
// entries are spread over GHOST_LANES lanes, so its loads take one or two rounds instead of a
// serial chain through L2, and the lanes' partial sums are added in a fixed butterfly order.
constexpr int GHOST_LANES = 8;
// Row r by the eight lanes l = 0..7 (r < 0: no row, zero); every lane of the warp calls it.
__device__ __forceinline__ double ghost_row(const double* __restrict__ f, const int64_t* __restrict__ ptr,
                                            const int64_t* __restrict__ col, const double* __restrict__ val, int r, int l) {
  double acc = 0.0;
  if (r >= 0)
    for (int64_t e = ptr[r] + l, e1 = ptr[r + 1]; e < e1; e += GHOST_LANES) acc += val[e] * f[col[e]];
  for (int o = GHOST_LANES / 2; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}
__global__ void k_ghost(double* __restrict__ f, int n, const int64_t* __restrict__ rows, const int64_t* __restrict__ ptr,
                        const int64_t* __restrict__ col, const double* __restrict__ val, Gate gate) {
  if (!gate_open(gate)) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = t / GHOST_LANES, l = t % GHOST_LANES;
  const double acc = ghost_row(f, ptr, col, val, r < n ? r : -1, l);
  if (r < n && l == 0) f[rows[r]] = acc;
}

void launch_ghost(double* field, int n, const int64_t* rows, const int64_t* ptr, const int64_t* col,
                  const double* val, const Gate& gate, cudaStream_t st) {
  if (n <= 0) return;
  note_launch();
  kt_mark(8, st);
  launch_pdl(k_ghost, dim3(blocks_for((int64_t)n * GHOST_LANES, 128)), dim3(128), 0, st, field, n, rows, ptr, col, val, gate);
  kt_mark(8, st);
}

// ---------------------------------------------------------------------------
// stencils on the staggered grid
// ---------------------------------------------------------------------------
struct Grid {
  int nx, ny;
  int64_t usize;
  __device__ __forceinline__ int64_t u(int j, int i) const { return (int64_t)j * (nx + 1) + i; }
  __device__ __forceinline__ int64_t v(int j, int i) const { return usize + (int64_t)j * nx + i; }
  __device__ __forceinline__ int64_t p(int j, int i) const { return (int64_t)j * nx + i; }
};

// -N(u) at u face (j,i), i>=1, before /(dx dy) (solver/numba_kernels.py:17-74 with nu=0);
// arithmetic in T (double for the plain path, float in the FP32 mode)
template <typename T, typename S>
__device__ __forceinline__ T adv_u(const S* __restrict__ U, const Grid& g, int j, int i, T dx, T dy) {
  const int nx = g.nx, ny = g.ny;
  const T h = (T)0.5;
  auto fxy = [&](int jj, int ii) -> T {  // corner flux at (jj, ii), jj in [0, ny]
    if (jj == 0 || jj == ny) return (T)0;
    T vf;
    if (ii == 0) vf = (T)U[g.v(jj, 0)];
    else if (ii == nx) vf = (T)U[g.v(jj, nx - 1)];
    else vf = h * ((T)U[g.v(jj, ii - 1)] + (T)U[g.v(jj, ii)]);
    T ua = h * ((T)U[g.u(jj - 1, ii)] + (T)U[g.u(jj, ii)]);
    return -((vf * ua) * dx);
  };
  T uW = (T)U[g.u(j, i - 1)], uC = (T)U[g.u(j, i)];
  T fl = h * (uW + uC);
  T fxxW = -((fl * fl) * dy);
  if (i < nx) {
    T fr = h * (uC + (T)U[g.u(j, i + 1)]);
    T fxxE = -((fr * fr) * dy);
    return (fxxE - fxxW) + (fxy(j + 1, i) - fxy(j, i));
  }
  return (-uC * uC) * dy - fxxW + h * (fxy(j + 1, nx) - fxy(j, nx));
}

// -N(v) at v face (j,i), 1<=j<=ny-1 (solver/numba_kernels.py:77-142 with nu=0)
template <typename T, typename S>
__device__ __forceinline__ T adv_v(const S* __restrict__ U, const Grid& g, int j, int i, T dx, T dy) {
  const int nx = g.nx;
  const T h = (T)0.5;
  auto fyx = [&](int jj, int ii) -> T {  // corner flux at (jj, ii), ii in [0, nx]
    if (ii == 0) return (T)0;
    T uf = h * ((T)U[g.u(jj - 1, ii)] + (T)U[g.u(jj, ii)]);
    if (ii == nx) return (-uf * (T)U[g.v(jj, nx - 1)]) * dy;
    T va = h * ((T)U[g.v(jj, ii - 1)] + (T)U[g.v(jj, ii)]);
    return -((uf * va) * dy);
  };
  T vS = (T)U[g.v(j - 1, i)], vC = (T)U[g.v(j, i)], vN = (T)U[g.v(j + 1, i)];
  T fb = h * (vS + vC), ft = h * (vC + vN);
  T fyyS = -((fb * fb) * dx), fyyN = -((ft * ft) * dx);
  return (fyx(j, i + 1) - fyx(j, i)) + (fyyN - fyyS);
}

// raw_l (5-point with channel-wall, inlet and outlet rules) at a u face (solver/optimized_ghost_cell.py:116-120)
template <typename T, typename S, typename GR = Grid>
__device__ __forceinline__ T lap_u(const S* __restrict__ U, const GR& g, int j, int i, T idx2, T idy2,
                                   bool inlet) {
  const int nx = g.nx, ny = g.ny;
  T acc = 0;
  if (j > 0) acc += idy2 * (T)U[g.u(j - 1, i)];
  if (i > 1 || inlet) acc += (i == nx ? (T)2 * idx2 : idx2) * (T)U[g.u(j, i - 1)];
  acc += ((T)-2 * idx2 - ((j == 0 || j == ny - 1) ? (T)3 : (T)2) * idy2) * (T)U[g.u(j, i)];
  if (i < nx) acc += idx2 * (T)U[g.u(j, i + 1)];
  if (j < ny - 1) acc += idy2 * (T)U[g.u(j + 1, i)];
  return acc;
}
// at a v face (solver/optimized_ghost_cell.py:121-123); walls v=0 are stored as zeros
template <typename T, typename S, typename GR = Grid>
__device__ __forceinline__ T lap_v(const S* __restrict__ U, const GR& g, int j, int i, T idx2, T idy2) {
  const int nx = g.nx;
  T acc = idy2 * (T)U[g.v(j - 1, i)];
  if (i > 0) acc += idx2 * (T)U[g.v(j, i - 1)];
  acc += (-(i == 0 ? (T)3 : (i == nx - 1 ? (T)1 : (T)2)) * idx2 - (T)2 * idy2) * (T)U[g.v(j, i)];
  if (i < nx - 1) acc += idx2 * (T)U[g.v(j, i + 1)];
  acc += idy2 * (T)U[g.v(j + 1, i)];
  return acc;
}
// G p at faces from a pressure grid with ghost values (solver/optimized_ghost_cell.py:94-107)
template <typename T, typename S, typename GR = Grid>
__device__ __forceinline__ T grad_u(const S* __restrict__ P, const GR& g, int j, int i, T gx) {
  if (i < g.nx) return gx * (T)P[g.p(j, i)] - gx * (T)P[g.p(j, i - 1)];
  return ((T)-2 * gx) * (T)P[g.p(j, g.nx - 1)];
}
template <typename T, typename S, typename GR = Grid>
__device__ __forceinline__ T grad_v(const S* __restrict__ P, const GR& g, int j, int i, T gy) {
  return gy * (T)P[g.p(j, i)] - gy * (T)P[g.p(j - 1, i)];
}

// decode a face-grid thread index
// (face grids hold fewer than 2^31 points, checked at set-up: 32-bit division suffices)
__device__ __forceinline__ bool face_of(int64_t t, const Grid& g, int& comp, int& j, int& i) {
  if (t < g.usize) {
    const unsigned ut = (unsigned)t, w = (unsigned)(g.nx + 1);
    comp = 0; j = (int)(ut / w); i = (int)(ut - (unsigned)j * w);
    return true;
  }
  int64_t r = t - g.usize;
  if (r >= (int64_t)(g.ny + 1) * g.nx) return false;
  const unsigned ur = (unsigned)r;
  comp = 1; j = (int)(ur / (unsigned)g.nx); i = (int)(ur - (unsigned)j * g.nx);
  return true;
}

// T: stencil arithmetic; S: storage type the stencils read (double, or the FP32 copies)
template <typename T, typename S>
__global__ void k_momentum(CaseDev c, MomentumArgs a, const S* __restrict__ Us, const S* __restrict__ Ps, Gate gate) {
  if (!gate_open(gate)) return;
  if (a.state_max && blockIdx.x + threadIdx.x == 0)
    check_cfl(gate.ctl, a.state_max, a.state_max + 1, a.dt, c.dx, c.dy, a.screen, a.counter);
  const Grid g{c.nx, c.ny, c.usize};
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int comp, j, i;
  if (!face_of(t, g, comp, j, i)) return;
  const uint8_t cls = comp == 0 ? c.cls_u[t] : c.cls_v[t - c.usize];
  if (!(cls & CLS_ACTIVE)) {
    double z = (comp == 0 && i == 0) ? c.inlet[j] : 0.0;
    if (a.mode != 2 && a.now) a.now[t] = 0.0;
    a.out[t] = a.mode == 1 ? z : 0.0;
    return;
  }
  constexpr bool F32 = sizeof(T) == 4;
  const T dx = F32 ? (T)c.fdx : (T)c.dx, dy = F32 ? (T)c.fdy : (T)c.dy;
  const T idx2 = F32 ? (T)c.fidx2 : (T)c.idx2, idy2 = F32 ? (T)c.fidy2 : (T)c.idy2;
  const T iarea = F32 ? (T)c.fiarea : (T)c.iarea, nu = F32 ? (T)c.fnu : (T)c.nu;
  const T dt = F32 ? (T)a.dt32 : (T)a.dt;
  const double q = a.U[t];
  T lq, gp, now = 0, off = 0;
  if (comp == 0) {
    lq = nu * lap_u<T>(Us, g, j, i, idx2, idy2, true);
    gp = grad_u<T>(Ps, g, j, i, F32 ? (T)c.fgx : (T)c.gx);
    if (a.mode != 2) {
      now = adv_u<T>(Us, g, j, i, dx, dy) * iarea;
      if (i == c.nx) now *= (T)2;
    }
    if (i == 1) off = nu * (idx2 * (T)c.inlet[j]);
  } else {
    lq = nu * lap_v<T>(Us, g, j, i, idx2, idy2);
    gp = grad_v<T>(Ps, g, j, i, F32 ? (T)c.fgy : (T)c.gy);
    if (a.mode != 2) now = adv_v<T>(Us, g, j, i, dx, dy) * iarea;
  }
  if (a.mode == 1) {
    a.now[t] = cvt_to<double>(now);
    a.out[t] = q + cvt_to<double>(((T)0.5 * dt) * ((now + lq) - gp));
    return;
  }
  T expl;
  if (a.mode == 0) {
    const T alpha = F32 ? (T)a.alpha32 : (T)a.alpha;
    expl = ((T)1 + alpha) * now - alpha * cvt_to<T>(a.prev[t]);
    a.now[t] = cvt_to<double>(now);
  } else {
    if (comp == 0) {
      expl = adv_u<T>(a.Uhalf, g, j, i, dx, dy) * iarea;
      if (i == c.nx) expl *= (T)2;
    } else {
      expl = adv_v<T>(a.Uhalf, g, j, i, dx, dy) * iarea;
    }
  }
  // rhs = q + dt (explicit + L q / 2 - G p) + dt/2 offset (solver/numba_kernels.py:596-601)
  if constexpr (sizeof(T) == 8)
    a.out[t] = (q + (double)(dt * (expl + (T)0.5 * lq - gp))) + (double)(((T)0.5 * dt) * off);
  else  // one FP64 add per face (the conversion runs on the integer pipe)
    a.out[t] = q + cvt_to<double>(dt * (expl + (T)0.5 * lq - gp) + ((T)0.5 * dt) * off);
}

// ---------------------------------------------------------------------------
// The AB2 momentum right-hand side (mode 0 of k_momentum) from a shared-memory tile.
//
// A block owns a TJ x TI patch of "points" (j, i), j in [0, ny], i in [0, nx]: point (j, i) is
// the u face (j, i) when j < ny and the v face (j, i) when i < nx.  It loads the u, v and p
// values its faces read (one halo row / column) once, with coalesced row loads, and forms each
// shared flux once instead of once per face that uses it:
//   corner products C = ua vf at the cell corners (jj, ii), 1 <= jj <= ny-1, 1 <= ii <= nx, where
//     ua = (u(jj-1, ii) + u(jj, ii)) / 2 and vf = (v(jj, ii-1) + v(jj, ii)) / 2 (v(jj, nx-1) at the
//     outlet); the u faces use -(C dx) (their fxy corner flux), the v faces -(C dy) (fyx): four
//     faces share each corner;
//   centre fluxes Xu = -((u(j, ii-1) + u(j, ii))^2 / 4 dy) of the u cells and
//     Yv = -((v(jj-1, i) + v(jj, i))^2 / 4 dx) of the v cells, two faces each
// (solver/numba_kernels.py:17-142: the same flux formulas as adv_u / adv_v).  The diffusion and
// pressure-gradient stencils read the tile through the same lap / grad functions as k_momentum.
// ---------------------------------------------------------------------------
static constexpr int MTI = 32, MTJ = 8;  // points per tile: 32 along x (one warp), 8 rows
// offsets of global (j, i) in the shared tiles: u and v tiles of (MTJ+2) x (MTI+2) (rows j0-1 ..
// j0+MTJ, columns i0-1 .. i0+MTI), the u tile first; the p tile (MTJ+1) x (MTI+1)
struct TileGrid {
  int nx, ny, j0, i0;
  static constexpr int W = MTI + 2, H = MTJ + 2, WP = MTI + 1;
  __device__ __forceinline__ int u(int j, int i) const { return (j - j0 + 1) * W + (i - i0 + 1); }
  __device__ __forceinline__ int v(int j, int i) const { return H * W + (j - j0 + 1) * W + (i - i0 + 1); }
  __device__ __forceinline__ int p(int j, int i) const { return (j - j0 + 1) * WP + (i - i0 + 1); }
};

// The FP32 mode converts as it fills the tiles (integer pipe; the halo points twice): a kernel that
// wrote FP32 copies of the state first took 12 us of the 800x820 step, and its own launch.
__global__ void __launch_bounds__(MTI * MTJ) k_momentum_tiled(CaseDev c, MomentumArgs a, const double* __restrict__ Us,
                                                              const double* __restrict__ Ps, Gate gate) {
  using T = float;
  using S = float;
  constexpr int W = TileGrid::W, H = TileGrid::H, WP = TileGrid::WP;
  __shared__ S suv[2 * H * W];
  __shared__ S sp[(MTJ + 1) * WP];
  __shared__ T fx[(MTJ + 1) * (MTI + 1)];  // -(C dx) at corner (j0 + r, i0 + q)
  __shared__ T fy[(MTJ + 1) * (MTI + 1)];  // -(C dy)
  __shared__ T xu[MTJ * (MTI + 1)];        // Xu at (j0 + r, i0 + q)
  __shared__ T yv[(MTJ + 1) * MTI];        // Yv at (j0 + r, i0 + q)
  if (!gate_open(gate)) return;
  // a raised screen stops every kernel behind this one, whose outputs are scratch until the step ends
  if (a.state_max && blockIdx.x + blockIdx.y + threadIdx.x + threadIdx.y == 0)
    check_cfl(gate.ctl, a.state_max, a.state_max + 1, a.dt, c.dx, c.dy, a.screen, a.counter);
  const int nx = c.nx, ny = c.ny;
  const int j0 = blockIdx.y * MTJ, i0 = blockIdx.x * MTI;
  const int tid = threadIdx.y * MTI + threadIdx.x;
  const Grid g{nx, ny, c.usize};
  const TileGrid tg{nx, ny, j0, i0};
  // 1. the tiles (zero outside the grids; no stencil below reads those entries)
  for (int e = tid; e < H * W; e += MTI * MTJ) {
    const int r = e / W, q = e - r * W;
    const int j = j0 - 1 + r, i = i0 - 1 + q;
    suv[e] = (j >= 0 && j < ny && i >= 0 && i <= nx) ? cvt_to<S>(Us[g.u(j, i)]) : (S)0;
    suv[H * W + e] = (j >= 0 && j <= ny && i >= 0 && i < nx) ? cvt_to<S>(Us[g.v(j, i)]) : (S)0;
  }
  for (int e = tid; e < (MTJ + 1) * WP; e += MTI * MTJ) {
    const int r = e / WP, q = e - r * WP;
    const int j = j0 - 1 + r, i = i0 - 1 + q;
    sp[e] = (j >= 0 && j < ny && i >= 0 && i < nx) ? cvt_to<S>(Ps[g.p(j, i)]) : (S)0;
  }
  __syncthreads();
  const T dx = c.fdx, dy = c.fdy;
  const T hh = (T)0.5;
  auto U = [&](int j, int i) -> T { return (T)suv[tg.u(j, i)]; };
  auto V = [&](int j, int i) -> T { return (T)suv[tg.v(j, i)]; };
  // 2. the shared fluxes
  for (int e = tid; e < (MTJ + 1) * (MTI + 1); e += MTI * MTJ) {
    const int r = e / (MTI + 1), q = e - r * (MTI + 1);
    const int jj = j0 + r, ii = i0 + q;
    T cx = (T)0, cy = (T)0;
    if (jj >= 1 && jj <= ny - 1 && ii >= 1 && ii <= nx) {
      const T vf = ii == nx ? V(jj, nx - 1) : hh * (V(jj, ii - 1) + V(jj, ii));
      const T ua = hh * (U(jj - 1, ii) + U(jj, ii));
      const T cc = vf * ua;
      cx = -(cc * dx);
      cy = -(cc * dy);
    }
    fx[e] = cx;
    fy[e] = cy;
  }
  for (int e = tid; e < MTJ * (MTI + 1); e += MTI * MTJ) {
    const int r = e / (MTI + 1), q = e - r * (MTI + 1);
    const int j = j0 + r, ii = i0 + q;
    T x = (T)0;
    if (j < ny && ii >= 1 && ii <= nx) {
      const T fl = hh * (U(j, ii - 1) + U(j, ii));
      x = -((fl * fl) * dy);
    }
    xu[e] = x;
  }
  for (int e = tid; e < (MTJ + 1) * MTI; e += MTI * MTJ) {
    const int r = e / MTI, q = e - r * MTI;
    const int jj = j0 + r, i = i0 + q;
    T y = (T)0;
    if (jj >= 1 && jj <= ny && i < nx) {
      const T fb = hh * (V(jj - 1, i) + V(jj, i));
      y = -((fb * fb) * dx);
    }
    yv[e] = y;
  }
  __syncthreads();
  const int r = threadIdx.y, q = threadIdx.x;
  const int j = j0 + r, i = i0 + q;
  const T idx2 = c.fidx2, idy2 = c.fidy2;
  const T iarea = c.fiarea, nu = c.fnu;
  const T dt = a.dt32;
  const T alpha = a.alpha32;
  auto FX = [&](int jj, int ii) -> T { return fx[(jj - j0) * (MTI + 1) + (ii - i0)]; };
  auto FY = [&](int jj, int ii) -> T { return fy[(jj - j0) * (MTI + 1) + (ii - i0)]; };
  auto XU = [&](int jj, int ii) -> T { return xu[(jj - j0) * (MTI + 1) + (ii - i0)]; };
  auto YV = [&](int jj, int ii) -> T { return yv[(jj - j0) * MTI + (ii - i0)]; };
  // 3. the faces of this point
  for (int comp = 0; comp < 2; ++comp) {
    if (comp == 0 ? (j >= ny || i > nx) : (j > ny || i >= nx)) continue;
    const int64_t t = comp == 0 ? g.u(j, i) : g.v(j, i);
    const uint8_t cls = comp == 0 ? c.cls_u[t] : c.cls_v[t - c.usize];
    if (!(cls & CLS_ACTIVE)) {
      a.now[t] = 0.0;
      a.out[t] = 0.0;
      continue;
    }
    const double qv = a.U[t];
    T lq, gp, now, off = 0;
    if (comp == 0) {
      lq = nu * lap_u<T>(suv, tg, j, i, idx2, idy2, true);
      gp = grad_u<T>(sp, tg, j, i, c.fgx);
      T adv;
      if (i < nx) {
        adv = (XU(j, i + 1) - XU(j, i)) + (FX(j + 1, i) - FX(j, i));
      } else {
        const T uC = U(j, i);
        adv = (-uC * uC) * dy - XU(j, nx) + hh * (FX(j + 1, nx) - FX(j, nx));
      }
      now = adv * iarea;
      if (i == nx) now *= (T)2;
      if (i == 1) off = nu * (idx2 * (T)c.inlet[j]);
    } else {
      lq = nu * lap_v<T>(suv, tg, j, i, idx2, idy2);
      gp = grad_v<T>(sp, tg, j, i, c.fgy);
      now = ((FY(j, i + 1) - FY(j, i)) + (YV(j + 1, i) - YV(j, i))) * iarea;
    }
    const T expl = ((T)1 + alpha) * now - alpha * cvt_to<T>(a.prev[t]);
    a.now[t] = cvt_to<double>(now);
    a.out[t] = qv + cvt_to<double>(dt * (expl + (T)0.5 * lq - gp) + ((T)0.5 * dt) * off);
  }
}

// The FP64 form.  The FP64 pipe is the bound (1/64 of the FP32 rate), so every constant is formed on the host
// and multiplied last: the tiles hold the unscaled products 4 C, (u + u)^2 and (v + v)^2 (seven
// instructions a point), and a face away from the channel's edges takes fifteen.  At 800x820 94 us with the
// fluxes scaled where they are formed (about 86 instructions a point), 67 now; other faces go the long way
// through the same functions as k_momentum.
__global__ void __launch_bounds__(MTI * MTJ, 4) k_momentum_tiled64(CaseDev c, MomentumArgs a, MomentumC m, Gate gate) {
  constexpr int W = TileGrid::W, H = TileGrid::H, WP = TileGrid::WP, WC = MTI + 1;
  __shared__ double suv[2 * H * W];
  __shared__ double sp[(MTJ + 1) * WP];
  __shared__ double cc[(MTJ + 1) * WC];  // 4 C at corner (j0 + r, i0 + q), zero on the walls
  __shared__ double xu[MTJ * WC];        // (u(j, ii - 1) + u(j, ii))^2 at (j0 + r, i0 + q)
  __shared__ double yv[(MTJ + 1) * MTI]; // (v(jj - 1, i) + v(jj, i))^2 at (j0 + r, i0 + q)
  if (!gate_open(gate)) return;
  // a raised screen stops every kernel behind this one, whose outputs are scratch until the step ends
  if (a.state_max && blockIdx.x + blockIdx.y + threadIdx.x + threadIdx.y == 0)
    check_cfl(gate.ctl, a.state_max, a.state_max + 1, a.dt, c.dx, c.dy, a.screen, a.counter);
  const int nx = c.nx, ny = c.ny;
  const int j0 = blockIdx.y * MTJ, i0 = blockIdx.x * MTI;
  const int tid = threadIdx.y * MTI + threadIdx.x;
  const Grid g{nx, ny, c.usize};
  const TileGrid tg{nx, ny, j0, i0};
  for (int e = tid; e < H * W; e += MTI * MTJ) {
    const int r = e / W, q = e - r * W;
    const int j = j0 - 1 + r, i = i0 - 1 + q;
    suv[e] = (j >= 0 && j < ny && i >= 0 && i <= nx) ? a.U[g.u(j, i)] : 0.0;
    suv[H * W + e] = (j >= 0 && j <= ny && i >= 0 && i < nx) ? a.U[g.v(j, i)] : 0.0;
  }
  for (int e = tid; e < (MTJ + 1) * WP; e += MTI * MTJ) {
    const int r = e / WP, q = e - r * WP;
    const int j = j0 - 1 + r, i = i0 - 1 + q;
    sp[e] = (j >= 0 && j < ny && i >= 0 && i < nx) ? a.P[g.p(j, i)] : 0.0;
  }
  __syncthreads();
  auto U = [&](int j, int i) { return suv[tg.u(j, i)]; };
  auto V = [&](int j, int i) { return suv[tg.v(j, i)]; };
  for (int e = tid; e < (MTJ + 1) * WC; e += MTI * MTJ) {
    const int r = e / WC, q = e - r * WC, jj = j0 + r, ii = i0 + q;
    double x = 0.0;
    if (jj >= 1 && jj <= ny - 1 && ii >= 1 && ii <= nx)
      x = (V(jj, ii - 1) + V(jj, ii == nx ? nx - 1 : ii)) * (U(jj - 1, ii) + U(jj, ii));
    cc[e] = x;
  }
  for (int e = tid; e < MTJ * WC; e += MTI * MTJ) {
    const int r = e / WC, q = e - r * WC, j = j0 + r, ii = i0 + q;
    double x = 0.0;
    if (j < ny && ii >= 1 && ii <= nx) { x = U(j, ii - 1) + U(j, ii); x *= x; }
    xu[e] = x;
  }
  for (int e = tid; e < (MTJ + 1) * MTI; e += MTI * MTJ) {
    const int r = e / MTI, q = e - r * MTI, jj = j0 + r, i = i0 + q;
    double y = 0.0;
    if (jj >= 1 && jj <= ny && i < nx) { y = V(jj - 1, i) + V(jj, i); y *= y; }
    yv[e] = y;
  }
  __syncthreads();
  const int r = threadIdx.y, q = threadIdx.x;
  const int j = j0 + r, i = i0 + q;
  auto C = [&](int jj, int ii) { return cc[(jj - j0) * WC + (ii - i0)]; };
  auto XU = [&](int jj, int ii) { return xu[(jj - j0) * WC + (ii - i0)]; };
  auto YV = [&](int jj, int ii) { return yv[(jj - j0) * MTI + (ii - i0)]; };
  const bool inner = j >= 1 && j < ny - 1 && i >= 2 && i < nx - 1;
  for (int comp = 0; comp < 2; ++comp) {
    if (comp == 0 ? (j >= ny || i > nx) : (j > ny || i >= nx)) continue;
    const int64_t t = comp == 0 ? g.u(j, i) : g.v(j, i);
    const uint8_t cls = comp == 0 ? c.cls_u[t] : c.cls_v[t - c.usize];
    if (!(cls & CLS_ACTIVE)) {
      a.now[t] = 0.0;
      a.out[t] = 0.0;
      continue;
    }
    if (inner) {
      double now, ew, ns, x, dp;
      if (comp == 0) {
        now = fma(m.ax, XU(j, i + 1) - XU(j, i), m.ay * (C(j + 1, i) - C(j, i)));
        x = U(j, i);
        ew = U(j, i - 1) + U(j, i + 1);
        ns = U(j - 1, i) + U(j + 1, i);
        dp = (sp[tg.p(j, i)] - sp[tg.p(j, i - 1)]) * m.gx;
      } else {
        now = fma(m.ax, C(j, i + 1) - C(j, i), m.ay * (YV(j + 1, i) - YV(j, i)));
        x = V(j, i);
        ew = V(j, i - 1) + V(j, i + 1);
        ns = V(j - 1, i) + V(j + 1, i);
        dp = (sp[tg.p(j, i)] - sp[tg.p(j - 1, i)]) * m.gy;
      }
      a.now[t] = now;
      a.out[t] = momentum_rhs(m, x, ew, ns, now, a.prev[t], dp);
      continue;
    }
    const double qv = a.U[t];
    double lq, gp, now, off = 0.0;
    if (comp == 0) {
      lq = c.nu * lap_u<double>(suv, tg, j, i, c.idx2, c.idy2, true);
      gp = grad_u<double>(sp, tg, j, i, c.gx);
      if (i < nx) {
        now = m.ax * (XU(j, i + 1) - XU(j, i)) + m.ay * (C(j + 1, i) - C(j, i));
      } else {  // half a volume with the outlet's flux u^2
        const double uC = U(j, i);
        now = 2.0 * (m.ax * (4.0 * (uC * uC) - XU(j, nx)) + (0.5 * m.ay) * (C(j + 1, nx) - C(j, nx)));
      }
      if (i == 1) off = c.nu * (c.idx2 * c.inlet[j]);
    } else {
      lq = c.nu * lap_v<double>(suv, tg, j, i, c.idx2, c.idy2);
      gp = grad_v<double>(sp, tg, j, i, c.gy);
      // the corner at the outlet is 2 v (u + u): uf v whole there
      now = m.ax * (C(j, i + 1) - C(j, i)) + m.ay * (YV(j + 1, i) - YV(j, i));
    }
    const double expl = (1.0 + a.alpha) * now - a.alpha * a.prev[t];
    a.now[t] = now;
    a.out[t] = (qv + a.dt * (expl + 0.5 * lq - gp)) + (0.5 * a.dt) * off;
  }
}

static dim3 momentum_tiles(const CaseDev& c) {
  return dim3((unsigned)((c.nx + 1 + MTI - 1) / MTI), (unsigned)((c.ny + 1 + MTJ - 1) / MTJ));
}

// Whether the AB2 right-hand side runs from shared-memory tiles (GHOSTMAC_MOMENTUM_TILED=0: the
// one-thread-per-face kernel, 1: the tiles; read at every launch, which graph replays do not repeat).
// FP64 grids of fewer tiles than SMs go by face: two barriers and three passes over the tile cost more than
// the instructions they save where most SMs idle (forty steps at 96x48, 28 tiles: 7.65 ms with tiles, 7.53
// by face; twenty at 400x200, 338 tiles: 5.55 and 5.62).
static bool momentum_tiled(const CaseDev& c, bool f32) {
  const char* e = std::getenv("GHOSTMAC_MOMENTUM_TILED");
  if (e && e[0]) return e[0] != '0';
  const dim3 t = momentum_tiles(c);
  return f32 || t.x * t.y >= 152;
}

__global__ void k_shadow(const double* __restrict__ U, float* __restrict__ U32, int64_t nf,
                         const double* __restrict__ P, float* __restrict__ P32, int64_t np, Gate gate) {
  if (!gate_open(gate)) return;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nf + np; t += (int64_t)gridDim.x * blockDim.x) {
    if (t < nf) U32[t] = f64_to_f32i(U[t]);
    else P32[t - nf] = f64_to_f32i(P[t - nf]);
  }
}
void launch_shadow(const double* U, float* U32, int64_t n_f, const double* P, float* P32, int64_t n_p,
                   const Gate& gate, cudaStream_t st) {
  note_launch();
  kt_mark(3, st);
  launch_pdl(k_shadow, dim3(reduce_blocks(n_f + n_p)), dim3(TPB), 0, st, U, U32, n_f, P, P32, n_p, gate);
  kt_mark(3, st);
}

void launch_momentum(const CaseDev& c, const MomentumArgs& a, const Gate& gate, cudaStream_t st) {
  note_launch();
  kt_mark(3, st);
  if (a.mode == 0 && momentum_tiled(c, false))
    launch_pdl(k_momentum_tiled64, dim3(momentum_tiles(c)), dim3(dim3(MTI, MTJ)), 0, st, c, a,
               MomentumC{-0.25 * c.dy * c.iarea, -0.25 * c.dx * c.iarea, a.dt * (1 + a.alpha), a.dt * a.alpha,
                         0.5 * a.dt * c.nu * c.idx2, 0.5 * a.dt * c.nu * c.idy2, a.dt * c.gx, a.dt * c.gy}, gate);
  else
    launch_pdl(k_momentum<double, double>, dim3(blocks_for(c.usize + c.vsize)), dim3(TPB), 0, st, c, a, a.U, a.P, gate);
  // algorithmic bytes: U, prev, class map read; now, out written; P read
  kt_mark(3, st, (double)(c.usize + c.vsize) * (8 * 4 + 1) + (double)c.psize * 8);
}
void launch_momentum_f32(const CaseDev& c, const MomentumArgs& a_in, const Gate& gate, cudaStream_t st) {
  MomentumArgs a = a_in;
  a.dt32 = (float)a.dt;
  a.alpha32 = (float)a.alpha;
  const bool tiled = momentum_tiled(c, true), shadow = a.mode == 0 && !tiled;
  if (shadow) launch_shadow(a.U, a.U32, c.usize + c.vsize, a.P, a.P32, c.psize, gate, st);
  note_launch();
  kt_mark(3, st);
  if (a.mode == 0 && tiled)
    launch_pdl(k_momentum_tiled, dim3(momentum_tiles(c)), dim3(dim3(MTI, MTJ)), 0, st, c, a, a.U, a.P, gate);
  else if (shadow)
    launch_pdl(k_momentum<float, float>, dim3(blocks_for(c.usize + c.vsize)), dim3(TPB), 0, st, c, a, a.U32, a.P32, gate);
  else
    launch_pdl(k_momentum<float, double>, dim3(blocks_for(c.usize + c.vsize)), dim3(TPB), 0, st, c, a, a.U, a.P, gate);
  kt_mark(3, st, (double)(c.usize + c.vsize) * (8 * 4 + 1) + (double)c.psize * 8);
}

__global__ void k_advection(CaseDev c, const double* __restrict__ U, double* __restrict__ out, Gate gate) {
  if (!gate_open(gate)) return;
  const Grid g{c.nx, c.ny, c.usize};
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int comp, j, i;
  if (!face_of(t, g, comp, j, i)) return;
  const uint8_t cls = comp == 0 ? c.cls_u[t] : c.cls_v[t - c.usize];
  if (!(cls & CLS_ACTIVE)) { out[t] = 0.0; return; }
  double r;
  if (comp == 0) {
    r = adv_u<double>(U, g, j, i, c.dx, c.dy) * c.iarea;
    if (i == c.nx) r *= 2;
  } else {
    r = adv_v<double>(U, g, j, i, c.dx, c.dy) * c.iarea;
  }
  out[t] = r;
}
void launch_advection(const CaseDev& c, const double* U, double* out, const Gate& gate, cudaStream_t st) {
  note_launch();
  k_advection<<<blocks_for(c.usize + c.vsize), TPB, 0, st>>>(c, U, out, gate);
}

__global__ void k_diffusion(CaseDev c, const double* __restrict__ U, double* __restrict__ out, int with_inlet,
                            double hdt, Gate gate) {
  if (!gate_open(gate)) return;
  const Grid g{c.nx, c.ny, c.usize};
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int comp, j, i;
  if (!face_of(t, g, comp, j, i)) return;
  const uint8_t cls = comp == 0 ? c.cls_u[t] : c.cls_v[t - c.usize];
  if (!(cls & CLS_ACTIVE)) { out[t] = 0.0; return; }
  const double idx2 = c.idx2, idy2 = c.idy2;
  double l = comp == 0 ? c.nu * lap_u<double>(U, g, j, i, idx2, idy2, with_inlet != 0) : c.nu * lap_v<double>(U, g, j, i, idx2, idy2);
  out[t] = hdt == 0.0 ? l : U[t] - hdt * l;
}
void launch_diffusion(const CaseDev& c, const double* U, double* out, bool with_inlet, double hdt, const Gate& gate,
                      cudaStream_t st) {
  note_launch();
  k_diffusion<<<blocks_for(c.usize + c.vsize), TPB, 0, st>>>(c, U, out, with_inlet ? 1 : 0, hdt, gate);
}

__global__ void k_gradient(CaseDev c, const double* __restrict__ P, double* __restrict__ out, Gate gate) {
  if (!gate_open(gate)) return;
  const Grid g{c.nx, c.ny, c.usize};
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int comp, j, i;
  if (!face_of(t, g, comp, j, i)) return;
  const uint8_t cls = comp == 0 ? c.cls_u[t] : c.cls_v[t - c.usize];
  if (!(cls & CLS_ACTIVE)) { out[t] = 0.0; return; }
  out[t] = comp == 0 ? grad_u<double>(P, g, j, i, c.gx) : grad_v<double>(P, g, j, i, c.gy);
}
void launch_gradient(const CaseDev& c, const double* P, double* out, const Gate& gate, cudaStream_t st) {
  note_launch();
  k_gradient<<<blocks_for(c.usize + c.vsize), TPB, 0, st>>>(c, P, out, gate);
}

// ---------------------------------------------------------------------------
// residual of the pressure operator A or the Helmholtz operators
// ---------------------------------------------------------------------------

// Residual res = b - A x of the pressure operator A (KIND 0, p grid) or the Helmholtz
// operators I - c L (KIND 1 u faces, KIND 2 v faces), with max |res| and sum res^2 per check.
// GB300 issues FP64 at 1/64 of the FP32 rate, so the regular rows use coefficients formed on
// the host (ResidualCoef): one add and four multiply-adds per point.  RES_F32: the residual
// is stored in FP32 (the input of the FP32 inverse).  Its max norm, which drives the
// refinement, is still taken from the FP64 residual; the diagnostic sums of res^2 and b^2 are
// FP32, so the only FP64 work left is the stencil.  The pressure gate's roundoff bound is formed
// in FP32 beside it.
// coefficient selection by value (indexing the parameter struct would copy it to local memory)
__device__ __forceinline__ double coef_cc(const ResidualCoef& rc, int ic, int jc) {
  const double c0 = jc ? rc.cc[0][1] : rc.cc[0][0];
  const double c1 = jc ? rc.cc[1][1] : rc.cc[1][0];
  const double c2 = jc ? rc.cc[2][1] : rc.cc[2][0];
  return ic == 0 ? c0 : (ic == 1 ? c1 : c2);
}
__device__ __forceinline__ double coef_cw(const ResidualCoef& rc, int ic) {
  return ic == 0 ? rc.cw[0] : (ic == 1 ? rc.cw[1] : rc.cw[2]);
}

template <int KIND, bool RES_F32>
__device__ __forceinline__ void residual_body(const CaseDev& c, const ResidualCoef& rc, const double* __restrict__ b,
                                              const double* __restrict__ x, void* __restrict__ res_out, SolveCtl* sc,
                                              int check, int first, int bid, int nblk) {
  if (check < 0) check = *(volatile int*)&sc->k;
  const int nx = c.nx, ny = c.ny;
  const int w = KIND == 1 ? nx + 1 : nx;            // row width of the grid
  const int64_t npts = KIND == 0 ? c.psize : (KIND == 1 ? c.usize : c.vsize);
  const int64_t base = KIND == 2 ? c.usize : 0;     // face-grid offset of the v field
  const uint8_t* cls = KIND == 0 ? c.cls_p : (KIND == 1 ? c.cls_u : c.cls_v);
  double* res64 = reinterpret_cast<double*>(res_out);
  float* res32 = reinterpret_cast<float*>(res_out);
  unsigned long long rm = 0, bm = 0, bd = 0, xb = 0;
  unsigned long long full = 0;  // largest |A| |x| + |b| over rows with five entries: scaling by their (2 nnz + 2) eps is monotonic
  double rs = 0.0, bs = 0.0;
  float rs32 = 0.0f;  // RES_F32: sum of the stored FP32 residuals squared (diagnostics only)
  float bs32 = 0.0f;  // RES_F32: sum of the right-hand side squared in FP32 (diagnostics only)
  // RES_F32, pressure: the roundoff bound (2 nnz + 2) eps (|A| |x| + |b|) in FP32 and integer
  // arithmetic, beside the FP64 stencil (the FP64 pipe is this kernel's bound)
  constexpr bool BOUND32 = KIND == 0 && RES_F32;
  float bd32 = 0.0f;
  for (int64_t t = (int64_t)bid * blockDim.x + threadIdx.x; t < npts; t += (int64_t)nblk * blockDim.x) {
    const uint8_t k = cls[t];
    const int64_t f = base + t;
    if (!(k & CLS_ACTIVE)) {
      if (RES_F32) res32[f] = 0.0f; else res64[f] = 0.0;
      continue;
    }
    const double xv = x[f], bv = b[f];
    double r, aabs = 0.0;
    float aabs32 = 0.0f;
    int nnz = 0;
    const int row = (k & CLS_IRREG) ? c.irr_index[KIND][t] : -1;
    if (row >= 0) {
      const int64_t* cp = c.irr_ptr[KIND];
      double ax = 0.0;
      const int64_t e0 = cp[row], e1 = cp[row + 1];
      csr_row<4>(c.irr_col[KIND], c.irr_val[KIND], e0, e1, x, base, [&](double a, double xv2) {
        ax += a * xv2;
        if (KIND == 0 && !RES_F32) aabs += absd(a) * absd(xv2);
        if (BOUND32) aabs32 += fabsf(f64_to_f32i(a)) * fabsf(f64_to_f32i(xv2));
      });
      r = bv - ax;
      nnz = (int)(e1 - e0);
    } else {
      const int j = (int)((unsigned)t / (unsigned)w), i = (int)((unsigned)t - (unsigned)j * w);
      // neighbours outside the operator's stencil read as zero
      double xw = 0.0, xe = 0.0, xs = 0.0, xn = 0.0;
      int ic, jc;
      if (KIND == 0) {
        if (i > 0) xw = x[f - 1];
        if (i < nx - 1) xe = x[f + 1];
        if (j > 0) xs = x[f - w];
        if (j < ny - 1) xn = x[f + w];
        ic = i == 0 ? 0 : (i == nx - 1 ? 2 : 1);
        jc = (j == 0 || j == ny - 1) ? 0 : 1;
      } else if (KIND == 1) {
        if (i > 1) xw = x[f - 1];
        if (i < nx) xe = x[f + 1];
        if (j > 0) xs = x[f - w];
        if (j < ny - 1) xn = x[f + w];
        ic = i == nx ? 2 : 1;
        jc = (j == 0 || j == ny - 1) ? 0 : 1;
      } else {
        if (i > 0) xw = x[f - 1];
        if (i < nx - 1) xe = x[f + 1];
        if (j > 1) xs = x[f - w];
        if (j < ny - 1) xn = x[f + w];
        ic = i == 0 ? 0 : (i == nx - 1 ? 2 : 1);
        jc = 1;
      }
      // r = b - (cc x + cw xw + ce xe + cy (xs + xn)); Helmholtz rows carry the factors of
      // I - c L.  One add and four fused multiply-adds that subtract from b, written out so
      // that nothing else reaches the FP64 pipe; each rounding stays inside the
      // (2 nnz + 2) eps (|A| |x| + |b|) bound of the pressure gate.
      const double ccv = coef_cc(rc, ic, jc), cwv = coef_cw(rc, ic);
      r = fma(-rc.cy, xs + xn, fma(-rc.ce, xe, fma(-cwv, xw, fma(-ccv, xv, bv))));
      if (KIND == 0 && !RES_F32) {
        aabs = absd(ccv) * absd(xv) + rc.ce * (absd(xw) + absd(xe)) + rc.cy * (absd(xs) + absd(xn));
        nnz = c.a_nnz[t];
      }
      if (BOUND32) {
        const float c0 = jc ? rc.fcc[0][1] : rc.fcc[0][0], c1 = jc ? rc.fcc[1][1] : rc.fcc[1][0];
        const float c2 = jc ? rc.fcc[2][1] : rc.fcc[2][0];
        const float fcc = ic == 0 ? c0 : (ic == 1 ? c1 : c2);
        aabs32 = fabsf(fcc) * fabsf(f64_to_f32i(xv)) +
                 rc.fce * (fabsf(f64_to_f32i(xw)) + fabsf(f64_to_f32i(xe))) +
                 rc.fcy * (fabsf(f64_to_f32i(xs)) + fabsf(f64_to_f32i(xn)));
        nnz = c.a_nnz[t];
      }
    }
    rm = umax64(rm, absbits(r));
    if constexpr (RES_F32) {
      const float r32 = f64_to_f32i(r);
      res32[f] = r32;
      rs32 = fmaf(r32, r32, rs32);
    } else {
      res64[f] = r;
      rs += r * r;
    }
    if (KIND == 0 && !RES_F32) {
      const double ab = aabs + absd(bv);
      if (nnz == 5) full = umax64(full, dbits(ab));
      else bd = umax64(bd, dbits((2.0 * nnz + 2.0) * EPS64 * ab));
    }
    if (BOUND32)
      bd32 = fmaxf(bd32, (2.0f * (float)nnz + 2.0f) * 2.220446049250313e-16f * (aabs32 + fabsf(f64_to_f32i(bv))));
    if (first) {
      bm = umax64(bm, absbits(bv));
      if constexpr (RES_F32) {
        const float b32 = f64_to_f32i(bv);
        bs32 = fmaf(b32, b32, bs32);
      } else {
        bs += bv * bv;
      }
    }
    if (nonfinite_bits(xv)) xb = 1;
  }
  block_commit_max(rm, &sc->rmax[check]);
  if constexpr (RES_F32) block_commit_sum_f32(rs32, &sc->rsq[check]);
  else block_commit_sum(rs, &sc->rsq[check]);
  if (KIND == 0 && !RES_F32) block_commit_max(umax64(bd, dbits((2.0 * 5 + 2.0) * EPS64 * bits2d(full))), &sc->bound[check]);
  // the FP32 bound times 1 + 2^-20 (above its own rounding), as an FP64 value; non-negative
  // doubles order like their bits
  if (BOUND32) block_commit_max(dbits(f32_to_f64i(bd32 * 1.00000095367431640625f)), &sc->bound[check]);
  if (first) {
    block_commit_max(bm, &sc->bmax);
    if constexpr (RES_F32) block_commit_sum_f32(bs32, &sc->bsq);
    else block_commit_sum(bs, &sc->bsq);
  }
  block_commit_max(xb, &sc->xbad);
}
template <int KIND, bool RES_F32>
__global__ void k_residual(CaseDev c, ResidualCoef rc, const double* __restrict__ b, const double* __restrict__ x,
                           void* __restrict__ res_out, SolveCtl* sc, int check, int first, Gate gate) {
  if (!gate_open(gate)) return;
  residual_body<KIND, RES_F32>(c, rc, b, x, res_out, sc, check, first, blockIdx.x, gridDim.x);
}

void launch_residual(const CaseDev& c, const ResidualCoef& rc, int kind, const double* b, const double* x, void* res,
                     bool res_f32, SolveCtl* sc, int check, bool first_check, const Gate& gate, cudaStream_t st) {
  const int64_t n = kind == 0 ? c.psize : (kind == 1 ? c.usize : c.vsize);
  const unsigned g = residual_blocks(n, res_f32);
  const int fc = first_check ? 1 : 0;
  note_launch();
  kt_mark(4, st);
  if (res_f32) {
    if (kind == 0) launch_pdl(k_residual<0, true>, dim3(g), dim3(TPB), 0, st, c, rc, b, x, res, sc, check, fc, gate);
    else if (kind == 1) launch_pdl(k_residual<1, true>, dim3(g), dim3(TPB), 0, st, c, rc, b, x, res, sc, check, fc, gate);
    else launch_pdl(k_residual<2, true>, dim3(g), dim3(TPB), 0, st, c, rc, b, x, res, sc, check, fc, gate);
  } else {
    if (kind == 0) launch_pdl(k_residual<0, false>, dim3(g), dim3(TPB), 0, st, c, rc, b, x, res, sc, check, fc, gate);
    else if (kind == 1) launch_pdl(k_residual<1, false>, dim3(g), dim3(TPB), 0, st, c, rc, b, x, res, sc, check, fc, gate);
    else launch_pdl(k_residual<2, false>, dim3(g), dim3(TPB), 0, st, c, rc, b, x, res, sc, check, fc, gate);
  }
  kt_mark(4, st, (double)n * (8 + 8 + (res_f32 ? 4 : 8) + 1));  // x, b, res, class map
}

// ---------------------------------------------------------------------------
// FP32 Jacobi sweeps of the CN Helmholtz systems (FP32 mode)
// ---------------------------------------------------------------------------
// The CN systems H = I - c L (c = dt nu / 2) are strongly diagonally dominant: the Jacobi
// iteration matrix has row-sum norm rho = max_i sum_{j != i} |H_ij| / |H_ii|, about 4 c / h^2
// (0.016 on the 800x820 Re 100 case), which the host computes from every row at set-up.  In
// the FP32 mode one application of the approximate inverse is then `iters` Jacobi
// iterations d <- D^{-1} (r - (H - D) d) from d = 0, in FP32, with the same regular-row
// coefficients and irregular rows as the residual kernel; x = [x +] d closes the last one.
// The FP64 residual and the refinement loop around it are those of the FFT inverse, so the
// answer meets the same residual targets; only the number of sweeps may differ.
static constexpr int JPT = 4;  // consecutive points per thread in the Jacobi iterations
template <int KIND, typename TR>
__global__ void __launch_bounds__(TPB) k_helm_jacobi(CaseDev c, ResidualCoef rc, HelmJacobi hj,
                                                    const TR* __restrict__ r, const float* __restrict__ din,
                                                    float* __restrict__ dout, double* __restrict__ x, int accumulate,
                                                    Gate gate) {
  if (!gate_open(gate)) return;
  const int nx = c.nx, ny = c.ny;
  const int w = KIND == 1 ? nx + 1 : nx;
  const int64_t npts = KIND == 1 ? c.usize : c.vsize;
  const int64_t base = KIND == 2 ? c.usize : 0;
  const uint8_t* cls = KIND == 1 ? c.cls_u : c.cls_v;
  const int64_t t0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * JPT;
  if (t0 >= npts) return;
  // every load of the thread's JPT points first (one round trip), then the arithmetic
  uint8_t k[JPT];
  float rv[JPT], dw[JPT], de[JPT], ds[JPT], dn[JPT];
#pragma unroll
  for (int u = 0; u < JPT; ++u) {
    const int64_t t = t0 + u;
    k[u] = 0;
    rv[u] = dw[u] = de[u] = ds[u] = dn[u] = 0.0f;
    if (t >= npts) continue;
    const int64_t f = base + t;
    k[u] = cls[t];
    if constexpr (sizeof(TR) == 8) rv[u] = f64_to_f32i(r[f]);
    else rv[u] = r[f];
    if (din) {
      const int j = (int)((unsigned)t / (unsigned)w), i = (int)((unsigned)t - (unsigned)j * w);
      if (KIND == 1) {
        if (i > 1) dw[u] = din[f - 1];
        if (i < nx) de[u] = din[f + 1];
        if (j > 0) ds[u] = din[f - w];
        if (j < ny - 1) dn[u] = din[f + w];
      } else {
        if (i > 0) dw[u] = din[f - 1];
        if (i < nx - 1) de[u] = din[f + 1];
        if (j > 1) ds[u] = din[f - w];
        if (j < ny - 1) dn[u] = din[f + w];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < JPT; ++u) {
    const int64_t t = t0 + u;
    if (t >= npts) continue;
    const int64_t f = base + t;
    float d = 0.0f;
    if (k[u] & CLS_ACTIVE) {
      const int row = (k[u] & CLS_IRREG) ? c.irr_index[KIND][t] : -1;
      if (row >= 0) {
        float sum = 0.0f;
        if (din) {
          const int64_t* cp = c.irr_ptr[KIND];
          const int64_t* col = c.irr_col[KIND];
          const float* val = hj.val[KIND - 1];
          for (int64_t e = cp[row]; e < cp[row + 1]; ++e) sum = fmaf(val[e], din[base + col[e]], sum);
        }
        d = (rv[u] - sum) * hj.idiag[KIND - 1][row];
      } else {
        const int j = (int)((unsigned)t / (unsigned)w), i = (int)((unsigned)t - (unsigned)j * w);
        int ic, jc;
        if (KIND == 1) {
          ic = i == nx ? 2 : 1;
          jc = (j == 0 || j == ny - 1) ? 0 : 1;
        } else {
          ic = i == 0 ? 0 : (i == nx - 1 ? 2 : 1);
          jc = 1;
        }
        const float cwv = ic == 0 ? rc.fcw[0] : (ic == 1 ? rc.fcw[1] : rc.fcw[2]);
        const float i0 = jc ? hj.icc[KIND - 1][0][1] : hj.icc[KIND - 1][0][0];
        const float i1 = jc ? hj.icc[KIND - 1][1][1] : hj.icc[KIND - 1][1][0];
        const float i2 = jc ? hj.icc[KIND - 1][2][1] : hj.icc[KIND - 1][2][0];
        const float icc = ic == 0 ? i0 : (ic == 1 ? i1 : i2);
        const float off = fmaf(rc.fcy, ds[u] + dn[u], fmaf(rc.fce, de[u], cwv * dw[u]));
        d = (rv[u] - off) * icc;
      }
    }
    if (x) {
      // inactive points of the solution are zero
      x[f] = !(k[u] & CLS_ACTIVE) ? 0.0 : (accumulate ? x[f] + f32_to_f64i(d) : f32_to_f64i(d));
    } else {
      dout[f] = d;
    }
  }
}

template <typename TR>
void launch_helm_jacobi(const CaseDev& c, const ResidualCoef& rc, const HelmJacobi& hj, int kind, const TR* r,
                        const float* din, float* dout, double* x, bool accumulate, const Gate& gate, cudaStream_t st) {
  const int64_t n = kind == 1 ? c.usize : c.vsize;
  note_launch();
  kt_mark(11, st);
  const unsigned g = blocks_for((n + JPT - 1) / JPT);
  if (kind == 1)
    launch_pdl(k_helm_jacobi<1, TR>, dim3(g), dim3(TPB), 0, st, c, rc, hj, r, din, dout, x, accumulate ? 1 : 0, gate);
  else
    launch_pdl(k_helm_jacobi<2, TR>, dim3(g), dim3(TPB), 0, st, c, rc, hj, r, din, dout, x, accumulate ? 1 : 0, gate);
  // algorithmic bytes: r, the class map, the five-point iterate (read once per point) and the
  // new iterate (or x read and written by the last iteration)
  kt_mark(11, st, (double)n * (sizeof(TR) + 1 + (din ? 4 : 0) + (x ? (accumulate ? 16 : 8) : 4)));
}
template void launch_helm_jacobi<double>(const CaseDev&, const ResidualCoef&, const HelmJacobi&, int, const double*,
                                         const float*, float*, double*, bool, const Gate&, cudaStream_t);
template void launch_helm_jacobi<float>(const CaseDev&, const ResidualCoef&, const HelmJacobi&, int, const float*,
                                        const float*, float*, double*, bool, const Gate&, cudaStream_t);

// Temporally blocked Jacobi application: every block loads the class map and the right-hand
// side of its region once, runs the iterations in shared memory and writes its output box.
// A point's value after `iters` iterations depends only on points that iters - 1 stencil
// applications reach from it, so a tile with a halo of iters - 1 five-point steps reproduces
// the global iteration exactly outside the body box (whose margin keeps every irregular row
// iters - 1 points away), and the body block's region holds everything its box reaches.
// Points of a regular tile's halo may be irregular rows updated with the five-point formula:
// their values never reach the tile's outputs.
// Shared memory of a region of rh x rw points, stored with a border of one zero point on each
// side (every neighbour read is then in bounds and a missing neighbour reads zero): four float
// arrays (two iterates, the right-hand side and each point's multiplier: 1 / diagonal, or 0 on
// an inactive point) and the west coefficient of each column.
__host__ __device__ inline size_t jacobi_region_bytes(int rh, int rw) {
  const size_t n = (size_t)(rh + 2) * (rw + 2);
  return (n * 4 + (size_t)(rw + 2) + 3) / 4 * 4 * sizeof(float);
}
size_t helm_jacobi_tiled_smem(const JacobiTiles& t, int iters) {
  const int h = iters - 1;
  const size_t reg = jacobi_region_bytes(t.th + 2 * h, t.tw + 2 * h);
  size_t body = 0;
  if (t.bj1 > t.bj0)
    body = jacobi_region_bytes(t.rj1 - t.rj0, t.ri1 - t.ri0) + (size_t)t.nnz * 8 + (size_t)t.nrow * 12 + 4;
  return (std::max(reg, body) + 15) / 16 * 16;
}

// Block 0 is the body block (it starts first); the others are the regular tiles.  Threads walk
// the region in rows of 32 points per warp, so no per-point index division is needed.  The
// operator's excluded neighbours (the u inlet column, the v wall rows) are inactive points whose
// iterate is zero, and points outside the grid are the zero border, so the five-point update
// needs no neighbour tests.
// threads of a tile block: every tile's work is latency bound (few warps per SM at this grid
// size), so a tile takes more warps than the other kernels' blocks
constexpr int JTPB = 512;
template <int KIND, typename TR>
__global__ void __launch_bounds__(JTPB) k_helm_jacobi_tiled(CaseDev c, ResidualCoef rc, HelmJacobi hj,
                                                          const TR* __restrict__ r, double* __restrict__ x,
                                                          int accumulate, Gate gate) {
  extern __shared__ __align__(16) float jsm[];
  if (!gate_open(gate)) return;
  const JacobiTiles& T = hj.jt[KIND - 1];
  const int nx = c.nx, ny = c.ny;
  const int W = KIND == 1 ? nx + 1 : nx;
  const int R = KIND == 1 ? ny : ny + 1;
  const int64_t base = KIND == 2 ? c.usize : 0;
  const uint8_t* cls = KIND == 1 ? c.cls_u : c.cls_v;
  const int h = hj.iters - 1;
  const bool has_body = T.bj1 > T.bj0;
  const bool body = has_body && blockIdx.x == 0;
  int j0, j1, i0, i1, oj0, oj1, oi0, oi1;
  if (body) {
    j0 = T.rj0; j1 = T.rj1; i0 = T.ri0; i1 = T.ri1;
    oj0 = T.bj0; oj1 = T.bj1; oi0 = T.bi0; oi1 = T.bi1;
  } else {
    const int b = (int)blockIdx.x - (has_body ? 1 : 0);
    const int ty = b / T.ntx, tx = b - ty * T.ntx;
    oj0 = ty * T.th; oj1 = min(oj0 + T.th, R);
    oi0 = tx * T.tw; oi1 = min(oi0 + T.tw, W);
    j0 = max(oj0 - h, 0); j1 = min(oj1 + h, R);
    i0 = max(oi0 - h, 0); i1 = min(oi1 + h, W);
  }
  const int rw = i1 - i0, rh = j1 - j0, pw = rw + 2, np = pw * (rh + 2);
  float* cur = jsm;
  float* nxt = jsm + np;
  float* rr = jsm + 2 * np;
  float* mm = jsm + 3 * np;   // 1 / diagonal of the point's regular row, 0 on inactive points
  float* colw = jsm + 4 * np; // west coefficient of each region column
  unsigned char* stage = reinterpret_cast<unsigned char*>(jsm) + jacobi_region_bytes(rh, rw);
  float* sval = reinterpret_cast<float*>(stage);
  int32_t* ssidx = reinterpret_cast<int32_t*>(sval + (body ? T.nnz : 0));
  int32_t* sptr = ssidx + (body ? T.nnz : 0);
  int32_t* spos = sptr + (body ? T.nrow + 1 : 0);
  float* sidg = reinterpret_cast<float*>(spos + (body ? T.nrow : 0));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  // zero borders of both iterates; the right-hand side and the multiplier of every point, and
  // the west coefficient of every column, formed once for all the iterations
  for (int q = threadIdx.x; q < np; q += blockDim.x) { cur[q] = 0.0f; nxt[q] = 0.0f; }
  for (int pi = threadIdx.x; pi < rw; pi += blockDim.x) {
    const int ii = i0 + pi;
    const int icl = KIND == 1 ? (ii == nx ? 2 : 1) : (ii == 0 ? 0 : (ii == nx - 1 ? 2 : 1));
    colw[pi] = icl == 0 ? rc.fcw[0] : (icl == 1 ? rc.fcw[1] : rc.fcw[2]);
  }
  for (int pj = warp; pj < rh; pj += nwarp) {
    const int jj = j0 + pj;
    const int jc = KIND == 1 ? ((jj == 0 || jj == ny - 1) ? 0 : 1) : 1;
    const float ia = hj.icc[KIND - 1][0][jc], ib = hj.icc[KIND - 1][1][jc], ic2 = hj.icc[KIND - 1][2][jc];
    const int64_t row = (int64_t)jj * W + i0;
    for (int pi = lane; pi < rw; pi += 32) {
      const int q = (pj + 1) * pw + pi + 1;
      const int ii = i0 + pi;
      const int icl = KIND == 1 ? (ii == nx ? 2 : 1) : (ii == 0 ? 0 : (ii == nx - 1 ? 2 : 1));
      const bool act = (cls[row + pi] & CLS_ACTIVE) != 0;
      mm[q] = act ? (icl == 0 ? ia : (icl == 1 ? ib : ic2)) : 0.0f;
      float rv;
      if constexpr (sizeof(TR) == 8) rv = f64_to_f32i(r[base + row + pi]);
      else rv = r[base + row + pi];
      rr[q] = act ? rv : 0.0f;
    }
  }
  if (body) {
    const int64_t* cp = c.irr_ptr[KIND];
    for (int e = threadIdx.x; e < T.nnz; e += blockDim.x) {
      sval[e] = hj.val[KIND - 1][e];
      const int sx = T.sidx[e];  // place in the unpadded region
      ssidx[e] = sx < 0 ? -1 : (sx / rw + 1) * pw + (sx - (sx / rw) * rw) + 1;
    }
    for (int q = threadIdx.x; q <= T.nrow; q += blockDim.x) {
      sptr[q] = (int32_t)cp[q];
      if (q < T.nrow) {
        const int sx = T.rpos[q];
        spos[q] = (sx / rw + 1) * pw + (sx - (sx / rw) * rw) + 1;
        sidg[q] = hj.idiag[KIND - 1][q];
      }
    }
  }
  __syncthreads();
  // the regular rows: d = (r - (cw d_w + ce d_e + cy (d_s + d_n))) / diagonal, zero on inactive
  // points (the arithmetic of the untiled kernel, in the same order)
  const float fce = rc.fce, fcy = rc.fcy;
  for (int it = 0; it < hj.iters; ++it) {
    for (int pj = warp; pj < rh; pj += nwarp) {
      const int q0 = (pj + 1) * pw + 1;
      for (int pi = lane; pi < rw; pi += 32) {
        const int q = q0 + pi;
        const float m = mm[q];
        const float off = it > 0 ? fmaf(fcy, cur[q - pw] + cur[q + pw], fmaf(fce, cur[q + 1], colw[pi] * cur[q - 1]))
                                 : 0.0f;
        nxt[q] = m != 0.0f ? (rr[q] - off) * m : 0.0f;
      }
    }
    if (body) {
      // the irregular rows overwrite their places with the rows' own entries
      __syncthreads();
      for (int q = threadIdx.x; q < T.nrow; q += blockDim.x) {
        const int p = spos[q];
        float sum = 0.0f;
        if (it > 0)
          for (int e = sptr[q]; e < sptr[q + 1]; ++e) {
            const int sx = ssidx[e];
            if (sx >= 0) sum = fmaf(sval[e], cur[sx], sum);
          }
        nxt[p] = (rr[p] - sum) * sidg[q];
      }
    }
    __syncthreads();
    float* tmp = cur;
    cur = nxt;
    nxt = tmp;
  }
  const int bj0 = T.bj0, bj1 = T.bj1, bi0 = T.bi0, bi1 = T.bi1;
  for (int pj = warp; pj < rh; pj += nwarp) {
    const int jj = j0 + pj;
    if (jj < oj0 || jj >= oj1) continue;
    const bool in_box_rows = has_body && jj >= bj0 && jj < bj1;
    const int64_t row = base + (int64_t)jj * W;
    for (int pi = lane; pi < rw; pi += 32) {
      const int ii = i0 + pi;
      if (ii < oi0 || ii >= oi1) continue;
      if (!body && in_box_rows && ii >= bi0 && ii < bi1) continue;
      const int q = (pj + 1) * pw + pi + 1;
      const int64_t f = row + ii;
      const float d = cur[q];
      x[f] = mm[q] == 0.0f ? 0.0 : (accumulate ? x[f] + f32_to_f64i(d) : f32_to_f64i(d));
    }
  }
}

// The kernels' dynamic shared-memory limit is a per-function, process-wide attribute shared by
// every case: it is raised to the device's opt-in maximum (never set to one case's size, which
// would make the launches of a larger case in the same process fail).
int helm_jacobi_tiled_optin(size_t smem) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  if (smem > (size_t)optin) return 1;
  const void* ks[4] = {(const void*)k_helm_jacobi_tiled<1, double>, (const void*)k_helm_jacobi_tiled<2, double>,
                       (const void*)k_helm_jacobi_tiled<1, float>, (const void*)k_helm_jacobi_tiled<2, float>};
  int e = 0;
  for (const void* k : ks) {
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, k) != cudaSuccess) { e = 1; continue; }
    const int dyn = optin - (int)a.sharedSizeBytes;
    if (smem > (size_t)dyn || cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess)
      e = 1;
  }
  if (e) cudaGetLastError();
  return e;
}

template <typename TR>
void launch_helm_jacobi_tiled(const CaseDev& c, const ResidualCoef& rc, const HelmJacobi& hj, int kind, const TR* r,
                              double* x, bool accumulate, size_t smem, const Gate& gate, cudaStream_t st) {
  const JacobiTiles& T = hj.jt[kind - 1];
  const unsigned g = (unsigned)(T.ntx * T.nty + (T.bj1 > T.bj0 ? 1 : 0));
  const int64_t n = kind == 1 ? c.usize : c.vsize;
  note_launch();
  kt_mark(11, st);
  if (kind == 1)
    launch_pdl(k_helm_jacobi_tiled<1, TR>, dim3(g), dim3(JTPB), smem, st, c, rc, hj, r, x, accumulate ? 1 : 0, gate);
  else
    launch_pdl(k_helm_jacobi_tiled<2, TR>, dim3(g), dim3(JTPB), smem, st, c, rc, hj, r, x, accumulate ? 1 : 0, gate);
  // algorithmic bytes: r and the class map read, x written (read too when accumulating)
  kt_mark(11, st, (double)n * (sizeof(TR) + 1 + (accumulate ? 16 : 8)));
}
template void launch_helm_jacobi_tiled<double>(const CaseDev&, const ResidualCoef&, const HelmJacobi&, int,
                                               const double*, double*, bool, size_t, const Gate&, cudaStream_t);
template void launch_helm_jacobi_tiled<float>(const CaseDev&, const ResidualCoef&, const HelmJacobi&, int,
                                              const float*, double*, bool, size_t, const Gate&, cudaStream_t);


// ---------------------------------------------------------------------------
// flexible GMRES on the pressure grid (solver/pressure_schur.py:20-57, iterative branch):
// operator apply, block-deterministic multi-dot products and multi-axpy updates
// ---------------------------------------------------------------------------
// w = A z on the pressure grid (zero at inactive cells)
__global__ void k_apply_pressure(CaseDev c, ResidualCoef rc, const double* __restrict__ z, double* __restrict__ w,
                                 Gate gate) {
  if (!gate_open(gate)) return;
  const int nx = c.nx, ny = c.ny;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < c.psize; t += (int64_t)gridDim.x * blockDim.x) {
    const uint8_t k = c.cls_p[t];
    if (!(k & CLS_ACTIVE)) {
      w[t] = 0.0;
      continue;
    }
    double ax;
    const int row = (k & CLS_IRREG) ? c.irr_index[0][t] : -1;
    if (row >= 0) {
      const int64_t* cp = c.irr_ptr[0];
      ax = 0.0;
      csr_row<4>(c.irr_col[0], c.irr_val[0], cp[row], cp[row + 1], z, 0, [&](double a, double zv) { ax += a * zv; });
    } else {
      const int j = (int)((unsigned)t / (unsigned)nx), i = (int)((unsigned)t - (unsigned)j * nx);
      const double xw = i > 0 ? z[t - 1] : 0.0, xe = i < nx - 1 ? z[t + 1] : 0.0;
      const double xs = j > 0 ? z[t - nx] : 0.0, xn = j < ny - 1 ? z[t + nx] : 0.0;
      const int ic = i == 0 ? 0 : (i == nx - 1 ? 2 : 1), jc = (j == 0 || j == ny - 1) ? 0 : 1;
      ax = coef_cc(rc, ic, jc) * z[t] + coef_cw(rc, ic) * xw + rc.ce * xe + rc.cy * (xs + xn);
    }
    w[t] = ax;
  }
}
void launch_apply_pressure(const CaseDev& c, const ResidualCoef& rc, const double* z, double* w, const Gate& gate,
                           cudaStream_t st) {
  note_launch();
  kt_mark(4, st);
  k_apply_pressure<<<reduce_blocks(c.psize), TPB, 0, st>>>(c, rc, z, w, gate);
  kt_mark(4, st, (double)c.psize * 17);
}

// Partial sums part[b * nv + i] = sum over block b's points of V_i[t] * w[t], i < nv (V_i at
// V + i * ld); the final pass sums the blocks in a fixed order (run-to-run identical).
static constexpr int GM_DOT_MAX = 64;
__global__ void k_multidot_part(const double* __restrict__ V, int64_t ld, int nv, const double* __restrict__ w,
                                int64_t n, double* __restrict__ part) {
  __shared__ double red[GM_DOT_MAX][TPB / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i0 = 0; i0 < nv; i0 += 8) {
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
      const double wt = w[t];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i0 + u < nv) acc[u] += V[(int64_t)(i0 + u) * ld + t] * wt;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const double sum = warp_sum(acc[u]);
      if (lane == 0 && i0 + u < nv) red[i0 + u][warp] = sum;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    double sum = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) sum += red[i][q];
    part[(int64_t)blockIdx.x * nv + i] = sum;
  }
}
__global__ void k_multidot_final(const double* __restrict__ part, int nblocks, int nv, double* __restrict__ out) {
  const int i = blockIdx.x;
  double acc = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += 32) acc += part[(int64_t)b * nv + i];
  acc = warp_sum(acc);
  if (threadIdx.x == 0) out[i] = acc;
}
void launch_multidot(const double* V, int64_t ld, int nv, const double* w, int64_t n, double* part, double* out,
                     cudaStream_t st) {
  const unsigned nb = reduce_blocks(n);
  note_launch();
  kt_mark(6, st);
  k_multidot_part<<<nb, TPB, 0, st>>>(V, ld, nv, w, n, part);
  kt_mark(6, st, (double)n * 8 * (nv + 1));
  note_launch();
  k_multidot_final<<<nv, 32, 0, st>>>(part, (int)nb, nv, out);
}
unsigned multidot_blocks(int64_t n) { return reduce_blocks(n); }

// y[t] = alpha * y[t] + sign * sum_i coef[i] V_i[t]   (coef on the device)
__global__ void k_multiaxpy(const double* __restrict__ V, int64_t ld, int nv, const double* __restrict__ coef,
                            double sign, double alpha, double* __restrict__ y, int64_t n) {
  __shared__ double cf[GM_DOT_MAX + 1];
  for (int i = threadIdx.x; i < nv; i += blockDim.x) cf[i] = coef[i];
  __syncthreads();
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int i = 0; i < nv; ++i) acc += cf[i] * V[(int64_t)i * ld + t];
    y[t] = alpha * y[t] + sign * acc;
  }
}
void launch_multiaxpy(const double* V, int64_t ld, int nv, const double* coef, double sign, double alpha, double* y,
                      int64_t n, cudaStream_t st) {
  note_launch();
  kt_mark(6, st);
  k_multiaxpy<<<reduce_blocks(n), TPB, 0, st>>>(V, ld, nv, coef, sign, alpha, y, n);
  kt_mark(6, st, (double)n * 8 * (nv + 2));
}

// Learned preconditioner input / output on the pressure grid: x = [v / s, mask] (float32,
// 2 planes), s = max |v| over the active cells (computed by the first kernel into *s_bits);
// z += s y on the active cells.
__global__ void k_learned_max(CaseDev c, const double* __restrict__ v, unsigned long long* s_bits) {
  unsigned long long m = 0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < c.psize; t += (int64_t)gridDim.x * blockDim.x)
    if (c.cls_p[t] & CLS_ACTIVE) m = umax64(m, absbits(v[t]));
  block_commit_max(m, s_bits);
}
__global__ void k_learned_in(CaseDev c, const double* __restrict__ v, const unsigned long long* __restrict__ s_bits,
                             float* __restrict__ x) {
  const double s = bits2d(*s_bits);
  const double inv = s > 0 ? 1.0 / s : 0.0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < c.psize; t += (int64_t)gridDim.x * blockDim.x) {
    const bool act = c.cls_p[t] & CLS_ACTIVE;
    x[t] = act ? (float)(v[t] * inv) : 0.f;
    x[c.psize + t] = act ? 1.f : 0.f;
  }
}
__global__ void k_learned_out(CaseDev c, const float* __restrict__ y, const unsigned long long* __restrict__ s_bits,
                              double* __restrict__ z) {
  const double s = bits2d(*s_bits);
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < c.psize; t += (int64_t)gridDim.x * blockDim.x)
    if (c.cls_p[t] & CLS_ACTIVE) z[t] += s * (double)y[t];
}
void launch_learned_prep(const CaseDev& c, const double* v, float* x, unsigned long long* s_bits, cudaStream_t st) {
  note_launch();
  k_learned_max<<<reduce_blocks(c.psize), TPB, 0, st>>>(c, v, s_bits);
  note_launch();
  k_learned_in<<<reduce_blocks(c.psize), TPB, 0, st>>>(c, v, s_bits, x);
}
void launch_learned_apply(const CaseDev& c, const float* y, const unsigned long long* s_bits, double* z,
                          cudaStream_t st) {
  note_launch();
  k_learned_out<<<reduce_blocks(c.psize), TPB, 0, st>>>(c, y, s_bits, z);
}

// ---------------------------------------------------------------------------
// projection pieces
// ---------------------------------------------------------------------------
// D U at the active cells (the operator; the projection's kernels are below)
__global__ void k_divergence(CaseDev c, const double* __restrict__ U, double* __restrict__ out) {
  const Grid g{c.nx, c.ny, c.usize};
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < c.psize; t += (int64_t)gridDim.x * blockDim.x) {
    if (c.cls_p[t] & CLS_ACTIVE) {
      int j = (int)((unsigned)t / (unsigned)c.nx), i = (int)((unsigned)t - (unsigned)j * c.nx);
      const double du = U[g.u(j, i + 1)] - U[g.u(j, i)], dv = U[g.v(j + 1, i)] - U[g.v(j, i)];
      out[t] = du * c.idx + dv * c.idy;
    } else {
      out[t] = 0.0;
    }
  }
}
void launch_divergence(const CaseDev& c, const double* U, double* out, cudaStream_t st) {
  note_launch();
  kt_mark(6, st);
  k_divergence<<<reduce_blocks(c.psize), TPB, 0, st>>>(c, U, out);
  kt_mark(6, st);
}

// ---- the projection ------------------------------------------------------------------------
// Each kernel is small (at 800x820 the grid passes take 8-13 us, at 96x48 about 4), so what a
// projection costs beside its solve is mostly the number of dependent kernels.  The ghost values
// therefore need none: the few points that read one (CLS_NEAR; about 400 at 800x820) go to the
// first blocks, eight lanes a ghost row in the order of k_ghost, and the gates sit in the first block
// of the kernel behind them.  A projection was nine kernels around its solve, now three;
// with the momentum kernel taking the CFL screen and the step's end one kernel of five, the step went from
// 259 to 220 us at 96x48, 347 to 309 at 400x200, 924 to 850 (FP64) and 584 to 531 (FP32) at 800x820.

// differences of the near cell's face values, on lane 0 of the warp (all lanes call)
__device__ __forceinline__ void near_diff(const CaseDev& c, const double* __restrict__ U, const NearCell& nc, double& du,
                                          double& dv) {
  const int lane = threadIdx.x & 31, l = lane % GHOST_LANES;
  const int32_t code = nc.code[lane / GHOST_LANES];
  double v = ghost_row(U, c.gf_ptr, c.gf_col, c.gf_val, code, l);
  if (code < 0 && l == 0) {
    const int f = ~code;
    v = (f < c.usize && f % (c.nx + 1) == 0) ? c.inlet[f / (c.nx + 1)] : U[f];
  }
  const double e = __shfl_sync(0xffffffffu, v, 0), w = __shfl_sync(0xffffffffu, v, GHOST_LANES);
  const double n = __shfl_sync(0xffffffffu, v, 2 * GHOST_LANES), s = __shfl_sync(0xffffffffu, v, 3 * GHOST_LANES);
  du = e - w;
  dv = n - s;
}
static inline int near_cell_blocks(const CaseDev& c) { return (c.n_near_c + TPB / 32 - 1) / (TPB / 32); }
static inline int ghost_blocks(int n) { return (int)blocks_for((int64_t)n * GHOST_LANES); }

__global__ void k_proj_rhs(CaseDev c, const double* __restrict__ U, double* __restrict__ out, double sx, double sy,
                           int chk, int nchk, int sweeps_u, int sweeps_v, int nbn, Gate gate) {
  if (!gate_open(gate)) return;
  if (chk && blockIdx.x + threadIdx.x == 0) {
    if (chk == PCHK_MOMENTUM) check_momentum(gate.ctl, nchk, sweeps_u, sweeps_v);
    else check_projection(gate.ctl, 1);
  }
  const Grid g{c.nx, c.ny, c.usize};
  bool bad = false;
  if ((int)blockIdx.x < nbn) {
    const int w = (blockIdx.x * TPB + threadIdx.x) >> 5;
    if (w >= c.n_near_c) return;
    double du, dv;
    near_diff(c, U, c.near_c[w], du, dv);
    if ((threadIdx.x & 31) == 0) {
      const double o = du * sx + dv * sy;
      out[c.near_c[w].cell] = o;
      bad = nonfinite_bits(o);
    }
  } else {
    for (int64_t t = (int64_t)(blockIdx.x - nbn) * TPB + threadIdx.x; t < c.psize; t += (int64_t)(gridDim.x - nbn) * TPB) {
      const uint8_t k = c.cls_p[t];
      if (k & CLS_NEAR) continue;
      double o = 0.0;
      if (k & CLS_ACTIVE) {
        const int j = (int)((unsigned)t / (unsigned)c.nx), i = (int)((unsigned)t - (unsigned)j * c.nx);
        const double uw = i > 0 ? U[g.u(j, i)] : c.inlet[j];
        const double du = U[g.u(j, i + 1)] - uw, dv = U[g.v(j + 1, i)] - U[g.v(j, i)];
        o = du * sx + dv * sy;
        bad = bad || nonfinite_bits(o);
      }
      out[t] = o;
    }
  }
  if (bad && gate.ctl) {
    // the gate in front comes first, whichever thread gets here first
    if (chk == PCHK_MOMENTUM) check_momentum(gate.ctl, nchk, sweeps_u, sweeps_v);
    else if (chk == PCHK_PROJECTION) check_projection(gate.ctl, 1);
    raise_gate(gate.ctl, 1, 4);
  }
}
void launch_proj_rhs(const CaseDev& c, const double* U, double* out, double dt, ProjCheck chk, int nchk, int sweeps_u,
                     int sweeps_v, const Gate& gate, cudaStream_t st) {
  const int nbn = near_cell_blocks(c);
  const double s = 1.0 / dt;
  note_launch();
  kt_mark(6, st);
  const dim3 grid((unsigned)nbn + reduce_blocks(c.psize));
  const int check = gate.ctl ? (int)chk : 0;
  if (chk == PCHK_MOMENTUM) k_proj_rhs<<<grid, TPB, 0, st>>>(c, U, out, c.idx * s, c.idy * s, check, nchk, sweeps_u,
                                                           sweeps_v, nbn, gate);
  else launch_pdl(k_proj_rhs, grid, dim3(TPB), 0, st, c, U, out, c.idx * s, c.idy * s, check, nchk, sweeps_u, sweeps_v, nbn, gate);
  kt_mark(6, st);
}

// out = q - dt G phi at the active faces, with dgx = dt gx and dgy = dt gy formed on the host:
// two fused multiply-adds per face (G phi is gx (phi_e - phi_w), at the outlet -2 gx phi_w).
// Blocks: nbf of near faces (16 lanes a face), nbg that fill phi's ghost values, then the grid.
__global__ void k_proj_update(CaseDev c, const double* __restrict__ q, double* phi, double dgx, double dgy,
                              double* __restrict__ out, int slot, int nchk, int sweeps, int nbf, int nbg, Gate gate) {
  if (!gate_open(gate)) return;
  if (gate.ctl && blockIdx.x + threadIdx.x == 0) check_pressure(gate.ctl, slot, nchk, sweeps);
  const Grid g{c.nx, c.ny, c.usize};
  const int b = blockIdx.x;
  if (b < nbf) {
    const int lane = threadIdx.x & 31, w = ((b * TPB + threadIdx.x) >> 5) * 2 + (lane >> 4);
    const bool in = w < c.n_near_f;
    NearFace nf{0, {NEAR_OUTLET, NEAR_OUTLET}};
    if (in) nf = c.near_f[w];
    const int l = lane % GHOST_LANES;
    const int32_t code = nf.code[(lane >> 3) & 1];
    double v = ghost_row(phi, c.gp_ptr, c.gp_col, c.gp_val, code, l);
    if (code < 0 && code != NEAR_OUTLET && l == 0) v = phi[~code];
    const double hi = __shfl_down_sync(0xffffffffu, v, GHOST_LANES);
    if (in && (lane & 15) == 0) {
      const int t = nf.face;
      if (t >= c.usize) out[t] = fma(dgy, v, fma(-dgy, hi, q[t]));
      else if (nf.code[1] != NEAR_OUTLET) out[t] = fma(dgx, v, fma(-dgx, hi, q[t]));
      else out[t] = fma(2.0 * dgx, v, q[t]);
    }
    return;
  }
  if (b < nbf + nbg) {
    const int t = (b - nbf) * TPB + threadIdx.x, r = t / GHOST_LANES, l = t % GHOST_LANES;
    const double v = ghost_row(phi, c.gp_ptr, c.gp_col, c.gp_val, r < c.n_ghost_p ? r : -1, l);
    if (r < c.n_ghost_p && l == 0) phi[c.gp_rows[r]] = v;
    return;
  }
  const int64_t t = (int64_t)(b - nbf - nbg) * TPB + threadIdx.x;
  int comp, j, i;
  if (!face_of(t, g, comp, j, i)) return;
  const uint8_t cls = comp == 0 ? c.cls_u[t] : c.cls_v[t - c.usize];
  if (cls & CLS_NEAR) return;
  if (!(cls & CLS_ACTIVE)) {
    out[t] = (comp == 0 && i == 0) ? c.inlet[j] : 0.0;
    return;
  }
  if (comp == 1) out[t] = fma(dgy, phi[g.p(j - 1, i)], fma(-dgy, phi[g.p(j, i)], q[t]));
  else if (i < c.nx) out[t] = fma(dgx, phi[g.p(j, i - 1)], fma(-dgx, phi[g.p(j, i)], q[t]));
  else out[t] = fma(2.0 * dgx, phi[g.p(j, c.nx - 1)], q[t]);
}
void launch_proj_update(const CaseDev& c, const double* q, double* phi, double dt, double* out, int slot, int nchk,
                        int sweeps, bool pdl, const Gate& gate, cudaStream_t st) {
  const int nbf = (c.n_near_f + TPB / 16 - 1) / (TPB / 16), nbg = ghost_blocks(c.n_ghost_p);
  const dim3 grid((unsigned)(nbf + nbg) + blocks_for(c.usize + c.vsize));
  const double dgx = dt * c.gx, dgy = dt * c.gy;
  note_launch();
  kt_mark(6, st);
  if (pdl) launch_pdl(k_proj_update, grid, dim3(TPB), 0, st, c, q, phi, dgx, dgy, out, slot, nchk, sweeps, nbf, nbg, gate);
  else k_proj_update<<<grid, TPB, 0, st>>>(c, q, phi, dgx, dgy, out, slot, nchk, sweeps, nbf, nbg, gate);
  kt_mark(6, st);
}

// H r at an active u (KIND 1) or v (KIND 2) face t (index within its face grid) for the
// Helmholtz operator H = I - c L of the CN solves: the same rows as residual_body's, i.e. the
// host-formed coefficients on regular rows (one add, one multiply, three fused multiply-adds)
// and the folded sparse rows next to the body.
template <int KIND>
__device__ __forceinline__ double helm_action(const CaseDev& c, const ResidualCoef& rc, const double* __restrict__ x,
                                              int64_t t, uint8_t k) {
  const int nx = c.nx, ny = c.ny;
  const int w = KIND == 1 ? nx + 1 : nx;
  const int64_t base = KIND == 2 ? c.usize : 0;
  const int64_t f = base + t;
  const int row = (k & CLS_IRREG) ? c.irr_index[KIND][t] : -1;
  if (row >= 0) {
    const int64_t* cp = c.irr_ptr[KIND];
    double ax = 0.0;
    csr_row<4>(c.irr_col[KIND], c.irr_val[KIND], cp[row], cp[row + 1], x, base,
               [&](double a, double xv2) { ax += a * xv2; });
    return ax;
  }
  const int j = (int)((unsigned)t / (unsigned)w), i = (int)((unsigned)t - (unsigned)j * w);
  double xw = 0.0, xe = 0.0, xs = 0.0, xn = 0.0;
  int ic, jc;
  if (KIND == 1) {
    if (i > 1) xw = x[f - 1];
    if (i < nx) xe = x[f + 1];
    if (j > 0) xs = x[f - w];
    if (j < ny - 1) xn = x[f + w];
    ic = i == nx ? 2 : 1;
    jc = (j == 0 || j == ny - 1) ? 0 : 1;
  } else {
    if (i > 0) xw = x[f - 1];
    if (i < nx - 1) xe = x[f + 1];
    if (j > 1) xs = x[f - w];
    if (j < ny - 1) xn = x[f + w];
    ic = i == 0 ? 0 : (i == nx - 1 ? 2 : 1);
    jc = 1;
  }
  const double ccv = coef_cc(rc, ic, jc), cwv = coef_cw(rc, ic);
  return fma(rc.cy, xs + xn, fma(rc.ce, xe, fma(cwv, xw, ccv * x[f])));
}

// Block-wide maxima of N words (block_commit_max for several, two barriers in all).
template <int N>
__device__ void block_commit_maxes(unsigned long long (&v)[N], unsigned long long* const (&dst)[N]) {
  __shared__ unsigned long long sm[N][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < N; ++q) {
    v[q] = warp_max_u64(v[q]);
    if (lane == 0) sm[q][wid] = v[q];
  }
  __syncthreads();
  if (wid < N) {
    unsigned long long x = 0;
    unsigned long long* d = nullptr;
#pragma unroll
    for (int q = 0; q < N; ++q)
      if (wid == q) {
        x = lane < (int)(blockDim.x >> 5) ? sm[q][lane] : 0ull;
        d = dst[q];
      }
    x = warp_max_u64(x);
    if (lane == 0 && x && d) atomicMax(d, x);
  }
}

// What follows a projection (TailArgs), one pass over the grids.  Blocks: nbn of near cells, nbg that
// fill U's ghost values (no other block reads them here: the defect's rows hold active faces only),
// then the grid.
//   DEFECT    the defect correction of the CN velocity (solver/time_integration.py): action = H U and
//             proj = U + (rhs - H U) at the active faces; inlet values and zeros elsewhere
//   PRESSURE  half = p + inc, pout = half + factor inc, max |action - rhs + dt G inc|, and the maxima of
//             the new velocity over the whole grids
template <int KIND>
__global__ void k_proj_tail(CaseDev c, ResidualCoef rcu, ResidualCoef rcv, TailArgs a, int nbn, int nbg, Gate gate) {
  if (!gate_open(gate)) return;
  const Grid g{c.nx, c.ny, c.usize};
  const int b = blockIdx.x;
  double* U = a.U;
  if (b < nbn) {
    const int w = (b * TPB + threadIdx.x) >> 5;
    if (w >= c.n_near_c) return;
    double du, dv;
    near_diff(c, U, c.near_c[w], du, dv);
    if ((threadIdx.x & 31) == 0) {
      const unsigned long long d = absbits(du * c.idx + dv * c.idy);
      if (d) atomicMax(a.divmax, d);
    }
    return;
  }
  if (b < nbn + nbg) {
    const int t = (b - nbn) * TPB + threadIdx.x, r = t / GHOST_LANES, l = t % GHOST_LANES;
    const double v = ghost_row(U, c.gf_ptr, c.gf_col, c.gf_val, r < c.n_ghost_f ? r : -1, l);
    if (r < c.n_ghost_f && l == 0) U[c.gf_rows[r]] = v;
    return;
  }
  const int64_t nf = c.usize + c.vsize, n = KIND == TAIL_PLAIN ? c.psize : nf + c.psize;
  unsigned long long dm = 0, cm = 0, um = 0, vm = 0;
  for (int64_t t = (int64_t)(b - nbn - nbg) * TPB + threadIdx.x; t < n; t += (int64_t)(gridDim.x - nbn - nbg) * TPB) {
    if (KIND == TAIL_PLAIN || t >= nf) {
      const int64_t k = KIND == TAIL_PLAIN ? t : t - nf;
      const uint8_t cls = c.cls_p[k];
      if (!(cls & CLS_ACTIVE)) {
        if (KIND == TAIL_PRESSURE) a.half[k] = a.pout[k] = 0.0;
        continue;
      }
      if (!(cls & CLS_NEAR)) {
        const int j = (int)((unsigned)k / (unsigned)c.nx), i = (int)((unsigned)k - (unsigned)j * c.nx);
        const double du = U[g.u(j, i + 1)] - U[g.u(j, i)], dv = U[g.v(j + 1, i)] - U[g.v(j, i)];
        dm = umax64(dm, absbits(du * c.idx + dv * c.idy));
      }
      if (KIND == TAIL_PRESSURE) {
        const double h = a.p[k] + a.inc[k];
        a.half[k] = h;
        a.pout[k] = h + a.factor * a.inc[k];
      }
    } else {
      int comp, j, i;
      face_of(t, g, comp, j, i);
      const uint8_t cls = comp == 0 ? c.cls_u[t] : c.cls_v[t - c.usize];
      if (KIND == TAIL_DEFECT) {
        if (!(cls & CLS_ACTIVE)) {
          a.action[t] = 0.0;
          a.proj[t] = (comp == 0 && i == 0) ? c.inlet[j] : 0.0;
          continue;
        }
        const double hr = comp == 0 ? helm_action<1>(c, rcu, U, t, cls) : helm_action<2>(c, rcv, U, t - c.usize, cls);
        a.action[t] = hr;
        a.proj[t] = U[t] + (a.rhs[t] - hr);
      } else {
        const unsigned long long x = absbits(a.unew[t]);
        if (comp == 0) um = umax64(um, x);
        else vm = umax64(vm, x);
        if (!(cls & CLS_ACTIVE)) continue;
        // action - rhs + dt G inc, with dgx = dt gx and dgy = dt gy formed on the host
        const double a0 = a.action[t] - a.rhs[t];
        double r;
        if (comp == 1) r = fma(-a.dgy, a.inc[g.p(j - 1, i)], fma(a.dgy, a.inc[g.p(j, i)], a0));
        else if (i < c.nx) r = fma(-a.dgx, a.inc[g.p(j, i - 1)], fma(a.dgx, a.inc[g.p(j, i)], a0));
        else r = fma(-2.0 * a.dgx, a.inc[g.p(j, c.nx - 1)], a0);
        cm = umax64(cm, absbits(r));
      }
    }
  }
  if (KIND == TAIL_PRESSURE) {
    unsigned long long v[4] = {dm, cm, um, vm};
    unsigned long long* const d[4] = {a.divmax, a.coupled, a.umax, a.umax + 1};
    block_commit_maxes<4>(v, d);
  } else {
    block_commit_max(dm, a.divmax);
  }
}
void launch_proj_tail(const CaseDev& c, const ResidualCoef& rcu, const ResidualCoef& rcv, ProjTail kind, const TailArgs& a,
                      const Gate& gate, cudaStream_t st) {
  const int nbn = near_cell_blocks(c), nbg = kind == TAIL_PRESSURE ? 0 : ghost_blocks(c.n_ghost_f);
  const int64_t n = kind == TAIL_PLAIN ? c.psize : c.usize + c.vsize + c.psize;
  // eight blocks an SM (a full one of threads): the passes wait on L2, the reductions are a block's end
  const dim3 grid((unsigned)(nbn + nbg) + std::min(blocks_for(n), 1216u));
  note_launch();
  kt_mark(7, st);
  if (kind == TAIL_PLAIN) launch_pdl(k_proj_tail<TAIL_PLAIN>, grid, dim3(TPB), 0, st, c, rcu, rcv, a, nbn, nbg, gate);
  else if (kind == TAIL_DEFECT) launch_pdl(k_proj_tail<TAIL_DEFECT>, grid, dim3(TPB), 0, st, c, rcu, rcv, a, nbn, nbg, gate);
  else launch_pdl(k_proj_tail<TAIL_PRESSURE>, grid, dim3(TPB), 0, st, c, rcu, rcv, a, nbn, nbg, gate);
  kt_mark(7, st);
}

__global__ void k_maxabs(CaseDev c, const double* __restrict__ U, unsigned long long* umax, unsigned long long* vmax,
                         Gate gate) {
  if (!gate_open(gate)) return;
  unsigned long long a = 0, b = 0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < c.usize + c.vsize;
       t += (int64_t)gridDim.x * blockDim.x) {
    if (t < c.usize) a = umax64(a, absbits(U[t]));
    else b = umax64(b, absbits(U[t]));
  }
  block_commit_max(a, umax);
  block_commit_max(b, vmax);
}
void launch_maxabs(const CaseDev& c, const double* U, unsigned long long* umax, unsigned long long* vmax,
                   const Gate& gate, cudaStream_t st) {
  note_launch();
  kt_mark(9, st);
  launch_pdl(k_maxabs, dim3(reduce_blocks(c.usize + c.vsize)), dim3(TPB), 0, st, c, U, umax, vmax, gate);
  kt_mark(9, st);
}

// ---------------------------------------------------------------------------
// surface forces (solver/optimized_ghost_cell.py:280-286) and step gates (solver/main.py:401-415)
// ---------------------------------------------------------------------------
// One warp a quadrature point (lanes over the stencils' nonzeros, the three rows' loads together):
// its four force terms to c.surf_part.
__device__ __forceinline__ void force_point(const CaseDev& c, const double* __restrict__ U, const double* __restrict__ P,
                                            double mu, int k) {
  const int lane = threadIdx.x & 31;
  if (k >= c.n_surf) return;
  const int64_t p0 = c.sp_ptr[k] + lane, p1 = c.sp_ptr[k + 1], u0 = c.su_ptr[k] + lane, u1 = c.su_ptr[k + 1];
  const int64_t v0 = c.sv_ptr[k] + lane, v1 = c.sv_ptr[k + 1];
  double ps = 0, du = 0, dv = 0;
  for (int64_t e = 0; p0 + e < p1 || u0 + e < u1 || v0 + e < v1; e += 32) {
    const bool bp = p0 + e < p1, bu = u0 + e < u1, bv = v0 + e < v1;
    const double xp = bp ? P[c.sp_col[p0 + e]] : 0.0, xu = bu ? U[c.su_col[u0 + e]] : 0.0;
    const double xv = bv ? U[c.usize + c.sv_col[v0 + e]] : 0.0;
    if (bp) ps += c.sp_val[p0 + e] * xp;
    if (bu) du += c.su_val[u0 + e] * xu;
    if (bv) dv += c.sv_val[v0 + e] * xv;
  }
  ps = warp_sum(ps);
  du = warp_sum(du);
  dv = warp_sum(dv);
  if (lane == 0) {
    const double nxk = c.nxx[k], nyk = c.nyy[k];
    const double dn = du * nxk + dv * nyk;
    double* o = c.surf_part + 4 * (int64_t)k;
    o[0] = ps * c.nwx[k];
    o[1] = ps * c.nwy[k];
    o[2] = mu * (du + nxk * dn);
    o[3] = mu * (dv + nyk * dn);
  }
}
// Whether this block is the last of the grid to get here (the others' force terms are visible to it).
__device__ __forceinline__ bool last_block(unsigned* ticket) {
  __threadfence();
  __syncthreads();
  __shared__ int last;
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  return true;
}
// The six forces from the point terms, in a fixed order, by the first four warps (w: arc length a
// point); on every thread after the barrier.
__device__ __forceinline__ void force_sums(const CaseDev& c, double w, double (&f6)[6]) {
  __shared__ double red[4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < 4) {
    double acc = 0.0;
#pragma unroll 4
    for (int q = lane; q < c.n_surf; q += 32) acc += __ldcg(c.surf_part + 4 * (int64_t)q + warp);
    acc = warp_sum(acc);
    if (lane == 0) red[warp] = acc;
  }
  __syncthreads();
  const double fp[2] = {-red[0], -red[1]}, fv[2] = {red[2] * w, red[3] * w};
  f6[0] = fp[0] + fv[0]; f6[1] = fp[1] + fv[1];
  f6[2] = fp[0]; f6[3] = fp[1];
  f6[4] = fv[0]; f6[5] = fv[1];
}
static inline double force_arc(const CaseDev& c) { return 3.141592653589793 * c.D / c.n_surf; }
constexpr int FORCE_WPB = 8;

__global__ void k_forces(CaseDev c, const double* __restrict__ U, const double* __restrict__ P, double mu, double w,
                         double* out6) {
  force_point(c, U, P, mu, (blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (!last_block(c.surf_ticket)) return;
  double f6[6];
  force_sums(c, w, f6);
  if (threadIdx.x == 0) {
    *c.surf_ticket = 0u;
    for (int q = 0; q < 6; ++q) out6[q] = f6[q];
  }
}
void launch_forces(const CaseDev& c, const double* U, const double* P, double mu, double* out6, cudaStream_t st) {
  note_launch();
  kt_mark(9, st);
  k_forces<<<(c.n_surf + FORCE_WPB - 1) / FORCE_WPB, 32 * FORCE_WPB, 0, st>>>(c, U, P, mu, force_arc(c), out6);
  kt_mark(9, st);
}

// The step record: the control block to the ring, the new maxima to the state (a good step), the
// counters, and the per-step part of the control block cleared for the next step.  One block.
__device__ void step_end(StepCtl* ctl, const StepTail& a) {
  __shared__ int slot, err;
  __syncthreads();
  if (threadIdx.x == 0) {
    slot = min(*a.ridx, a.cap - 1);
    err = *(volatile int*)&ctl->err;
    if (!err) {
      a.state_max[0] = ctl->umax;
      a.state_max[1] = ctl->vmax;
    }
  }
  __syncthreads();
  int* src = reinterpret_cast<int*>(ctl);
  int* dst = reinterpret_cast<int*>(a.ring + slot);
  constexpr int N = (int)(sizeof(StepCtl) / sizeof(int)), KEEP = (int)(offsetof(StepCtl, solve) / sizeof(int));
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    dst[i] = src[i];
    if (!err && i >= KEEP) src[i] = 0;
  }
  if (threadIdx.x == 0) {
    *a.ridx = slot + 1;
    *a.counter = *a.counter + 1;
  }
}

// The end of a step (StepTail): nbf blocks of force points, then blocks of both pressures' ghost rows;
// the last to finish sums the forces, applies the step gates and writes the record.  (Pressure ghost
// rows, maxima, forces, record and the next step's clearing of the control block were five launches.)
__global__ void k_step_tail(CaseDev c, StepTail a, double w, double denom, int nbf, int nbg, Gate gate) {
  StepCtl* ctl = gate.ctl;
  const bool open = gate_open(gate);
  if (!open || !projection_ok(ctl, 2)) {  // the same words for every block: all of them leave here
    if (blockIdx.x == 0) {
      if (open && threadIdx.x == 0) check_projection(ctl, 2);
      step_end(ctl, a);
    }
    return;
  }
  const int b = blockIdx.x;
  if (b < nbf) {
    force_point(c, a.U, a.pout, a.mu, (b * blockDim.x + threadIdx.x) >> 5);
  } else {
    double* f = b < nbf + nbg ? a.pout : a.half;
    const int t = (b - nbf - (b < nbf + nbg ? 0 : nbg)) * (int)blockDim.x + threadIdx.x, r = t / GHOST_LANES, l = t % GHOST_LANES;
    const double v = ghost_row(f, c.gp_ptr, c.gp_col, c.gp_val, r < c.n_ghost_p ? r : -1, l);
    if (r < c.n_ghost_p && l == 0) f[c.gp_rows[r]] = v;
  }
  if (!last_block(c.surf_ticket)) return;
  double f6[6];
  force_sums(c, w, f6);
  // the four quotients on four lanes: one divide's latency instead of four
  __shared__ double quot[4];
  if (threadIdx.x < 4) {
    const double um = bits2d(ctl->umax), vm = bits2d(ctl->vmax);
    const double num = threadIdx.x == 0 ? f6[0] : threadIdx.x == 1 ? f6[1] : threadIdx.x == 2 ? um : vm;
    quot[threadIdx.x] = num / (threadIdx.x < 2 ? denom : threadIdx.x == 2 ? c.dx : c.dy);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *c.surf_ticket = 0u;
    for (int q = 0; q < 6; ++q) ctl->forces[q] = f6[q];
    const double cd = quot[0], cl = quot[1];
    ctl->cd = cd;
    ctl->cl = cl;
    if (!isfinite(cd) || !isfinite(cl)) {
      raise_gate(ctl, 3, 6);
    } else {
      const double div = bits2d(ctl->div_max[1]), cfl = a.dt * (quot[2] + quot[3]);
      if (!(div < 1e-10) || !(cfl < 0.5)) raise_gate(ctl, 2, 5);
    }
  }
  step_end(ctl, a);
}
void launch_step_tail(const CaseDev& c, const StepTail& a, const Gate& gate, cudaStream_t st) {
  const int nbf = (c.n_surf + FORCE_WPB - 1) / FORCE_WPB, nbg = ghost_blocks(c.n_ghost_p);
  note_launch();
  kt_mark(9, st);
  launch_pdl(k_step_tail, dim3((unsigned)std::max(1, nbf + 2 * nbg)), dim3(32 * FORCE_WPB), 0, st, c, a, force_arc(c),
             ((0.5 * c.rho) * (c.U_ref * c.U_ref)) * c.D, nbf, nbg, gate);
  kt_mark(9, st);
}

__global__ void k_gate_pressure(StepCtl* ctl, int slot, int nchk, int sweeps) {
  if (!ctl->err) check_pressure(ctl, slot, nchk, sweeps);
}
void launch_gate_pressure(StepCtl* ctl, int slot, int nchk, int sweeps, cudaStream_t st) {
  note_launch();
  kt_mark(10, st);
  k_gate_pressure<<<1, 1, 0, st>>>(ctl, slot, nchk, sweeps);
  kt_mark(10, st);
}

__global__ void k_gate_projection(StepCtl* ctl, int k) {
  if (!ctl->err) check_projection(ctl, k);
}
void launch_gate_projection(StepCtl* ctl, int k, cudaStream_t st) {
  note_launch();
  kt_mark(10, st);
  k_gate_projection<<<1, 1, 0, st>>>(ctl, k);
  kt_mark(10, st);
}

__global__ void k_cfl_screen(StepCtl* ctl, const unsigned long long* umax, const unsigned long long* vmax, double dt,
                             double dx, double dy, int screen, const long long* counter) {
  if (!ctl->err) check_cfl(ctl, umax, vmax, dt, dx, dy, screen, counter);
}
void launch_cfl_screen(StepCtl* ctl, const unsigned long long* umax, const unsigned long long* vmax, double dt,
                       double dx, double dy, int screen, const long long* counter, cudaStream_t st) {
  note_launch();
  kt_mark(10, st);
  k_cfl_screen<<<1, 1, 0, st>>>(ctl, umax, vmax, dt, dx, dy, screen, counter);
  kt_mark(10, st);
}

// ---------------------------------------------------------------------------
// Flexible GMRES(50) with its control on the device (solver/pressure_schur.py:20-41): the
// Hessenberg column, the Givens rotations, the residual estimate, the convergence test and
// the least-squares update run in one-thread kernels on the device-resident GmresDev, and the
// loops are conditional graph nodes (restart cycles: WHILE; Arnoldi steps: one IF node per
// step, its condition set by the previous step).  The arithmetic is that of the host loop it
// replaces, in the same order.
// ---------------------------------------------------------------------------
__global__ void k_gm_init(GmresDev* gd, const double* __restrict__ bn2, cudaGraphConditionalHandle cycle,
                          double rtol, double atol) {
  gd->tol = fmax(rtol * sqrt(bn2[0]), atol);
  gd->iterations = 0;
  gd->converged = 0;
  gd->stop = 0;
  gd->cycle = 0;
  gd->jend = -1;
  gd->polish = 0;
  cudaGraphSetConditional(cycle, 1u);
}
// beta = ||b - A x||; the cycle's first step runs while beta > tol
__global__ void k_gm_cycle_begin(GmresDev* gd, const double* __restrict__ beta2, GmresHandles hs) {
  const double beta = sqrt(beta2[0]);
  gd->jend = -1;
  bool go = beta > gd->tol;
  if (!go) {
    gd->converged = isfinite(beta) ? 1 : 0;
    gd->stop = 1;
    gd->hscale = 1.0;
  } else {
    for (int i = 0; i <= GmresDev::M; ++i) gd->g[i] = 0.0;
    gd->g[0] = beta;
    gd->hscale = 1.0 / beta;
  }
  for (int j = 0; j < hs.count; ++j) cudaGraphSetConditional(hs.step[j], (j == 0 && go) ? 1u : 0u);
}
// w *= hscale (the new basis vector, or V_0 at the start of a cycle)
__global__ void k_gm_scale(double* __restrict__ w, int64_t n, const GmresDev* __restrict__ gd) {
  const double s = gd->hscale;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    w[t] *= s;
}
// end of Arnoldi step j: column j of H from the two Gram-Schmidt passes and the norm, the
// rotations, the residual estimate g[j+1]; step j + 1 runs while it is finite and above tol
__global__ void k_gm_step_end(GmresDev* gd, int j, const double* __restrict__ d1, const double* __restrict__ d2,
                              const double* __restrict__ wn2, cudaGraphConditionalHandle next, int has_next) {
  double hc[GmresDev::M + 1];
  for (int i = 0; i <= j; ++i) hc[i] = d1[i] + d2[i];
  hc[j + 1] = sqrt(wn2[0]);
  gd->hscale = hc[j + 1] > 0 ? 1.0 / hc[j + 1] : 1.0;
  for (int i = 0; i < j; ++i) {
    const double a = gd->cs[i] * hc[i] + gd->sn[i] * hc[i + 1];
    hc[i + 1] = -gd->sn[i] * hc[i] + gd->cs[i] * hc[i + 1];
    hc[i] = a;
  }
  const double den = hypot(hc[j], hc[j + 1]);
  gd->cs[j] = den > 0 ? hc[j] / den : 1.0;
  gd->sn[j] = den > 0 ? hc[j + 1] / den : 0.0;
  hc[j] = den;
  gd->g[j + 1] = -gd->sn[j] * gd->g[j];
  gd->g[j] = gd->cs[j] * gd->g[j];
  for (int i = 0; i <= j; ++i) gd->H[i * GmresDev::M + j] = hc[i];
  gd->iterations += 1;
  gd->jend = j;
  const double r = gd->g[j + 1];
  bool go = true;
  if (!isfinite(r)) go = false;
  else if (fabs(r) <= gd->tol) { gd->converged = 1; go = false; }
  if (has_next) cudaGraphSetConditional(next, go ? 1u : 0u);
}
// end of a cycle: y = R^{-1} g (the solve of the host loop), nv = its length for x += Z y; the
// next cycle runs while not converged, a step was taken and fewer than 100 cycles ran
__global__ void k_gm_cycle_end(GmresDev* gd, double* __restrict__ y, int* __restrict__ nv,
                               cudaGraphConditionalHandle cycle) {
  const int jend = gd->jend;
  for (int i = jend; i >= 0; --i) {
    double acc = gd->g[i];
    for (int k = i + 1; k <= jend; ++k) acc -= gd->H[i * GmresDev::M + k] * gd->y[k];
    gd->y[i] = acc / gd->H[i * GmresDev::M + i];
  }
  for (int i = 0; i <= jend; ++i) y[i] = gd->y[i];
  *nv = jend + 1;
  gd->cycle += 1;
  const bool go = jend >= 0 && !gd->converged && !gd->stop && gd->cycle < 100;
  cudaGraphSetConditional(cycle, go ? 1u : 0u);
}
// y += sum_{i < *nv} coef[i] V_i (the count on the device)
__global__ void k_multiaxpy_dev(const double* __restrict__ V, int64_t ld, const int* __restrict__ nvp,
                                const double* __restrict__ coef, double* __restrict__ y, int64_t n) {
  __shared__ double cf[GM_DOT_MAX + 1];
  const int nv = *nvp;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) cf[i] = coef[i];
  __syncthreads();
  if (nv <= 0) return;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int i = 0; i < nv; ++i) acc += cf[i] * V[(int64_t)i * ld + t];
    y[t] = 1.0 * y[t] + 1.0 * acc;
  }
}
void launch_gm_init(GmresDev* gd, const double* bn2, cudaGraphConditionalHandle cycle, cudaStream_t st, double rtol,
                    double atol) {
  note_launch();
  k_gm_init<<<1, 1, 0, st>>>(gd, bn2, cycle, rtol, atol);
}
void launch_gm_cycle_begin(GmresDev* gd, const double* beta2, const GmresHandles& hs, cudaStream_t st) {
  note_launch();
  k_gm_cycle_begin<<<1, 1, 0, st>>>(gd, beta2, hs);
}
void launch_gm_scale(double* w, int64_t n, const GmresDev* gd, cudaStream_t st) {
  note_launch();
  k_gm_scale<<<reduce_blocks(n), TPB, 0, st>>>(w, n, gd);
}
void launch_gm_step_end(GmresDev* gd, int j, const double* d1, const double* d2, const double* wn2,
                        cudaGraphConditionalHandle next, bool has_next, cudaStream_t st) {
  note_launch();
  k_gm_step_end<<<1, 1, 0, st>>>(gd, j, d1, d2, wn2, next, has_next ? 1 : 0);
}
void launch_gm_cycle_end(GmresDev* gd, double* y, int* nv, cudaGraphConditionalHandle cycle, cudaStream_t st) {
  note_launch();
  k_gm_cycle_end<<<1, 1, 0, st>>>(gd, y, nv, cycle);
}
void launch_multiaxpy_dev(const double* V, int64_t ld, const int* nv, const double* coef, double* y, int64_t n,
                          cudaStream_t st) {
  note_launch();
  k_multiaxpy_dev<<<reduce_blocks(n), TPB, 0, st>>>(V, ld, nv, coef, y, n);
}

// ---- FGMRES in the boundary rows' space (CompactGmres) ----------------------------------------
// An Arnoldi step over the grid is a rectangle inverse, the operator and two Gram-Schmidt passes over
// up to 50 grid vectors, some 15 kernels: 146 us at 512x256, 18 steps a solve.  With right
// preconditioning by T^-1 the operator is v -> v + E C T^-1 v, so in the coordinates (alpha, d) it is
// alpha' = alpha, d' = alpha G + K d with G = C T^-1 r / |r| and K formed with the boundary Schur matrix
// at set-up.  r / |r| and E are orthonormal, so the dot products, the rotations and the iterates are
// those of the grid iteration up to rounding.  V y = c v_0 + E e, so x takes c z_0 (z_0 = T^-1 v_0, formed as
// the grid iteration forms it, gives G as well) and T^-1 E e: two inverses a cycle.  A cycle is then some 15 kernels, of which k_cg_cycle does all Arnoldi
// steps on one cluster of eight SMs: the product with K by slices of rows (exchanged through distributed
// shared memory, one cluster barrier a step), Gram-Schmidt and rotations by every SM on its own copy.
// The model takes T^-1 as exact where the grid iteration sees the rounding of A T^-1, which left x with
// the direct solver's error (3e-12 against 2e-13 at 400x200).  A converged solve therefore runs one more,
// uncounted cycle on its true residual to CG_POLISH of it, after which x is nearer the exact solution
// than the grid iteration's.  FP32 preconditioning is not linear to 1e-12, so that mode keeps the grid iteration, and so do
// bodies with more rows than one SM's shared memory holds vectors of (CG_ROWS).  At 512x256 (58
// rows, 15-18 steps a solve) a time step took 5.3 ms, now 1.3.
constexpr int CG_CTAS = 8, CG_TPB = 256, CG_ROWS = 448;
constexpr int CG_M = GmresDev::M;
bool compact_gmres_fits(int n) { return n > 0 && n <= CG_ROWS; }
static size_t cg_smem(int n) {
  // V (M + 1 vectors), two copies of the exchanged vector, H, cs, sn, g, y, the step's coefficients, scratch
  return ((size_t)(CG_M + 1 + 2) * (n + 1) + CG_M * CG_M + 6 * (CG_M + 2) + 64) * sizeof(double);
}

// (k_gm_cycle_begin, and the correcting cycle's start)
constexpr double CG_POLISH = 0.02;
__global__ void k_cg_begin(GmresDev* gd, const double* __restrict__ beta2) {
  const double beta = sqrt(beta2[0]);
  gd->jend = -1;
  const bool go = gd->polish ? beta > 0.0 && isfinite(beta) : beta > gd->tol;
  if (!go) {
    if (!gd->polish) gd->converged = isfinite(beta) ? 1 : 0;
    gd->stop = 1;
    gd->hscale = 1.0;
    return;
  }
  gd->g[0] = beta;
  gd->hscale = 1.0 / beta;
  gd->ptol = CG_POLISH * beta;
}
void launch_cg_begin(GmresDev* gd, const double* beta2, cudaStream_t st) {
  note_launch();
  k_cg_begin<<<1, 1, 0, st>>>(gd, beta2);
}
__global__ void k_cg_offnorm(CaseDev c, const double* __restrict__ r, double* __restrict__ part) {
  __shared__ double red[TPB / 32];
  double acc = 0.0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < c.psize; t += (int64_t)gridDim.x * blockDim.x)
    if (!(c.cls_p[t] & CLS_IRREG)) acc += r[t] * r[t];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int q = 0; q < TPB / 32; ++q) s += red[q];
    part[blockIdx.x] = s;
  }
}
void launch_cg_offnorm(const CaseDev& c, const double* r, double* part, cudaStream_t st) {
  note_launch();
  kt_mark(6, st);
  k_cg_offnorm<<<reduce_blocks(c.psize), TPB, 0, st>>>(c, r, part);
  kt_mark(6, st, (double)c.psize * 9);
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_store(double* local, unsigned rank, double v) {  // to the same place in CTA `rank`
  unsigned a = (unsigned)__cvta_generic_to_shared(local), r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}

__global__ void __launch_bounds__(CG_TPB) k_cg_cycle(CompactGmres g, const double* __restrict__ v0, const double* __restrict__ z0,
                                                     const double* __restrict__ part, int npart, GmresDev* gd,
                                                     cudaGraphConditionalHandle cycle, double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = g.n, n1 = n + 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = CG_TPB / 32;
  double* V = reinterpret_cast<double*>(smem_raw);      // V_i at i n1: d (n values), then alpha
  double* wx = V + (size_t)(CG_M + 1) * n1;              // the exchanged vector, two copies by step parity
  double* H = wx + 2 * (size_t)n1;                       // rotated columns: H[i M + j]
  double* cs = H + CG_M * CG_M;
  double* sn = cs + CG_M + 2;
  double* gv = sn + CG_M + 2;
  double* y = gv + CG_M + 2;
  double* hc = y + CG_M + 2;                             // the step's column
  double* cf = hc + CG_M + 2;                            // a pass's coefficients
  double* sc = cf + CG_M + 2;                            // scratch: warp sums, broadcast scalars
  unsigned rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int slice = (n + CG_CTAS - 1) / CG_CTAS, ra = min(n, (int)rank * slice), rb = min(n, ra + slice);
  // block-wide sum of one value a thread, the same for every thread (two barriers)
  auto total = [&](double v) {
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) sc[warp] = v;
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < NW; ++q) s += sc[q];
    return s;
  };
  double acc = 0.0;
  for (int q = tid; q < npart; q += CG_TPB) acc += part[q];
  // k_cg_begin has decided whether the cycle runs; v0 is scaled
  const bool polish = gd->polish != 0;
  const double alpha0 = sqrt(total(acc)) * gd->hscale, tol = polish ? gd->ptol : gd->tol;
  int jend = -1, its = 0, converged = 0;
  const bool stop = gd->stop != 0;
  if (!stop) {
    for (int k = tid; k < n; k += CG_TPB) V[k] = v0[g.field[k]];
    if (tid == 0) {
      V[n] = alpha0;
      gv[0] = gd->g[0];
    }
    // K times the boundary part of `v` by rows of this CTA's slice, to every CTA's `w`; the barrier in
    // front of the first call makes the clusters' shared memory ready for remote stores
    auto product = [&](const double* v, double* w) {
      for (int r = ra + warp; r < rb; r += NW) {
        double s = 0.0;
        for (int k = lane; k < n; k += 32) s += g.K[(size_t)r * n + k] * v[k];
        s = warp_sum(s);
        if (lane < CG_CTAS) cluster_store(w + r, lane, s);
      }
      cluster_sync_all();
    };
    cluster_sync_all();
    product(V, wx + n1);
    // G = (C z0 - (K - I) d0) / alpha0 by this thread's rows, kept in registers (n <= 2 CG_TPB)
    const double ia = alpha0 > 0.0 ? 1.0 / alpha0 : 0.0;
    double G[2] = {0.0, 0.0};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int k = tid + u * CG_TPB;
      if (k < n) {
        const int r = g.crow[k];
        double s = 0.0;
        for (int64_t e = g.cptr[r]; e < g.cptr[r + 1]; ++e) s += g.cval[e] * z0[g.ccol[e]];
        G[u] = (s - (wx[n1 + k] - V[k])) * ia;
      }
    }
    for (int j = 0; j < CG_M; ++j) {
      const double* v = V + (size_t)j * n1;
      double* w = wx + (size_t)(j & 1) * n1;
      __syncthreads();
      if (tid == 0) w[n] = v[n];
      product(v, w);
      const double alpha = v[n];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = tid + u * CG_TPB;
        if (k < n) w[k] += alpha * G[u];
      }
      __syncthreads();
      // two classical Gram-Schmidt passes against V_0..V_j, then the norm
      for (int pass = 0; pass < 2; ++pass) {
        for (int i = warp; i <= j; i += NW) {
          const double* vi = V + (size_t)i * n1;
          double s = 0.0;
          for (int k = lane; k < n1; k += 32) s += vi[k] * w[k];
          s = warp_sum(s);
          if (lane == 0) {
            cf[i] = s;
            hc[i] = pass ? hc[i] + s : s;
          }
        }
        __syncthreads();
        for (int k = tid; k < n1; k += CG_TPB) {
          double s0 = 0.0, s1 = 0.0;
          int i = 0;
          for (; i + 1 <= j; i += 2) {
            s0 += cf[i] * V[(size_t)i * n1 + k];
            s1 += cf[i + 1] * V[(size_t)(i + 1) * n1 + k];
          }
          if (i <= j) s0 += cf[i] * V[(size_t)i * n1 + k];
          w[k] -= s0 + s1;
        }
        __syncthreads();
      }
      acc = 0.0;
      for (int k = tid; k < n1; k += CG_TPB) acc += w[k] * w[k];
      const double hn = sqrt(total(acc)), scale = hn > 0 ? 1.0 / hn : 1.0;
      for (int k = tid; k < n1; k += CG_TPB) V[(size_t)(j + 1) * n1 + k] = w[k] * scale;
      // the rotations of k_gm_step_end
      if (tid == 0) {
        hc[j + 1] = hn;
        for (int i = 0; i < j; ++i) {
          const double a = cs[i] * hc[i] + sn[i] * hc[i + 1];
          hc[i + 1] = -sn[i] * hc[i] + cs[i] * hc[i + 1];
          H[i * CG_M + j] = a;
        }
        const double den = hypot(hc[j], hc[j + 1]);
        cs[j] = den > 0 ? hc[j] / den : 1.0;
        sn[j] = den > 0 ? hc[j + 1] / den : 0.0;
        H[j * CG_M + j] = den;
        gv[j + 1] = -sn[j] * gv[j];
        gv[j] = cs[j] * gv[j];
      }
      __syncthreads();
      ++its;
      jend = j;
      const double r = gv[j + 1];
      if (!isfinite(r)) break;
      if (fabs(r) <= tol) { converged = 1; break; }
    }
  }
  // no CTA leaves (or ends) while another may still store into its shared memory: the last exchange
  // is behind every CTA's last cluster barrier, so none can
  if (rank != 0) return;
  if (tid == 0) {
    for (int i = jend; i >= 0; --i) {
      double a = gv[i];
      for (int k = i + 1; k <= jend; ++k) a -= H[i * CG_M + k] * y[k];
      y[i] = a / H[i * CG_M + i];
    }
    gd->jend = jend;
    gd->cycle += 1;
    bool go = false;
    if (!polish) {
      gd->iterations += its;
      if (converged) gd->converged = 1;
      go = jend >= 0 && !stop && (converged || gd->cycle < 100);
      if (go && converged) gd->polish = 1;
    }
    cudaGraphSetConditional(cycle, go ? 1u : 0u);
  }
  __syncthreads();
  double f = 0.0;  // the factor of v0
  if (jend >= 0 && alpha0 > 0.0) {
    for (int i = 0; i <= jend; ++i) f += y[i] * V[(size_t)i * n1 + n];
    f /= alpha0;
  }
  for (int k = tid; k < n; k += CG_TPB) {
    double s = 0.0;
    for (int i = 0; i <= jend; ++i) s += y[i] * V[(size_t)i * n1 + k];
    out[1 + k] = jend >= 0 ? s - f * V[k] : 0.0;
  }
  if (tid == 0) out[0] = f;
}
void launch_cg_cycle(const CaseDev& c, const CompactGmres& g, const double* v0, const double* z0, const double* part,
                     GmresDev* gd, cudaGraphConditionalHandle cycle, double* out, cudaStream_t st) {
  note_launch();
  kt_mark(6, st);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(CG_CTAS);
  cfg.blockDim = dim3(CG_TPB);
  cfg.dynamicSmemBytes = cg_smem(g.n);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CG_CTAS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_cg_cycle, g, v0, z0, part, (int)reduce_blocks(c.psize), gd, cycle, out);
  kt_mark(6, st);
}

__global__ void k_cg_combine(CaseDev c, CompactGmres g, const double* __restrict__ z0, const double* __restrict__ out,
                             double* __restrict__ x, double* __restrict__ e) {
  const double f = out[0];
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < c.psize; t += (int64_t)gridDim.x * blockDim.x)
    if (c.cls_p[t] & CLS_ACTIVE) x[t] += f * z0[t];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.n; k += gridDim.x * blockDim.x) e[g.field[k]] = out[1 + k];
}
void launch_cg_combine(const CaseDev& c, const CompactGmres& g, const double* z0, const double* out, double* x, double* e,
                       cudaStream_t st) {
  note_launch();
  kt_mark(6, st);
  k_cg_combine<<<reduce_blocks(c.psize), TPB, 0, st>>>(c, g, z0, out, x, e);
  kt_mark(6, st, (double)c.psize * 25);
}

__global__ void k_copy_active(const uint8_t* __restrict__ cls, int64_t n, const double* __restrict__ src,
                              double* __restrict__ dst, Gate gate) {
  if (!gate_open(gate)) return;
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) dst[t] = (cls[t] & CLS_ACTIVE) ? src[t] : 0.0;
}
void launch_copy_active(const uint8_t* cls, int64_t n, const double* src, double* dst, const Gate& gate,
                        cudaStream_t st) {
  note_launch();
  launch_pdl(k_copy_active, dim3(blocks_for(n)), dim3(TPB), 0, st, cls, n, src, dst, gate);
}

__global__ void k_set_inlet(CaseDev c, double* U, int zero) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < c.ny) U[(int64_t)j * (c.nx + 1)] = zero ? 0.0 : c.inlet[j];
}
void launch_set_inlet(const CaseDev& c, double* U, bool zero, cudaStream_t st) {
  note_launch();
  kt_mark(6, st);
  k_set_inlet<<<blocks_for(c.ny, 128), 128, 0, st>>>(c, U, zero ? 1 : 0);
  kt_mark(6, st);
}

// mac_engine.calculate_mac_divergence_cpp (solver/src/bindings.cpp:343-390)
__global__ void k_div_stats(CaseDev c, const double* __restrict__ U, const uint8_t* __restrict__ mask, double* out5) {
  const Grid g{c.nx, c.ny, c.usize};
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long m = 0;
  double s = 0, cs = 0, n = 0, cn = 0;
  if (t < c.psize && !mask[t]) {
    int j = (int)(t / c.nx), i = (int)(t % c.nx);
    double d = (U[g.u(j, i + 1)] - U[g.u(j, i)]) / c.dx + (U[g.v(j + 1, i)] - U[g.v(j, i)]) / c.dy;
    m = absbits(d);
    s = d * d;
    n = 1;
    bool core = true;
    if (i > 0 && mask[t - 1]) core = false;
    if (i < c.nx - 1 && mask[t + 1]) core = false;
    if (j > 0 && mask[t - c.nx]) core = false;
    if (j < c.ny - 1 && mask[t + c.nx]) core = false;
    if (core) { cs = d * d; cn = 1; }
  }
  block_commit_max(m, reinterpret_cast<unsigned long long*>(&out5[0]));
  block_commit_sum(s, &out5[1]);
  block_commit_sum(n, &out5[2]);
  block_commit_sum(cs, &out5[3]);
  block_commit_sum(cn, &out5[4]);
}
void launch_divergence_stats(const CaseDev& c, const double* U, const uint8_t* mask, double* out5, cudaStream_t st) {
  note_launch();
  k_div_stats<<<blocks_for(c.psize), TPB, 0, st>>>(c, U, mask, out5);
}

__global__ void k_gather(const double* __restrict__ src, const int64_t* __restrict__ idx, int64_t n,
                         double* __restrict__ dst) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) dst[t] = src[idx[t]];
}
__global__ void k_scatter(const double* __restrict__ src, const int64_t* __restrict__ idx, int64_t n,
                          double* __restrict__ dst) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) dst[idx[t]] = src[t];
}
void launch_gather(const double* src, const int64_t* idx, int64_t n, double* dst, cudaStream_t st) {
  if (n > 0) {
    note_launch();
    k_gather<<<blocks_for(n), TPB, 0, st>>>(src, idx, n, dst);
  }
}
void launch_scatter(const double* src, const int64_t* idx, int64_t n, double* dst, cudaStream_t st) {
  if (n > 0) {
    note_launch();
    k_scatter<<<blocks_for(n), TPB, 0, st>>>(src, idx, n, dst);
  }
}

__global__ void k_schur_column(const double* __restrict__ first, RectView v, int rank, const int64_t* __restrict__ cp,
                               const int64_t* __restrict__ cc, const double* __restrict__ cv, double* __restrict__ S,
                               int col) {
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rank) return;
  double acc = 0.0;
  for (int64_t e = cp[r]; e < cp[r + 1]; ++e) acc += cv[e] * first[cc[e]];  // cc: field-grid flat indices
  S[(int64_t)r * rank + col] = acc;
}
void launch_schur_column(const double* first, const RectView& view, int rank, const int64_t* c_ptr,
                         const int64_t* c_col, const double* c_val, double* S, int col, cudaStream_t st) {
  if (rank > 0) {
    note_launch();
    k_schur_column<<<blocks_for(rank, 128), 128, 0, st>>>(first, view, rank, c_ptr, c_col, c_val, S, col);
  }
}

// ---------------------------------------------------------------------------
// case-indexed launches: blockIdx.y selects the case, its arguments come from the kernel's
// parameter space; blocks past the case's own grid return at once
// ---------------------------------------------------------------------------
template <typename T, typename TI, typename TO>
__global__ void k_xpass_multi(const __grid_constant__ ArgPack<XpassArgs<T, TI, TO>> p) {
  const XpassArgs<T, TI, TO>& a = p.a[blockIdx.y];
  if ((int)blockIdx.x >= a.nblk) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const R2RTables<T> ts = xpass_stage_tables<T>(a.type, a.n, a.plan, a.tb, smem_raw);
  if (!gate_open(a.gate)) return;
  xpass_block<T, TI, TO, false>(blockIdx.x, a.n, a.r0, a.nr, a.type, a.plan, ts, a.in, a.ibase, a.ipitch, a.icls, a.out,
                         a.obase, a.opitch, a.ocls, a.add, a.corr, a.gthreads, a.gpb, smem_raw);
}
template <typename T, int L>
__global__ void k_ysolve_multi(const __grid_constant__ ArgPack<YsolveArgs<T>> p) {
  const YsolveArgs<T>& a = p.a[blockIdx.y];
  if ((int)blockIdx.x >= a.nblk) return;
  if (!gate_open(a.gate)) return;
  ysolve_body<T, L>(a.rows, a.cols, a.ch, a.gamma, a.scale, a.t0, a.t1, a.t2, a.S, blockIdx.x);
}
template <typename T>
__global__ void __launch_bounds__(BAND_TPB) k_band_first_multi(const __grid_constant__ ArgPack<BandFirstArgs<T>> p) {
  const BandFirstArgs<T>& a = p.a[blockIdx.y];
  if ((int)blockIdx.x >= a.m) return;
  if (!gate_open(a.gate)) return;
  band_first_body<T>(a.n, a.mrow, a.binv, a.spec, a.firstm, blockIdx.x);
}
template <typename T>
__global__ void __launch_bounds__(BAND_TPB) k_band_gemv_multi(const __grid_constant__ ArgPack<BandGemvArgs<T>> p) {
  const BandGemvArgs<T>& a = p.a[blockIdx.y];
  if ((int)blockIdx.x >= a.rank) return;
  if (!gate_open(a.gate)) return;
  band_gemv_body<T>(a.m, a.M, a.firstm, a.c, blockIdx.x);
}
template <typename T>
__global__ void __launch_bounds__(BAND_TPB) k_band_direct_multi(const __grid_constant__ ArgPack<BandDirectArgs<T>> p) {
  const BandDirectArgs<T>& a = p.a[blockIdx.y];
  if ((int)blockIdx.x >= a.rank * BAND_SPLIT) return;
  if (!gate_open(a.gate)) return;
  band_direct_body<T>(a.L, a.G, a.S, a.part, blockIdx.x / BAND_SPLIT, blockIdx.x % BAND_SPLIT);
}
template <typename T>
__global__ void __launch_bounds__(BAND_COLS * BAND_ROWT) k_band_fwd_solve_multi(
    const __grid_constant__ ArgPack<BandFwdArgs<T>> p) {
  const BandFwdArgs<T>& a = p.a[blockIdx.y];
  if ((int)blockIdx.x >= a.nblk) return;
  if (!gate_open(a.gate)) return;
  band_fwd_solve_body<T>(a.nb, a.n, a.rank, a.bptr, a.c, a.bfwd, a.gamma, a.scale, a.bpiv, a.band,
                         blockIdx.x, a.nsplit);
}
template <int KIND, bool RES_F32>
__global__ void k_residual_multi(const __grid_constant__ ArgPack<ResidualArgs> p) {
  const ResidualArgs& a = p.a[blockIdx.y];
  if ((int)blockIdx.x >= a.nblk) return;
  if (!gate_open(a.gate)) return;
  residual_body<KIND, RES_F32>(a.c, a.rc, a.b, a.x, a.res, a.sc, a.check, a.first, blockIdx.x, a.nblk);
}
__global__ void k_refine_decide_multi(const __grid_constant__ ArgPack<StepCtl*> ctls, int n, int slot, int nchk,
                                      cudaGraphConditionalHandle cond) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  for (int c = threadIdx.x; c < n; c += blockDim.x) {
    StepCtl* ctl = ctls.a[c];
    SolveCtl* sc = &ctl->solve[slot];
    const int k = sc->k;
    bool need = false;
    if (!ctl->err) need = bits2d(sc->rmax[k]) > inner_target(sc) && k + 1 < nchk;
    if (need) {
      sc->k = k + 1;
      atomicOr(&any, 1);
    }
    sc->act = need ? 1 : 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) cudaGraphSetConditional(cond, any ? 1u : 0u);
}

template <typename T, typename TI, typename TO>
XpassArgs<T, TI, TO> xpass_args(const TransformTables& tt, bool inverse, int r0, int nr, const TI* in, int64_t ibase,
                                int64_t ipitch, const uint8_t* icls, TO* out, int64_t obase, int64_t opitch,
                                const uint8_t* ocls, const double* add, const YCorr<T>& corr, const Gate& gate) {
  using Cx = cplx<T>;
  XpassArgs<T, TI, TO> a{};
  a.n = tt.n;
  a.r0 = r0;
  a.nr = nr;
  a.type = inverse ? tt.tx_inv : tt.tx_fwd;
  a.plan = tt.plan_x;
  a.tb = R2RTables<T>{(const Cx*)tt.Wx, (const Cx*)(inverse ? tt.prex_inv : tt.prex),
                      (const Cx*)(inverse ? tt.postx_inv : tt.postx)};
  a.in = in;
  a.ibase = ibase;
  a.ipitch = ipitch;
  a.icls = icls;
  a.out = out;
  a.obase = obase;
  a.opitch = opitch;
  a.ocls = ocls;
  a.add = add;
  a.corr = corr;
  a.gthreads = tt.xg_threads;
  a.gpb = tt.xg_pb;
  a.gate = gate;
  const int per_block = tt.xg_pb * xpass_lines(a.type, 0);
  a.nblk = (nr + per_block - 1) / per_block;
  return a;
}
template <typename T>
YsolveArgs<T> ysolve_args(const TransformTables& tt, int cols, int rows, T* S, const Gate& gate) {
  YsolveArgs<T> a{};
  a.rows = rows;
  a.cols = cols;
  a.ch = tt.ych;
  a.gamma = (T)tt.gamma;
  a.scale = (T)tt.yscale;
  a.t0 = (const T*)tt.t0;
  a.t1 = (const T*)tt.t1;
  a.t2 = (const T*)tt.t2;
  a.S = S;
  a.gate = gate;
  a.nblk = (cols + tt.lpb_y - 1) / tt.lpb_y;
  return a;
}
ResidualArgs residual_args(const CaseDev& c, const ResidualCoef& rc, int kind, const double* b, const double* x,
                           void* res, bool res_f32, SolveCtl* sc, int check, bool first_check, const Gate& gate) {
  ResidualArgs a{};
  a.c = c;
  a.rc = rc;
  a.b = b;
  a.x = x;
  a.res = res;
  a.sc = sc;
  a.check = check;
  a.first = first_check ? 1 : 0;
  a.gate = gate;
  a.nblk = (int)residual_blocks(kind == 0 ? c.psize : (kind == 1 ? c.usize : c.vsize), res_f32);
  return a;
}

static_assert(sizeof(ArgPack<ResidualArgs>) <= 32000 &&
                  sizeof(ArgPack<YsolveArgs<double>>) <= 32000 &&
                  sizeof(ArgPack<XpassArgs<double, double, double>>) <= 32000,
              "case-indexed argument packs must fit the kernel parameter space");
template <typename A>
static unsigned max_blocks(const ArgPack<A>& p, int n) {
  int m = 0;
  for (int c = 0; c < n; ++c) m = std::max(m, p.a[c].nblk);
  return (unsigned)std::max(m, 1);
}
template <typename T, typename TI, typename TO>
void launch_xpass_multi(const ArgPack<XpassArgs<T, TI, TO>>& p, int n, const TransformTables& tt0, cudaStream_t st) {
  if (n <= 0) return;
  note_launch();
  k_xpass_multi<T, TI, TO><<<dim3(max_blocks(p, n), (unsigned)n), tt0.xg_threads * tt0.xg_pb, tt0.smem_x, st>>>(p);
}
template <typename T>
void launch_ysolve_multi(const ArgPack<YsolveArgs<T>>& p, int n, const TransformTables& tt0, cudaStream_t st) {
  if (n <= 0) return;
  note_launch();
  const dim3 g(max_blocks(p, n), (unsigned)n);
  switch (tt0.lpb_y) {
    case 2: k_ysolve_multi<T, 2><<<g, tt0.threads_y, tt0.smem_y, st>>>(p); break;
    case 4: k_ysolve_multi<T, 4><<<g, tt0.threads_y, tt0.smem_y, st>>>(p); break;
    case 8: k_ysolve_multi<T, 8><<<g, tt0.threads_y, tt0.smem_y, st>>>(p); break;
    default: k_ysolve_multi<T, 16><<<g, tt0.threads_y, tt0.smem_y, st>>>(p); break;
  }
}
template <typename T>
void launch_band_first_multi(const ArgPack<BandFirstArgs<T>>& p, int n, cudaStream_t st) {
  if (n <= 0) return;
  int m = 1;
  for (int c = 0; c < n; ++c) m = std::max(m, p.a[c].m);
  note_launch();
  k_band_first_multi<T><<<dim3((unsigned)m, (unsigned)n), BAND_TPB, 0, st>>>(p);
}
template <typename T>
void launch_band_gemv_multi(const ArgPack<BandGemvArgs<T>>& p, int n, cudaStream_t st) {
  if (n <= 0) return;
  int r = 1;
  for (int c = 0; c < n; ++c) r = std::max(r, p.a[c].rank);
  note_launch();
  k_band_gemv_multi<T><<<dim3((unsigned)r, (unsigned)n), BAND_TPB, 0, st>>>(p);
}
template <typename T>
void launch_band_direct_multi(const ArgPack<BandDirectArgs<T>>& p, int n, cudaStream_t st) {
  if (n <= 0) return;
  int r = 1;
  for (int c = 0; c < n; ++c) r = std::max(r, p.a[c].rank);
  note_launch();
  k_band_direct_multi<T><<<dim3((unsigned)(r * BAND_SPLIT), (unsigned)n), BAND_TPB, 0, st>>>(p);
}
template <typename T>
void launch_band_fwd_solve_multi(const ArgPack<BandFwdArgs<T>>& p, int n, cudaStream_t st) {
  if (n <= 0) return;
  size_t smem = 0;
  for (int c = 0; c < n; ++c) smem = std::max(smem, band_fwd_smem(p.a[c].nb, p.a[c].rank, sizeof(T) == 4));
  note_launch();
  k_band_fwd_solve_multi<T><<<dim3(max_blocks(p, n), (unsigned)n), BAND_COLS * BAND_ROWT, smem, st>>>(p);
}
void launch_residual_multi(const ArgPack<ResidualArgs>& p, int n, int kind, bool res_f32, cudaStream_t st) {
  if (n <= 0) return;
  note_launch();
  const dim3 g(max_blocks(p, n), (unsigned)n);
  if (res_f32) {
    if (kind == 0) k_residual_multi<0, true><<<g, TPB, 0, st>>>(p);
    else if (kind == 1) k_residual_multi<1, true><<<g, TPB, 0, st>>>(p);
    else k_residual_multi<2, true><<<g, TPB, 0, st>>>(p);
  } else {
    if (kind == 0) k_residual_multi<0, false><<<g, TPB, 0, st>>>(p);
    else if (kind == 1) k_residual_multi<1, false><<<g, TPB, 0, st>>>(p);
    else k_residual_multi<2, false><<<g, TPB, 0, st>>>(p);
  }
}
void launch_refine_decide_multi(const ArgPack<StepCtl*>& ctls, int n, int slot, int nchk,
                                cudaGraphConditionalHandle cond, cudaStream_t st) {
  note_launch();
  k_refine_decide_multi<<<1, 32, 0, st>>>(ctls, n, slot, nchk, cond);
}

#define GM_XPASS_MULTI(T, TI, TO)                                                                                   \
  template XpassArgs<T, TI, TO> xpass_args<T, TI, TO>(const TransformTables&, bool, int, int, const TI*, int64_t, \
                                                      int64_t, const uint8_t*, TO*, int64_t, int64_t,             \
                                                      const uint8_t*, const double*, const YCorr<T>&, const Gate&); \
  template void launch_xpass_multi<T, TI, TO>(const ArgPack<XpassArgs<T, TI, TO>>&, int, const TransformTables&,   \
                                              cudaStream_t);
GM_XPASS_MULTI(double, double, double)
GM_XPASS_MULTI(float, double, float)
GM_XPASS_MULTI(float, float, float)
GM_XPASS_MULTI(float, float, double)
#undef GM_XPASS_MULTI
template YsolveArgs<double> ysolve_args<double>(const TransformTables&, int, int, double*, const Gate&);
template YsolveArgs<float> ysolve_args<float>(const TransformTables&, int, int, float*, const Gate&);
template void launch_ysolve_multi<double>(const ArgPack<YsolveArgs<double>>&, int, const TransformTables&,
                                          cudaStream_t);
template void launch_ysolve_multi<float>(const ArgPack<YsolveArgs<float>>&, int, const TransformTables&,
                                         cudaStream_t);
template void launch_band_first_multi<double>(const ArgPack<BandFirstArgs<double>>&, int, cudaStream_t);
template void launch_band_first_multi<float>(const ArgPack<BandFirstArgs<float>>&, int, cudaStream_t);
template void launch_band_gemv_multi<double>(const ArgPack<BandGemvArgs<double>>&, int, cudaStream_t);
template void launch_band_gemv_multi<float>(const ArgPack<BandGemvArgs<float>>&, int, cudaStream_t);
template void launch_band_direct_multi<double>(const ArgPack<BandDirectArgs<double>>&, int, cudaStream_t);
template void launch_band_direct_multi<float>(const ArgPack<BandDirectArgs<float>>&, int, cudaStream_t);
template void launch_band_fwd_solve_multi<double>(const ArgPack<BandFwdArgs<double>>&, int, cudaStream_t);
template void launch_band_fwd_solve_multi<float>(const ArgPack<BandFwdArgs<float>>&, int, cudaStream_t);

}  // namespace gmk
