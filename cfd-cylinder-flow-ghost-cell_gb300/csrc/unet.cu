// Learned pressure preconditioner: a 4-level convolutional U-Net on the pressure grid with
// BF16 weights and FP32 activations / accumulation; forward, backward (data and weight
// gradients) and Adam kernels.  It has no reference counterpart: it is the learned slot in
// the GMRES preconditioner (solver/pressure_schur.py:20-27, 39-41).
//
// Architecture (fixed): channels c = (16, 32, 64, 64) on levels 0..3 (level l has the grid
// coarsened 2^l times by 2x2 averaging).  Encoder: two 3x3 convolutions + ReLU per level
// (input: 2 channels, the normalised residual and the active mask).  Decoder: nearest 2x
// upsampling, concatenation with the encoder output of the level, one 3x3 convolution +
// ReLU.  Output: a 3x3 convolution to one channel (linear).  Twelve convolutions, 253,872
// weights and 465 biases.  Tensors are [batch][channel][height][width], zero padding.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "../../include/ghostmac.h"

namespace gmk {
void kernel_launch_adjust(long long delta);  // the library's launch counter (kernels.cu)
}

namespace {

constexpr int NL = 12;
struct LayerDef {
  int cin, cout, level;
  bool relu;
};
constexpr LayerDef LAYERS[NL] = {{2, 16, 0, true},   {16, 16, 0, true},  {16, 32, 1, true}, {32, 32, 1, true},
                                 {32, 64, 2, true},  {64, 64, 2, true},  {64, 64, 3, true}, {64, 64, 3, true},
                                 {128, 64, 2, true}, {96, 32, 1, true},  {48, 16, 0, true}, {16, 1, 0, false}};

struct UnetError : std::exception {
  std::string msg;
  explicit UnetError(std::string m) : msg(std::move(m)) {}
  const char* what() const noexcept override { return msg.c_str(); }
};
#define UN_CK(call)                                                                                \
  do {                                                                                             \
    cudaError_t e_ = (call);                                                                       \
    if (e_ != cudaSuccess) throw UnetError(std::string(#call) + ": " + cudaGetErrorString(e_));    \
  } while (0)

// ---- 3x3 convolution ------------------------------------------------------------------------
// forward:        out[b][co] = bias[co] + sum_ci sum_k W[co][ci][k] in[b][ci](p + d_k)
// transposed:     out[b][ci] = sum_co sum_k W[co][ci][k] in[b][co](p - d_k)      (data gradient)
//
// FP32 on the CUDA cores (activations stay FP32, so the tensor cores' BF16 operands would need
// three-way splits), bound by the fused multiply-adds: a thread keeps 4 x 2 pixels x CO = 8 channels in
// registers, so that an input channel's 576 multiply-adds take 8 loads of its 6 x 4 window and 18
// broadcast loads of weights from shared memory; one pixel x 8 channels (72 multiply-adds for 27 loads)
// ran at 8 TFLOP/s.  Every output adds its products in the order ci, k, two output channels an
// instruction (fma.rn.f32x2, each half rounded as a single one): as single multiply-adds they left the
// FMA pipe at half of its rate, the issue slots at 70 %.  The forward pass of 4 x 512 x 1024 took 8.0 ms,
// 4.0 in this form with single multiply-adds, 3.5 now (35 TFLOP/s of 74); data gradients 3.4 ms, weight
// gradients 5.7 (21 TFLOP/s: 35 % of their issue slots are products, the rest staging and copies into
// pairs); a whole training pass 45 ms, now 13.
// The layers' glue runs in the loads and stores: the decoder's concatenation with the upsampled half
// (load), bias, ReLU and the 2 x 2 average for the next level (forward store), the ReLU masks, the
// upsampling's and the pooling's adjoints (gradient store).
// Inputs are staged KC channels at a time, row by row with asynchronous copies two stages ahead.
constexpr int CO = 8, PX = 4, PY = 2, NT = 256, KC = 2, STAGES = 3;

typedef unsigned long long f32x2;  // two floats, low word first
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// A tensor of cin channels on an H x W grid: channels [0, cu) of `up` (half the resolution, nearest
// 2x upsampling), the rest of `in`.
struct ConvIn {
  const float* in;
  const float* up;
  int cin, cu;
};
__device__ __forceinline__ void copy_async4(float* dst, const float* src, bool take) {  // zero when not taken
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(take ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Rows y0 - HALO .. (up to ROWS, those that points inside the grid read) x COLS columns from x0 - HALO
// of channels c0 .. c0 + nc - 1 into dst[channel][row][PITCH], zero outside the grid; a warp a row, lanes along x (coalesced, one
// address a row: forming every element's indices cost as many instructions as half the products).
// PAIRS: two channels side by side, dst[channel / 2][row][column][channel % 2].
template <int ROWS, int COLS, int PITCH, int HALO, bool PAIRS = false>
__device__ __forceinline__ void stage_rows(float* dst, const ConvIn& c, int b, int c0, int nc, int H, int W, int y0, int x0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto row = [&](int cc, int yy) {
    const int ci = c0 + cc, gy = y0 + yy - HALO;
    const bool up = ci < c.cu, ok = gy >= 0 && gy < H && ci < c.cin;
    const float* src = c.in;
    if (ok)
      src = up ? c.up + (((size_t)b * c.cu + ci) * (H >> 1) + (gy >> 1)) * (W >> 1)
               : c.in + (((size_t)b * (c.cin - c.cu) + ci - c.cu) * H + gy) * W;
    float* d = PAIRS ? dst + ((cc >> 1) * ROWS + yy) * PITCH * 2 + (cc & 1) : dst + (cc * ROWS + yy) * PITCH;
#pragma unroll
    for (int j = 0; j < COLS; j += 32) {
      const int xx = j + lane, gx = x0 + xx - HALO;
      const bool take = ok && gx >= 0 && gx < W;
      if (xx < COLS) copy_async4(d + (PAIRS ? 2 * xx : xx), src + (take ? (up ? gx >> 1 : gx) : 0), take);
    }
  };
  const int rows = min(ROWS, H - y0 + 2 * HALO);
  if (rows == ROWS)
    for (int r = warp; r < nc * ROWS; r += NT / 32) row(r / ROWS, r % ROWS);
  else  // the grid's last rows
    for (int r = warp; r < nc * rows; r += NT / 32) row(r / rows, r % rows);
}

enum : int { EPI_FWD = 0, EPI_MASK = 1, EPI_CAT = 2, EPI_POOL = 3 };
// What the store does with the convolution's value v at (b, co, y, x):
//   FWD   out = [relu](v); pool (may be null): the 2 x 2 averages of out
//   MASK  out = v where act > 0, else 0
//   CAT   co < cu: out2 (half resolution, cu channels) = the 2 x 2 sums of v where act > 0; the rest:
//         out = v (cout - cu channels), the encoder output's part from this skip
//   POOL  the four pixels of the double-resolution out under (y, x): (out + v / 4) where act > 0
struct ConvOut {
  float* out;
  float* out2;
  const float* act;
  int cu, relu;
};

template <int TX, int CB>
struct ConvTile {
  static constexpr int TY = NT / TX, TW = TX * PX, TH = TY * PY, PITCH = TW + 4;
  float tile[STAGES][KC][TH + 2][PITCH];
  float wt[STAGES][KC][9][CB];
};
// CB output channels a thread: 8, or 4 where 8 would leave SMs without a block
template <bool TRANSPOSED, int EPI, int TX, int CB>
__global__ void __launch_bounds__(NT, 2) k_conv3(int H, int W, int cout, ConvIn in, const __nv_bfloat16* __restrict__ w,
                                                 const float* __restrict__ bias, ConvOut o) {
  using T = ConvTile<TX, CB>;
  constexpr int TW = T::TW, TH = T::TH, PITCH = T::PITCH, CO = CB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T& sm = *reinterpret_cast<T*>(smem_raw);
  const int nco = (cout + CO - 1) / CO;
  const int b = blockIdx.z / nco, co0 = (blockIdx.z % nco) * CO;
  const int x0 = blockIdx.x * TW, y0 = blockIdx.y * TH;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const bool busy = __any_sync(0xffffffffu, x0 + tx * PX < W && y0 + ty * PY < H);  // a pixel of this warp is inside
  f32x2 acc[PY][PX][CO / 2];
#pragma unroll
  for (int c = 0; c < CO; c += 2) {
    const bool has = !TRANSPOSED && bias;
    const f32x2 v = pack2(has && co0 + c < cout ? bias[co0 + c] : 0.f, has && co0 + c + 1 < cout ? bias[co0 + c + 1] : 0.f);
#pragma unroll
    for (int r = 0; r < PY; ++r)
#pragma unroll
      for (int q = 0; q < PX; ++q) acc[r][q][c / 2] = v;
  }
  // this thread's weight of a stage (KC x 9 x CO of them): channel wcc, tap wk, output wc
  static_assert(KC * 9 * CO <= NT, "one weight a thread");
  const int wcc = threadIdx.x / (9 * CO), wk = threadIdx.x / CO % 9, wc = threadIdx.x % CO;
  auto stage = [&](int c0, int buf) {
    stage_rows<TH + 2, TW + 2, PITCH, 1>(&sm.tile[buf][0][0][0], in, b, c0, min(KC, in.cin - c0), H, W, y0, x0);
    copy_commit();
    if (threadIdx.x < KC * 9 * CO) {
      const int ci = c0 + wcc, co = co0 + wc;
      float v = 0.f;
      if (ci < in.cin && co < cout)
        // forward: W[co][ci][k]; transposed: the output channel is an input channel of the
        // layer (ci here runs over the layer's outputs) and the taps are mirrored
        v = __bfloat162float(TRANSPOSED ? w[((size_t)ci * cout + co) * 9 + (8 - wk)] : w[((size_t)co * in.cin + ci) * 9 + wk]);
      sm.wt[buf][wcc][wk][wc] = v;
    }
  };
  // STAGES - 1 stages ahead; a stage past the last channel is an empty group
#pragma unroll
  for (int q = 0; q < STAGES - 1; ++q)
    if (q * KC < in.cin) stage(q * KC, q);
    else copy_commit();
  for (int c0 = 0, buf = 0; c0 < in.cin; c0 += KC, buf = buf + 1 < STAGES ? buf + 1 : 0) {
    copy_wait<STAGES - 2>();
    __syncthreads();  // this stage is there, and the one that is filled next has been read
    const int ahead = c0 + (STAGES - 1) * KC;
    if (ahead < in.cin) stage(ahead, buf > 0 ? buf - 1 : STAGES - 1);
    else copy_commit();
    auto channel = [&](int cc) {
      f32x2 v[PY + 2][PX + 2];  // each value twice
#pragma unroll
      for (int r = 0; r < PY + 2; ++r) {
        const float* s = &sm.tile[buf][cc][ty * PY + r][tx * PX];
        const float4 a = *reinterpret_cast<const float4*>(s);
        const float2 e = *reinterpret_cast<const float2*>(s + 4);
        v[r][0] = pack2(a.x, a.x); v[r][1] = pack2(a.y, a.y); v[r][2] = pack2(a.z, a.z);
        v[r][3] = pack2(a.w, a.w); v[r][4] = pack2(e.x, e.x); v[r][5] = pack2(e.y, e.y);
      }
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        f32x2 wr[CO / 2];
#pragma unroll
        for (int c = 0; c < CO / 2; c += 2)
          *reinterpret_cast<ulonglong2*>(wr + c) = *reinterpret_cast<const ulonglong2*>(&sm.wt[buf][cc][k][2 * c]);
#pragma unroll
        for (int r = 0; r < PY; ++r)
#pragma unroll
          for (int q = 0; q < PX; ++q)
#pragma unroll
            for (int c = 0; c < CO / 2; ++c) acc[r][q][c] = fma2(wr[c], v[r + k / 3][q + k % 3], acc[r][q][c]);
      }
    };
    if (busy) {
      channel(0);
      if (c0 + 1 < in.cin) channel(1);
    }
    static_assert(KC == 2, "two channels a stage");
  }
  const int x = x0 + tx * PX, y = y0 + ty * PY;
  if (x >= W || y >= H) return;
  auto val = [&](int r, int q, int c) {
    const float2 t = unpack2(acc[r][q][c / 2]);
    return c & 1 ? t.y : t.x;
  };
  const size_t plane = (size_t)H * W;
  // rows start on 16 bytes and the four pixels are inside (o.out may be the caller's)
  const bool vec = W % PX == 0 && (reinterpret_cast<uintptr_t>(o.out) & 15) == 0;
  auto store4 = [&](float* d, const float (&f)[PX], int n) {
    if (vec) *reinterpret_cast<float4*>(d) = make_float4(f[0], f[1], f[2], f[3]);
    else
#pragma unroll
      for (int q = 0; q < PX; ++q)
        if (q < n) d[q] = f[q];
  };
  auto load4 = [&](const float* d, float (&f)[PX], int n) {
    if (vec) {
      const float4 a = *reinterpret_cast<const float4*>(d);
      f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    } else {
#pragma unroll
      for (int q = 0; q < PX; ++q) f[q] = q < n ? d[q] : 0.f;
    }
  };
  const int nx = min(PX, W - x);
#pragma unroll
  for (int c = 0; c < CO; ++c) {
    const int co = co0 + c;
    if (co >= cout) break;
    if (EPI == EPI_POOL) {
      // double-resolution rows of 2 W: the pixels under (y + r, x + q)
#pragma unroll
      for (int r = 0; r < PY; ++r) {
        if (y + r >= H) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const size_t at = (((size_t)b * cout + co) * 2 * H + 2 * (y + r) + h) * 2 * W + 2 * x;
#pragma unroll
          for (int q = 0; q < PX; ++q) {
            if (q >= nx) break;
            const float g = 0.25f * val(r, q, c);
            float2* d = reinterpret_cast<float2*>(o.out + at + 2 * q);
            const float2 a = *reinterpret_cast<const float2*>(o.act + at + 2 * q), p = *d;
            *d = make_float2(a.x > 0.f ? p.x + g : 0.f, a.y > 0.f ? p.y + g : 0.f);
          }
        }
      }
      continue;
    }
    if (EPI == EPI_CAT && co < o.cu) {
      if (y + 1 < H) {  // H and W are even on the levels that have a skip
        const size_t at = (((size_t)b * o.cu + co) * (H / 2) + y / 2) * (W / 2) + x / 2;
#pragma unroll
        for (int q = 0; q < PX / 2; ++q) {
          if (2 * q >= nx) break;
          const float g = val(0, 2 * q, c) + val(0, 2 * q + 1, c) + val(1, 2 * q, c) + val(1, 2 * q + 1, c);
          o.out2[at + q] = o.act[at + q] > 0.f ? g : 0.f;
        }
      }
      continue;
    }
    float f[PY][PX];
#pragma unroll
    for (int r = 0; r < PY; ++r)
#pragma unroll
      for (int q = 0; q < PX; ++q) {
        f[r][q] = val(r, q, c);
        if (EPI == EPI_FWD && o.relu && f[r][q] < 0.f) f[r][q] = 0.f;
      }
    const size_t ch = EPI == EPI_CAT ? (size_t)b * (cout - o.cu) + co - o.cu : (size_t)b * cout + co;
#pragma unroll
    for (int r = 0; r < PY; ++r) {
      if (y + r >= H) break;
      const size_t at = ch * plane + (size_t)(y + r) * W + x;
      if (EPI == EPI_MASK) {
        float a[PX];
        load4(o.act + at, a, nx);
#pragma unroll
        for (int q = 0; q < PX; ++q)
          if (!(a[q] > 0.f)) f[r][q] = 0.f;
      }
      store4(o.out + at, f[r], nx);
    }
    if (EPI == EPI_FWD && o.out2 && y + 1 < H) {
      const size_t at = (((size_t)b * cout + co) * (H / 2) + y / 2) * (W / 2) + x / 2;
#pragma unroll
      for (int q = 0; q < PX / 2; ++q)
        if (2 * q < nx) o.out2[at + q] = 0.25f * (f[0][2 * q] + f[0][2 * q + 1] + f[1][2 * q] + f[1][2 * q + 1]);
    }
  }
}

// Weight and bias gradients: dW[co][ci][k] += sum_b,p dz[b][co](p) in[b][ci](p + d_k), db[co] += sum dz.
// A block takes 8 output x up to 8 input channels and every gridDim.y-th tile of 512 pixels (BW wide),
// staged one tile ahead; a warp takes one input channel (with fewer than 8 the warps share the rows),
// a lane 4 neighbouring pixels x RL rows: 288 multiply-adds for 8 + 6 wide loads a row.  Each lane adds
// its products in row order; the warp's sums go to its slot of `part` (cout cin 9 weights,
// then cout biases a slot) and k_wgrad_fold adds the slots in FP64 in order: no atomics, so two runs
// agree bit for bit, and the sums are at least as near the exact ones as the old ones were.
constexpr int RL = 4, CI = 8;
template <int BW>
struct WgradTile {
  static constexpr int LX = BW / PX, BH = 32 / LX * RL, PITCH = BW + 4;
  float g[2][CO / 2][BH][BW][2];  // output channels in pairs, as the products take them
  float in[2][CI][BH + 2][PITCH];
};
template <int BW>
__global__ void __launch_bounds__(NT, 2) k_conv3_wgrad(int B, int H, int W, int cout, ConvIn in, const float* __restrict__ dz,
                                                       float* __restrict__ part, int bias) {
  using T = WgradTile<BW>;
  constexpr int LX = T::LX, BH = T::BH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T& sm = *reinterpret_cast<T*>(smem_raw);
  const int nco = (cout + CO - 1) / CO, co0 = (blockIdx.x % nco) * CO, ci0 = (blockIdx.x / nco) * CI;
  const int nci = min(CI, in.cin - ci0), nog = min(CO, cout - co0), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int share = CI / min(CI, in.cin);  // warps a channel: the same for every group of the layer
  const int wc = warp / share, sub = warp % share;
  const bool work = wc < nci;
  const int lx = lane % LX, ly = lane / LX;
  f32x2 tot[CO / 2][9], btot[CO / 2];  // two output channels a word
#pragma unroll
  for (int c = 0; c < CO / 2; ++c) {
    btot[c] = 0;
#pragma unroll
    for (int k = 0; k < 9; ++k) tot[c][k] = 0;
  }
  const bool do_bias = bias && ci0 == 0 && wc == 0;
  const int nxt = (W + BW - 1) / BW, nyt = (H + BH - 1) / BH, ntile = B * nxt * nyt;
  const ConvIn gin{dz, nullptr, cout, 0};
  auto stage = [&](int tl, int buf) {
    const int b = tl / (nxt * nyt), r0 = tl - b * nxt * nyt, y0 = r0 / nxt * BH, x0 = r0 % nxt * BW;
    stage_rows<BH, BW, BW, 0, true>(&sm.g[buf][0][0][0][0], gin, b, co0, CO, H, W, y0, x0);  // zero past cout
    stage_rows<BH + 2, BW + 2, T::PITCH, 1>(&sm.in[buf][0][0][0], in, b, ci0, nci, H, W, y0, x0);
    copy_commit();
  };
  if ((int)blockIdx.y < ntile) stage(blockIdx.y, 0);
  for (int tl = blockIdx.y, buf = 0; tl < ntile; tl += gridDim.y, buf ^= 1) {
    if (tl + (int)gridDim.y < ntile) {
      stage(tl + gridDim.y, buf ^ 1);
      copy_wait<1>();
    } else {
      copy_wait<0>();
    }
    __syncthreads();
    if (work) {
      const int below = H - (tl % (nxt * nyt)) / nxt * BH;  // rows of this tile inside the grid
      auto row = [&](int i) {
        const int yy = ly * RL + i;
        if (yy >= below) return;  // rows past the grid are not staged
        f32x2 v[3][PX + 2];  // each value twice
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const float* s = &sm.in[buf][wc][yy + r][lx * PX];
          const float4 a = *reinterpret_cast<const float4*>(s);
          const float2 e = *reinterpret_cast<const float2*>(s + 4);
          v[r][0] = pack2(a.x, a.x); v[r][1] = pack2(a.y, a.y); v[r][2] = pack2(a.z, a.z);
          v[r][3] = pack2(a.w, a.w); v[r][4] = pack2(e.x, e.x); v[r][5] = pack2(e.y, e.y);
        }
#pragma unroll
        for (int c = 0; c < CO / 2; ++c) {
          f32x2 g[PX];
#pragma unroll
          for (int q = 0; q < PX; q += 2)
            *reinterpret_cast<ulonglong2*>(g + q) = *reinterpret_cast<const ulonglong2*>(&sm.g[buf][c][yy][lx * PX + q][0]);
          if (do_bias) btot[c] = add2(btot[c], add2(add2(g[0], g[1]), add2(g[2], g[3])));
          // pixel by pixel: nine independent sums between two additions to the same one
#pragma unroll
          for (int q = 0; q < PX; ++q)
#pragma unroll
            for (int k = 0; k < 9; ++k) tot[c][k] = fma2(g[q], v[k / 3][k % 3 + q], tot[c][k]);
        }
      };
      if (share == 1) {
#pragma unroll
        for (int i = 0; i < RL; ++i) row(i);
      } else {
        for (int i = sub; i < RL; i += share) row(i);
      }
    }
    __syncthreads();
  }
  if (!work) return;
  float* o = part + (size_t)(blockIdx.y * share + sub) * ((size_t)cout * in.cin * 9 + cout);
#pragma unroll
  for (int c = 0; c < CO; ++c) {
    if (c >= nog) break;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const float2 t2 = unpack2(tot[c / 2][k]);
      float v = c & 1 ? t2.y : t2.x;
      for (int q = 16; q > 0; q >>= 1) v += __shfl_xor_sync(0xffffffffu, v, q);
      if (lane == 0) o[((size_t)(co0 + c) * in.cin + ci0 + wc) * 9 + k] = v;
    }
    if (do_bias) {
      const float2 t2 = unpack2(btot[c / 2]);
      float v = c & 1 ? t2.y : t2.x;
      for (int q = 16; q > 0; q >>= 1) v += __shfl_xor_sync(0xffffffffu, v, q);
      if (lane == 0) o[(size_t)cout * in.cin * 9 + co0 + c] = v;
    }
  }
}
__global__ void k_wgrad_fold(const float* __restrict__ part, int slots, int nw, int nb, float* __restrict__ dw,
                             float* __restrict__ db) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nw + (db ? nb : 0)) return;
  double s = 0.0;
#pragma unroll 8
  for (int q = 0; q < slots; ++q) s += (double)part[(size_t)q * (nw + nb) + t];
  float& d = t < nw ? dw[t] : db[t - nw];
  d = (float)((double)d + s);
}

// The tile width (threads or lanes along x) that covers W with the least padding, wider at a tie.
int tile_width(int W, int w0, int w1, int w2) {
  const int c[3] = {w0, w1, w2};
  int best = w0, pad = (W + w0 - 1) / w0 * w0;
  for (int k = 1; k < 3; ++k) {
    const int p = (W + c[k] - 1) / c[k] * c[k];
    if (p < pad) { pad = p; best = c[k]; }
  }
  return best;
}

template <bool TRANSPOSED, int EPI, int TX, int CB>
void run_conv3(dim3 grid, int H, int W, int cout, const ConvIn& in, const __nv_bfloat16* w, const float* bias, const ConvOut& o,
               cudaStream_t st) {
  k_conv3<TRANSPOSED, EPI, TX, CB><<<grid, NT, sizeof(ConvTile<TX, CB>), st>>>(H, W, cout, in, w, bias, o);
}
template <bool TRANSPOSED, int EPI>
void launch_conv3(int B, int H, int W, int cout, const ConvIn& in, const __nv_bfloat16* w, const float* bias, const ConvOut& o,
                  cudaStream_t st) {
  const int tw = tile_width(W, 32 * PX, 16 * PX, 8 * PX), th = NT / (tw / PX) * PY;
  dim3 grid((W + tw - 1) / tw, (H + th - 1) / th, B * ((cout + 7) / 8));
  const bool half = (long long)grid.x * grid.y * grid.z < 152 && cout > 4;
  if (half) grid.z = B * ((cout + 3) / 4);
  auto* run = tw == 32 * PX   ? (half ? run_conv3<TRANSPOSED, EPI, 32, 4> : run_conv3<TRANSPOSED, EPI, 32, 8>)
              : tw == 16 * PX ? (half ? run_conv3<TRANSPOSED, EPI, 16, 4> : run_conv3<TRANSPOSED, EPI, 16, 8>)
                              : (half ? run_conv3<TRANSPOSED, EPI, 8, 4> : run_conv3<TRANSPOSED, EPI, 8, 8>);
  gmk::kernel_launch_adjust(1);
  run(grid, H, W, cout, in, w, bias, o, st);
}

// slices of the tile range a weight gradient is split over, and the slots its partial sums take
struct WgradPlan {
  int bw, groups, slices, slots;
  size_t floats;
};
WgradPlan wgrad_plan(int B, int H, int W, int cin, int cout) {
  WgradPlan p;
  p.bw = tile_width(W, 128, 64, 32);
  const int bh = 512 / p.bw;
  p.groups = ((cout + CO - 1) / CO) * ((cin + CI - 1) / CI);
  const long long tiles = (long long)B * ((W + p.bw - 1) / p.bw) * ((H + bh - 1) / bh);
  p.slices = (int)std::max<long long>(1, std::min<long long>(tiles, 304 / p.groups));  // two blocks an SM
  p.slots = p.slices * (CI / std::min(CI, cin));
  p.floats = (size_t)p.slots * ((size_t)cout * cin * 9 + cout);
  return p;
}
template <int BW>
void run_wgrad(const WgradPlan& p, int B, int H, int W, int cout, const ConvIn& in, const float* dz, float* part, int bias,
               cudaStream_t st) {
  k_conv3_wgrad<BW><<<dim3(p.groups, p.slices), NT, sizeof(WgradTile<BW>), st>>>(B, H, W, cout, in, dz, part, bias);
}
void launch_wgrad(int B, int H, int W, int cout, const ConvIn& in, const float* dz, float* dw, float* db, float* part,
                  cudaStream_t st) {
  const WgradPlan p = wgrad_plan(B, H, W, in.cin, cout);
  const int nw = cout * in.cin * 9, bias = db ? 1 : 0;
  gmk::kernel_launch_adjust(2);
  if (p.bw == 128) run_wgrad<128>(p, B, H, W, cout, in, dz, part, bias, st);
  else if (p.bw == 64) run_wgrad<64>(p, B, H, W, cout, in, dz, part, bias, st);
  else run_wgrad<32>(p, B, H, W, cout, in, dz, part, bias, st);
  k_wgrad_fold<<<(nw + cout + 127) / 128, 128, 0, st>>>(part, p.slots, nw, cout, dw, db);
}

// The kernels' dynamic shared memory on the current device (set when a workspace is made).
template <typename K>
void allow_smem(K kernel, size_t bytes) {
  UN_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}
template <bool TRANSPOSED, int EPI>
void allow_conv3() {
  allow_smem(k_conv3<TRANSPOSED, EPI, 32, 8>, sizeof(ConvTile<32, 8>));
  allow_smem(k_conv3<TRANSPOSED, EPI, 16, 8>, sizeof(ConvTile<16, 8>));
  allow_smem(k_conv3<TRANSPOSED, EPI, 8, 8>, sizeof(ConvTile<8, 8>));
  allow_smem(k_conv3<TRANSPOSED, EPI, 32, 4>, sizeof(ConvTile<32, 4>));
  allow_smem(k_conv3<TRANSPOSED, EPI, 16, 4>, sizeof(ConvTile<16, 4>));
  allow_smem(k_conv3<TRANSPOSED, EPI, 8, 4>, sizeof(ConvTile<8, 4>));
}
void allow_kernels() {
  allow_conv3<false, EPI_FWD>();
  allow_conv3<true, EPI_MASK>();
  allow_conv3<true, EPI_CAT>();
  allow_conv3<true, EPI_POOL>();
  allow_smem(k_conv3_wgrad<128>, sizeof(WgradTile<128>));
  allow_smem(k_conv3_wgrad<64>, sizeof(WgradTile<64>));
  allow_smem(k_conv3_wgrad<32>, sizeof(WgradTile<32>));
}

}  // namespace

struct gm_unet {
  int B = 0, H = 0, W = 0;
  // activations per layer output and the per-layer inputs that are not another layer's output
  float* act[NL] = {};     // outputs of the twelve convolutions
  float* pooled[3] = {};   // pool(e0), pool(e1), pool(e2)
  float* x = nullptr;      // network input (2 channels)
  float* part = nullptr;   // partial sums of one layer's weight gradient (wgrad_plan)
  float* g_act[NL] = {};   // gradients of the layer outputs before their ReLU (not of the last)
  std::vector<void*> allocs;
  std::string err;
  ~gm_unet() {
    for (void* p : allocs) cudaFree(p);
  }
  float* alloc(size_t n) {
    void* p = nullptr;
    UN_CK(cudaMalloc(&p, n * sizeof(float)));
    allocs.push_back(p);
    return (float*)p;
  }
  size_t plane(int level) const { return (size_t)(H >> level) * (W >> level); }
};

namespace {

// the encoder output that decoder layer k = 8, 9, 10 takes beside the layer before it
constexpr int skip_of(int k) { return 5 - 2 * (k - 8); }

// input tensor of layer k
ConvIn layer_input(const gm_unet* u, int k) {
  if (k == 0) return {u->x, nullptr, LAYERS[0].cin, 0};
  if (k == 2 || k == 4 || k == 6) return {u->pooled[k / 2 - 1], nullptr, LAYERS[k].cin, 0};
  if (k >= 8 && k <= 10) return {u->act[skip_of(k)], u->act[k - 1], LAYERS[k].cin, LAYERS[k - 1].cout};
  return {u->act[k - 1], nullptr, LAYERS[k].cin, 0};
}

void forward(gm_unet* u, const __nv_bfloat16* const* w, const float* const* b, float* y, cudaStream_t st) {
  for (int k = 0; k < NL; ++k) {
    const LayerDef& L = LAYERS[k];
    const bool pool = k == 1 || k == 3 || k == 5;
    const ConvOut o{k == NL - 1 && y ? y : u->act[k], pool ? u->pooled[k / 2] : nullptr, nullptr, 0, L.relu ? 1 : 0};
    launch_conv3<false, EPI_FWD>(u->B, u->H >> L.level, u->W >> L.level, L.cout, layer_input(u, k), w[k], b[k], o, st);
  }
}

// dw and db accumulate (zeroed by the caller).  g_act[k] is the gradient in front of layer k's ReLU
// when its own turn comes: the layers run from the last to the first, a decoder layer leaves its
// skip's part in the encoder output's gradient, and the convolution behind that output's pooling
// (layer 6, 4 or 2, always later) adds its part and the mask.
void backward(gm_unet* u, const __nv_bfloat16* const* w, const float* dy, float* const* dw, float* const* db, cudaStream_t st) {
  for (int k = NL - 1; k >= 0; --k) {
    const LayerDef& L = LAYERS[k];
    const int H = u->H >> L.level, W = u->W >> L.level;
    const float* g = k == NL - 1 ? dy : u->g_act[k];
    launch_wgrad(u->B, H, W, L.cout, layer_input(u, k), g, dw[k], db[k], u->part, st);
    if (k == 0) break;
    const ConvIn gin{g, nullptr, L.cout, 0};
    if (k >= 8 && k <= 10) {
      const ConvOut o{u->g_act[skip_of(k)], u->g_act[k - 1], u->act[k - 1], LAYERS[k - 1].cout, 0};
      launch_conv3<true, EPI_CAT>(u->B, H, W, L.cin, gin, w[k], nullptr, o, st);
    } else if (k == 2 || k == 4 || k == 6) {
      const ConvOut o{u->g_act[k - 1], nullptr, u->act[k - 1], 0, 0};
      launch_conv3<true, EPI_POOL>(u->B, H, W, L.cin, gin, w[k], nullptr, o, st);
    } else {
      const ConvOut o{u->g_act[k - 1], nullptr, u->act[k - 1], 0, 0};
      launch_conv3<true, EPI_MASK>(u->B, H, W, L.cin, gin, w[k], nullptr, o, st);
    }
  }
}

std::string g_unet_error;

}  // namespace

extern "C" {

int gm_unet_layers(int32_t* n_layers, int32_t* cin, int32_t* cout) {
  if (n_layers) *n_layers = NL;
  for (int k = 0; k < NL; ++k) {
    if (cin) cin[k] = LAYERS[k].cin;
    if (cout) cout[k] = LAYERS[k].cout;
  }
  return GM_OK;
}

int gm_unet_create(int32_t batch, int32_t height, int32_t width, gm_unet** out) {
  if (!out) return GM_EVALUE;
  *out = nullptr;
  if (batch < 1 || height < 8 || width < 8 || height % 8 || width % 8) {
    g_unet_error = "the network needs batch >= 1 and a grid whose sides are multiples of 8";
    return GM_EVALUE;
  }
  auto u = std::make_unique<gm_unet>();
  u->B = batch;
  u->H = height;
  u->W = width;
  try {
    allow_kernels();
    u->x = u->alloc((size_t)batch * 2 * u->plane(0));
    for (int k = 0; k < NL; ++k) {
      const size_t n = (size_t)batch * LAYERS[k].cout * u->plane(LAYERS[k].level);
      u->act[k] = u->alloc(n);
      if (k < NL - 1) u->g_act[k] = u->alloc(n);
    }
    for (int p = 0; p < 3; ++p) {
      const size_t n = (size_t)batch * LAYERS[2 * p + 1].cout * u->plane(p + 1);
      u->pooled[p] = u->alloc(n);
    }
    size_t np = 0;
    for (const LayerDef& L : LAYERS)
      np = std::max(np, wgrad_plan(batch, height >> L.level, width >> L.level, L.cin, L.cout).floats);
    u->part = u->alloc(np);
  } catch (const std::exception& e) {
    g_unet_error = e.what();
    return GM_ECUDA;
  }
  *out = u.release();
  return GM_OK;
}

int gm_unet_destroy(gm_unet* u) {
  delete u;
  return GM_OK;
}

const char* gm_unet_last_error(const gm_unet* u) { return u ? u->err.c_str() : g_unet_error.c_str(); }

int gm_unet_input(gm_unet* u, float** x) {
  if (!u || !x) return GM_EVALUE;
  *x = u->x;
  return GM_OK;
}

int gm_unet_forward(gm_unet* u, const uint16_t* const* w_bf16, const float* const* bias, const float* x, float* y,
                    void* stream) {
  if (!u || !w_bf16 || !bias) return GM_EVALUE;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    if (x && x != u->x) UN_CK(cudaMemcpyAsync(u->x, x, (size_t)u->B * 2 * u->plane(0) * 4, cudaMemcpyDeviceToDevice, st));
    forward(u, reinterpret_cast<const __nv_bfloat16* const*>(w_bf16), bias, y, st);
    UN_CK(cudaGetLastError());
  } catch (const std::exception& e) {
    u->err = e.what();
    return GM_ECUDA;
  }
  return GM_OK;
}

int gm_unet_backward(gm_unet* u, const uint16_t* const* w_bf16, const float* dy, float* const* dw, float* const* db,
                     void* stream) {
  if (!u || !w_bf16 || !dy || !dw || !db) return GM_EVALUE;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    backward(u, reinterpret_cast<const __nv_bfloat16* const*>(w_bf16), dy, dw, db, st);
    UN_CK(cudaGetLastError());
  } catch (const std::exception& e) {
    u->err = e.what();
    return GM_ECUDA;
  }
  return GM_OK;
}

}  // extern "C"
