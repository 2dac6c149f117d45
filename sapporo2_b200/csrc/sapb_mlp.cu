// Neighbour-radius network: a 5 -> 64 -> 64 -> 64 -> 1 perceptron with ReLU
// hidden layers, FP32 weights, trained on the GPU with hand-written forward,
// backward and Adam kernels.  It proposes log(h2) for each i-particle from
// five features of its previous evaluation; the host side (Python) builds
// features and targets from the neighbour counts the force kernel reports.
// Declared in include/sapporo_b200.h (sapb_mlp_*).
//
// Parameter layout (floats): W1[64][5] b1[64] W2[64][64] b2[64] W3[64][64]
// b3[64] W4[64] b4[1]  -- 8769 parameters.
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <vector>

#include "../../include/sapporo_b200.h"
#include "sapb_dev.h"

namespace {

constexpr int kIn = 5, kH = 64;
constexpr int oW1 = 0, oB1 = oW1 + kH * kIn, oW2 = oB1 + kH, oB2 = oW2 + kH * kH,
              oW3 = oB2 + kH, oB3 = oW3 + kH * kH, oW4 = oB3 + kH, oB4 = oW4 + kH,
              kNP = oB4 + 1;

// One block = 128 threads on a chunk of 64 samples.  Activations and deltas
// sit in shared memory as [sample][unit] rows of kS floats (16-byte aligned,
// 4 banks apart, so 8 consecutive rows of a 16-byte load touch every bank
// once); the 64 x 64 weights as [out][in] rows of the same length.
//
// Every 64 x 64 x 64 product of the network (two forward, two backward, two
// weight gradients per chunk) is an 8 x 4 tile per thread, read as float4
// along the rows of both operands and done in packed FP32 pairs: 12 vector
// loads per 64 packed FMAs.  A warp's 16-byte load takes two cycles of the
// SM's shared-memory pipe when every aligned group of four lanes reads at
// most two addresses, four otherwise (measured over 20 address patterns), so
// a product needs 96 cycles there against 128 on the FMA pipes; a 4 x 4 tile
// needs 128 against 128.  An epoch of 65536 samples, Adam step included, on
// B200: one sample per thread, scalar weight loads, 4 warps per SM 216 us
// (FMA pipe 21 % busy); 4 x 4 tiles with four-cycle loads 121 us; as here
// 103 us (55 %), and 24.6 us against 68 at 256 to 2048 samples, where one
// chunk's serial chain of layers is the bound.  All sums stay FP32.
constexpr int kT = 128;  // threads per block
constexpr int kM = 64;   // samples per chunk
constexpr int kS = 68;   // row length in floats

// thread -> tile: sample rows sg + 8 i, units ug + 16 j or 4 ug + j.  Lane
// bits 0, 2, 3 are sg and 1, 4 ug: four adjacent lanes share two rows of
// either operand.
struct Lane {
  int sg, ug;
};
__device__ __forceinline__ Lane lane_of(int t) {
  return Lane{(t & 1) | ((t >> 1) & 6), ((t >> 1) & 1) | ((t >> 3) & 2) | ((t >> 5) << 2)};
}

__device__ __forceinline__ float4 ld4(const float *p) {
  return *reinterpret_cast<const float4 *>(p);
}
__device__ __forceinline__ float2 lo2(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 &v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
// sum over the lanes that hold the other sample rows / the other units of a warp
__device__ __forceinline__ float sum_sg(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  return v + __shfl_xor_sync(0xffffffffu, v, 8);
}
__device__ __forceinline__ float sum_ug(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v + __shfl_xor_sync(0xffffffffu, v, 16);
}

struct Weights {  // shared memory
  float W2[kH * kS], W3[kH * kS];
  float W1[kH * kIn], b1[kH], b2[kH], b3[kH], W4[kH];
  float b4, pad[3];
};

__device__ __forceinline__ void load_weights(Weights &w, const float *__restrict__ P, int t) {
  for (int k = t; k < kH * kH / 4; k += kT) {
    const int o = k >> 4, c = (k & 15) * 4;
    *reinterpret_cast<float4 *>(w.W2 + o * kS + c) = ld4(P + oW2 + 4 * k);
    *reinterpret_cast<float4 *>(w.W3 + o * kS + c) = ld4(P + oW3 + 4 * k);
  }
  for (int k = t; k < kH * kIn; k += kT) w.W1[k] = P[oW1 + k];
  if (t < kH) {
    w.b1[t] = P[oB1 + t];
    w.b2[t] = P[oB2 + t];
    w.b3[t] = P[oB3 + t];
    w.W4[t] = P[oW4 + t];
  }
  if (t == 0) w.b4 = P[oB4];
}

// relu(b1 + W1 x) for samples sg + 8 i, units ug + 16 j; xs: [sample][8].
__device__ __forceinline__ void layer1(const Weights &w, const float *xs, Lane L, float *out) {
  float wk[4][kIn];
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int k = 0; k < kIn; k++) wk[j][k] = w.W1[(L.ug + 16 * j) * kIn + k];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int s = L.sg + 8 * i;
    const float4 x4 = ld4(xs + s * 8);
    const float x[kIn] = {x4.x, x4.y, x4.z, x4.w, xs[s * 8 + 4]};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float v = w.b1[L.ug + 16 * j];
#pragma unroll
      for (int k = 0; k < kIn; k++) v = fmaf(wk[j][k], x[k], v);
      out[s * kS + L.ug + 16 * j] = fmaxf(v, 0.f);
    }
  }
}

// h[i][j] = relu(b + W a) for samples sg + 8 i, units ug + 16 j.
__device__ __forceinline__ void dense(const float *W, const float *b, const float *a, Lane L,
                                      float h[8][4]) {
  float2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = make_float2(b[L.ug + 16 * j], 0.f);
#pragma unroll 2
  for (int k = 0; k < kH; k += 4) {
    float4 wv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) wv[j] = ld4(W + (L.ug + 16 * j) * kS + k);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float4 av = ld4(a + (L.sg + 8 * i) * kS + k);
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] = __ffma2_rn(lo2(av), lo2(wv[j]), acc[i][j]);
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] = __ffma2_rn(hi2(av), hi2(wv[j]), acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) h[i][j] = fmaxf(acc[i][j].x + acc[i][j].y, 0.f);
}

__device__ __forceinline__ void store_units(float *out, Lane L, const float h[8][4]) {
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) out[(L.sg + 8 * i) * kS + L.ug + 16 * j] = h[i][j];
}

// Sum over the units of W4 h3 for this thread's eight samples into yp[4][kM]
// (one row per warp, i.e. per four unit groups); the caller sums the rows
// after a barrier.
__device__ __forceinline__ void layer4(const Weights &w, const float h[8][4], Lane L, int t,
                                       float *yp) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 4; j++) s = fmaf(w.W4[L.ug + 16 * j], h[i][j], s);
    s = sum_ug(s);
    if ((t & 18) == 0) yp[(t >> 5) * kM + L.sg + 8 * i] = s;
  }
}
__device__ __forceinline__ float output_of(const Weights &w, const float *yp, int s) {
  return w.b4 + ((yp[s] + yp[kM + s]) + (yp[2 * kM + s] + yp[3 * kM + s]));
}

// Proposal: the five features of each particle from its raw previous state
// (n_prev, h2_prev, a[3], jerk[3], L; features: log rho with the density
// estimate rho = n / (4/3 pi h^3), n = max(n_prev, 1/2), log |a|, log |jerk|,
// L - log rho with L the particle's running mean of log rho over its past
// evaluations, log h2_prev), standardised with (mu, sd), the network's correction
// clipped to [-max_down, max_up] and added to the count-scaled step
// 2/3 log(target/n); out: h2_prev * exp(clip(step, -clip, clip)).
struct MlpScale {
  float mu[kIn], sd[kIn];
  float target, max_down, max_up, clip;
};
constexpr int kPropIn = 9;

struct EvalSmem {
  Weights w;
  float A1[kM * kS], A2[kM * kS], xs[kM * 8], yp[4 * kM];
};

// y of each sample (PROPOSE: the proposed h2), one chunk of 64 per block.
template <bool PROPOSE>
__global__ void __launch_bounds__(kT) mlp_eval_kernel(const float *__restrict__ P, int n,
                                                      const float *__restrict__ IN, MlpScale sc,
                                                      float *__restrict__ OUT) {
  extern __shared__ __align__(16) unsigned char smem[];
  EvalSmem &S = *reinterpret_cast<EvalSmem *>(smem);
  const int t = threadIdx.x;
  const Lane L = lane_of(t);
  const int i = blockIdx.x * kM + t;  // threads 0..63: this thread's sample
  const bool mine = t < kM && i < n;
  load_weights(S.w, P, t);
  float np = 1.f, h2 = 1.f;
  if (t < kM) {
    float x[kIn] = {0, 0, 0, 0, 0};
    if (mine && PROPOSE) {
      const float *r = IN + (size_t)i * kPropIn;
      np = fmaxf(r[0], 0.5f);
      h2 = r[1];
      const float an = sqrtf(r[2] * r[2] + r[3] * r[3] + r[4] * r[4]) + 1e-30f;
      const float jn = sqrtf(r[5] * r[5] + r[6] * r[6] + r[7] * r[7]) + 1e-30f;
      const float lh2 = logf(h2);
      const float lrho = logf(np) - logf(4.18879020f) - 1.5f * lh2;
      const float f[kIn] = {lrho, logf(an), logf(jn), r[8] - lrho, lh2};
#pragma unroll
      for (int k = 0; k < kIn; k++) x[k] = (f[k] - sc.mu[k]) / sc.sd[k];
    } else if (mine) {
#pragma unroll
      for (int k = 0; k < kIn; k++) x[k] = IN[(size_t)i * kIn + k];
    }
#pragma unroll
    for (int k = 0; k < kIn; k++) S.xs[t * 8 + k] = x[k];
  }
  __syncthreads();
  layer1(S.w, S.xs, L, S.A1);
  __syncthreads();
  float h[8][4];
  dense(S.w.W2, S.w.b2, S.A1, L, h);
  store_units(S.A2, L, h);
  __syncthreads();
  dense(S.w.W3, S.w.b3, S.A2, L, h);
  layer4(S.w, h, L, t, S.yp);
  __syncthreads();
  if (!mine) return;
  const float y = output_of(S.w, S.yp, t);
  if (PROPOSE) {
    const float corr = fminf(fmaxf(y, -sc.max_down), sc.max_up);
    const float step = (2.f / 3.f) * logf(sc.target / np) + corr;
    OUT[i] = h2 * expf(fminf(fmaxf(step, -sc.clip), sc.clip));
  } else {
    OUT[i] = y;
  }
}

// Gradient of L = 1/(2n) sum (y - t)^2: each block loops over chunks of 64
// samples, keeps its share of every gradient in registers and writes it (and
// its share of the loss, entry kNP) to its own row of `part`; the rows are
// summed by mlp_update_kernel in a fixed order, so training is bit-stable and
// needs neither atomics nor cleared sums.  110 KB of shared memory and at most
// 255 registers per thread: two blocks per SM, one computing while the other
// waits at a barrier (six per chunk).
constexpr int kRow = (kNP + 1 + 3) / 4 * 4;  // floats per row of `part`
struct BackSmem {
  Weights w;
  float A1[kM * kS], A2[kM * kS], D2[kM * kS], D3[kM * kS];  // D3: delta 3, then delta 1
  float xs[kM * 8], yp[4 * kM], tg[kM];
};

// acc[r][*] += sum over the chunk's samples of d[sample][o_r] a[sample][4 kg + *],
// o_r = 4 og + r for r < 4, 32 + 4 og + r - 4 above
__device__ __forceinline__ void weight_grad(const float *d, const float *a, int og, int kg,
                                            float2 acc[8][2]) {
#pragma unroll 4
  for (int s = 0; s < kM; s++) {
    const float4 d0 = ld4(d + s * kS + 4 * og), d1 = ld4(d + s * kS + 32 + 4 * og);
    const float4 av = ld4(a + s * kS + 4 * kg);
    const float dr[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
#pragma unroll
    for (int r = 0; r < 8; r++) {
      acc[r][0] = __ffma2_rn(both(dr[r]), lo2(av), acc[r][0]);
      acc[r][1] = __ffma2_rn(both(dr[r]), hi2(av), acc[r][1]);
    }
  }
}

// out = (W^T d)[4 ug ..] of samples sg + 8 i where act > 0, else 0; the sums
// over the eight samples are added to gb.
__device__ __forceinline__ void back(const float *W, const float *d, const float *act, Lane L,
                                     float *out, float gb[4]) {
  float2 acc[8][2];
#pragma unroll
  for (int i = 0; i < 8; i++) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
#pragma unroll 2
  for (int o = 0; o < kH; o += 4) {
    float4 wv[4];
#pragma unroll
    for (int r = 0; r < 4; r++) wv[r] = ld4(W + (o + r) * kS + 4 * L.ug);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float4 dv = ld4(d + (L.sg + 8 * i) * kS + o);
      const float dr[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
      for (int r = 0; r < 4; r++) {
        acc[i][0] = __ffma2_rn(both(dr[r]), lo2(wv[r]), acc[i][0]);
        acc[i][1] = __ffma2_rn(both(dr[r]), hi2(wv[r]), acc[i][1]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int at = (L.sg + 8 * i) * kS + 4 * L.ug;
    const float4 a = ld4(act + at);
    const float4 v = make_float4(a.x > 0.f ? acc[i][0].x : 0.f, a.y > 0.f ? acc[i][0].y : 0.f,
                                 a.z > 0.f ? acc[i][1].x : 0.f, a.w > 0.f ? acc[i][1].y : 0.f);
    *reinterpret_cast<float4 *>(out + at) = v;
    gb[0] += v.x; gb[1] += v.y; gb[2] += v.z; gb[3] += v.w;
  }
}

__global__ void __launch_bounds__(kT, 2) mlp_backward_kernel(const float *__restrict__ P, int n,
                                                             const float *__restrict__ X,
                                                             const float *__restrict__ T,
                                                             float *__restrict__ part) {
  extern __shared__ __align__(16) unsigned char smem[];
  BackSmem &S = *reinterpret_cast<BackSmem *>(smem);
  const int t = threadIdx.x;
  const Lane L = lane_of(t);
  // weight-gradient tiles: outputs 4 og .. and 32 + 4 og .., inputs 4 kg ..
  const int og = L.sg, kg = L.ug;
  float2 gW3[8][2], gW2[8][2];
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < 2; c++) gW3[r][c] = gW2[r][c] = make_float2(0.f, 0.f);
  float gW4[4] = {0, 0, 0, 0}, gB3[4] = {0, 0, 0, 0};  // units ug + 16 j
  float gB2[4] = {0, 0, 0, 0}, gB1[4] = {0, 0, 0, 0};  // units 4 ug + j
  float gW1[kIn] = {0, 0, 0, 0, 0};  // unit t % 64, samples 32 (t / 64) ..
  float gB4 = 0.f, lsum = 0.f;
  // a chunk's samples are fetched while the chunk before is computed
  float fx[3], ft;
  auto fetch = [&](int chunk) {
    const long left = (long)n - (long)chunk * kM;  // samples from this chunk on
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const int q = t + r * kT;
      fx[r] = q < kM * kIn && q < left * kIn ? X[(size_t)chunk * kM * kIn + q] : 0.f;
    }
    ft = t < kM && t < left ? T[(size_t)chunk * kM + t] : 0.f;
  };
  fetch(blockIdx.x);
  load_weights(S.w, P, t);

  const float inv_n = 1.f / (float)n;
  const int nchunks = (n + kM - 1) / kM;
  for (int chunk = blockIdx.x; chunk < nchunks; chunk += gridDim.x) {
    const int i0 = chunk * kM;
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const int q = t + r * kT;
      if (q < kM * kIn) S.xs[(q / kIn) * 8 + q % kIn] = fx[r];
    }
    if (t < kM) S.tg[t] = ft;
    fetch(chunk + gridDim.x);
    __syncthreads();
    layer1(S.w, S.xs, L, S.A1);
    __syncthreads();
    float h[8][4];
    dense(S.w.W2, S.w.b2, S.A1, L, h);
    store_units(S.A2, L, h);
    __syncthreads();
    dense(S.w.W3, S.w.b3, S.A2, L, h);
    layer4(S.w, h, L, t, S.yp);
    __syncthreads();
    // delta 3, and the gradients that need this thread's h3 only
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int s = L.sg + 8 * i;
      const float err = i0 + s < n ? output_of(S.w, S.yp, s) - S.tg[s] : 0.f;
      const float dy = err * inv_n;
      if (L.ug == 0) {
        lsum += 0.5f * err * dy;
        gB4 += dy;
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int o = L.ug + 16 * j;
        const float d = h[i][j] > 0.f ? dy * S.w.W4[o] : 0.f;
        S.D3[s * kS + o] = d;
        gB3[j] += d;
        gW4[j] = fmaf(dy, h[i][j], gW4[j]);
      }
    }
    __syncthreads();
    weight_grad(S.D3, S.A2, og, kg, gW3);
    back(S.w.W3, S.D3, S.A2, L, S.D2, gB2);
    __syncthreads();
    float *D1 = S.D3;  // delta 3 was last read before the barrier
    weight_grad(S.D2, S.A1, og, kg, gW2);
    back(S.w.W2, S.D2, S.A1, L, D1, gB1);
    __syncthreads();
#pragma unroll 4
    for (int s = 32 * (t >> 6); s < 32 * (t >> 6) + 32; s++) {
      const float d = D1[s * kS + (t & 63)];
      const float4 x4 = ld4(S.xs + s * 8);
      const float x[kIn] = {x4.x, x4.y, x4.z, x4.w, S.xs[s * 8 + 4]};
#pragma unroll
      for (int k = 0; k < kIn; k++) gW1[k] = fmaf(d, x[k], gW1[k]);
    }
    __syncthreads();  // the next chunk overwrites xs and the targets
  }

  // ---- this block's row ----
  float *row = part + (size_t)blockIdx.x * kRow;
#pragma unroll
  for (int r = 0; r < 8; r++) {
    const int at = (4 * og + r + (r < 4 ? 0 : 28)) * kH + 4 * kg;
    *reinterpret_cast<float4 *>(row + oW3 + at) =
        make_float4(gW3[r][0].x, gW3[r][0].y, gW3[r][1].x, gW3[r][1].y);
    *reinterpret_cast<float4 *>(row + oW2 + at) =
        make_float4(gW2[r][0].x, gW2[r][0].y, gW2[r][1].x, gW2[r][1].y);
  }
  // each unit group lies in one warp: sum over its lanes' sample rows
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float w4 = sum_sg(gW4[j]), b3 = sum_sg(gB3[j]);
    const float b2 = sum_sg(gB2[j]), b1 = sum_sg(gB1[j]);
    if (L.sg == 0) {
      row[oW4 + L.ug + 16 * j] = w4;
      row[oB3 + L.ug + 16 * j] = b3;
      row[oB2 + 4 * L.ug + j] = b2;
      row[oB1 + 4 * L.ug + j] = b1;
    }
  }
  lsum = sum_sg(lsum);  // ug == 0: lanes of warp 0
  gB4 = sum_sg(gB4);
  if (t == 0) {
    row[kNP] = lsum;
    row[oB4] = gB4;
  }
  float *red = S.A1;  // [2][64][5], free after the loop's last barrier
#pragma unroll
  for (int k = 0; k < kIn; k++) red[t * kIn + k] = gW1[k];
  __syncthreads();
  for (int q = t; q < kH * kIn; q += kT) row[oW1 + q] = red[q] + red[kH * kIn + q];
}

// Sums the blocks' rows (fixed order) and takes an Adam step (bias-corrected)
// or, with M == nullptr, writes the gradient to G.  32 parameters per block and
// 32 threads for each, striding over the rows: a full grid's 296 rows (10 MB,
// from L2) are ten loads per thread, all in flight together (with eight
// threads per parameter it took 10.5 us of the epoch, under ncu).
// The step is taken in FP64 on the FP32 moments and parameters: with FP32
// constants 1 - 0.999f is 1.3e-5 off and 1 - 0.999f^8 4e-6, the same for every
// parameter, and the loss after a few epochs of a steep start moves by ten
// times as much.
struct AdamStep {
  double lr, b1, b2, eps, c1, c2;  // c = 1 - b^step
};
static AdamStep adam_step(float lr, int step) {
  const double b1 = 0.9, b2 = 0.999;
  return AdamStep{(double)lr, b1, b2, 1e-8, 1.0 - pow(b1, step), 1.0 - pow(b2, step)};
}
__global__ void __launch_bounds__(1024) mlp_update_kernel(const float *__restrict__ part, int rows,
                                                          float *P, float *M, float *V, AdamStep a,
                                                          float *G, float *loss) {
  __shared__ double red[32][33];
  const int c = threadIdx.x & 31, r0 = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + c;
  double s = 0.0;  // the rows are FP32 sums of a few hundred samples each
  if (k <= kNP) {
#pragma unroll 10
    for (int r = r0; r < rows; r += 32) s += part[(size_t)r * kRow + k];
  }
  red[r0][c] = s;
  __syncthreads();
  if (r0) return;
  s = 0.0;
#pragma unroll
  for (int r = 0; r < 32; r++) s += red[r][c];
  if (k > kNP) return;
  const double g = s;
  if (k == kNP) {
    *loss = (float)g;
  } else if (M) {
    const double m = a.b1 * M[k] + (1.0 - a.b1) * g;
    const double v = a.b2 * V[k] + (1.0 - a.b2) * g * g;
    M[k] = (float)m;
    V[k] = (float)v;
    P[k] = (float)(P[k] - a.lr * (m / a.c1) / (sqrt(v / a.c2) + a.eps));
  } else {
    G[k] = (float)g;
  }
}


uint64_t splitmix(uint64_t &s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

}  // namespace

struct sapb_mlp {
  sapb_dev *d = nullptr;
  float *P = nullptr, *G = nullptr, *M = nullptr, *V = nullptr, *loss = nullptr;
  float *part = nullptr;  // gradient rows, one per block of the backward grid
  int part_rows = 0;
  float *X = nullptr, *T = nullptr, *Y = nullptr;  // device staging
  int cap = 0;
  int steps = 0;
};

#define MK(m, call)                                                                        \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess)                                                                 \
      return sapb_fail((m)->d, SAPB_ECUDA, "%s: %s", #call, cudaGetErrorString(e_));       \
  } while (0)

// backward grid: two blocks per SM at most, never more than chunks
static int bwd_grid(const sapb_mlp *m, int n) {
  return std::max(1, std::min((n + kM - 1) / kM, 2 * m->d->num_sms));
}

static int mlp_reserve_part(sapb_mlp *m, int n) {
  const int rows = bwd_grid(m, n);
  if (rows <= m->part_rows) return SAPB_OK;
  cudaFree(m->part);
  m->part = nullptr;
  m->part_rows = 0;
  if (cudaMalloc(&m->part, sizeof(float) * kRow * (size_t)rows) != cudaSuccess) {
    cudaGetLastError();
    m->part = nullptr;
    return sapb_fail(m->d, SAPB_ENOMEM, "mlp gradient rows for %d samples", n);
  }
  m->part_rows = rows;
  return SAPB_OK;
}

// Gradient of the staged samples into G (a == nullptr) or one Adam step.
static cudaError_t mlp_step(sapb_mlp *m, int n, const AdamStep *a, cudaStream_t st) {
  const int rows = bwd_grid(m, n);
  mlp_backward_kernel<<<rows, kT, sizeof(BackSmem), st>>>(m->P, n, m->X, m->T, m->part);
  mlp_update_kernel<<<(kNP + 1 + 31) / 32, 1024, 0, st>>>(m->part, rows, m->P, a ? m->M : nullptr,
                                                         m->V, a ? *a : AdamStep{}, m->G, m->loss);
  return cudaGetLastError();
}

static int mlp_reserve(sapb_mlp *m, int n) {
  if (n <= m->cap) return SAPB_OK;
  const int cap = n + n / 2 + 1024;
  cudaFree(m->X);
  m->X = m->T = m->Y = nullptr;
  m->cap = 0;
  // one allocation: X, T, Y
  if (cudaMalloc(&m->X, sizeof(float) * (kPropIn + 2) * (size_t)cap) != cudaSuccess) {
    cudaGetLastError();
    m->X = nullptr;
    return sapb_fail(m->d, SAPB_ENOMEM, "mlp staging for %d samples", cap);
  }
  m->T = m->X + (size_t)kPropIn * cap;
  m->Y = m->T + cap;
  m->cap = cap;
  return SAPB_OK;
}

extern "C" {

int sapb_mlp_num_params(void) { return kNP; }

int sapb_mlp_create(sapb_dev *d, unsigned long long seed, sapb_mlp **out) {
  if (!d || !out) return sapb_fail(d, SAPB_EINVAL, "bad arguments");
  *out = nullptr;
  sapb_mlp *m = new (std::nothrow) sapb_mlp();
  if (!m) return sapb_fail(d, SAPB_ENOMEM, "host allocation");
  m->d = d;
  if (cudaSetDevice(d->device) != cudaSuccess ||
      cudaMalloc(&m->P, sizeof(float) * 4 * kRow) != cudaSuccess ||  // P G M V, loss
      cudaFuncSetAttribute(mlp_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(BackSmem)) != cudaSuccess ||
      cudaFuncSetAttribute(mlp_eval_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(EvalSmem)) != cudaSuccess ||
      cudaFuncSetAttribute(mlp_eval_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(EvalSmem)) != cudaSuccess) {
    cudaGetLastError();
    sapb_mlp_destroy(m);
    return sapb_fail(d, SAPB_ENOMEM, "mlp parameter buffers");
  }
  m->G = m->P + kRow;
  m->M = m->G + kRow;
  m->V = m->M + kRow;
  m->loss = m->V + kNP;
  // He-uniform hidden layers, Glorot-uniform output layer, zero biases,
  // from a seeded splitmix64 stream.
  std::vector<float> p(kNP, 0.f);
  uint64_t s = seed;
  auto uni = [&](float lim) {
    const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
    return (float)((2.0 * u - 1.0) * lim);
  };
  for (int k = 0; k < kH * kIn; k++) p[oW1 + k] = uni(sqrtf(6.f / kIn));
  for (int k = 0; k < kH * kH; k++) p[oW2 + k] = uni(sqrtf(6.f / kH));
  for (int k = 0; k < kH * kH; k++) p[oW3 + k] = uni(sqrtf(6.f / kH));
  for (int k = 0; k < kH; k++) p[oW4 + k] = uni(sqrtf(6.f / (kH + 1)));
  int rc = sapb_mlp_set_params(m, p.data());
  if (rc) {
    sapb_mlp_destroy(m);
    return rc;
  }
  *out = m;
  return SAPB_OK;
}

int sapb_mlp_destroy(sapb_mlp *m) {
  if (!m) return SAPB_OK;
  cudaFree(m->P);
  cudaFree(m->part);
  cudaFree(m->X);
  delete m;
  return SAPB_OK;
}

// Parameters and moments travel on the handle's stream, where the kernels that
// use them run: the stream is non-blocking, so nothing orders it after a copy or
// a memset on the default stream (a pageable copy this small returns before it
// has landed, a memset at once).
int sapb_mlp_set_params(sapb_mlp *m, const float *params) {
  if (!m || !params) return sapb_fail(m ? m->d : nullptr, SAPB_EINVAL, "bad arguments");
  MK(m, cudaSetDevice(m->d->device));
  cudaStream_t st = m->d->stream;
  // captured, the copy would read `params` at each replay
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  MK(m, cudaStreamIsCapturing(st, &capture));
  if (capture != cudaStreamCaptureStatusNone)
    return sapb_fail(m->d, SAPB_ECUDA, "network parameters set on a stream that is being captured");
  MK(m, cudaMemcpyAsync(m->P, params, sizeof(float) * kNP, cudaMemcpyHostToDevice, st));
  MK(m, cudaMemsetAsync(m->M, 0, sizeof(float) * kNP, st));
  MK(m, cudaMemsetAsync(m->V, 0, sizeof(float) * kNP, st));
  // a pageable source has been staged by now, a pinned one may still be read
  cudaPointerAttributes at{};
  MK(m, cudaPointerGetAttributes(&at, params));
  if (at.type != cudaMemoryTypeUnregistered) MK(m, cudaStreamSynchronize(st));
  m->steps = 0;
  return SAPB_OK;
}

int sapb_mlp_get_params(sapb_mlp *m, float *params) {
  if (!m || !params) return sapb_fail(m ? m->d : nullptr, SAPB_EINVAL, "bad arguments");
  MK(m, cudaSetDevice(m->d->device));
  cudaStream_t st = m->d->stream;
  MK(m, cudaMemcpyAsync(params, m->P, sizeof(float) * kNP, cudaMemcpyDeviceToHost, st));
  MK(m, cudaStreamSynchronize(st));
  return SAPB_OK;
}

int sapb_mlp_forward(sapb_mlp *m, int n, const float *x, float *y) {
  if (!m || n < 0 || (n && (!x || !y))) return sapb_fail(m ? m->d : nullptr, SAPB_EINVAL, "bad arguments");
  if (n == 0) return SAPB_OK;
  MK(m, cudaSetDevice(m->d->device));
  int rc = mlp_reserve(m, n);
  if (rc) return rc;
  cudaStream_t st = m->d->stream;
  MK(m, cudaMemcpyAsync(m->X, x, sizeof(float) * kIn * (size_t)n, cudaMemcpyHostToDevice, st));
  mlp_eval_kernel<false><<<(n + kM - 1) / kM, kT, sizeof(EvalSmem), st>>>(m->P, n, m->X,
                                                                          MlpScale{}, m->Y);
  MK(m, cudaGetLastError());
  MK(m, cudaMemcpyAsync(y, m->Y, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost, st));
  MK(m, cudaStreamSynchronize(st));
  return SAPB_OK;
}

int sapb_mlp_propose(sapb_mlp *m, int n, const float *in, const float *mu, const float *sd,
                     float target, float max_down, float max_up, float clip, float *h2_out) {
  if (!m || n < 0 || (n && (!in || !mu || !sd || !h2_out)) || !(target > 0.f))
    return sapb_fail(m ? m->d : nullptr, SAPB_EINVAL, "bad arguments");
  if (n == 0) return SAPB_OK;
  MK(m, cudaSetDevice(m->d->device));
  int rc = mlp_reserve(m, n);
  if (rc) return rc;
  MlpScale sc;
  for (int k = 0; k < kIn; k++) {
    sc.mu[k] = mu[k];
    sc.sd[k] = sd[k];
  }
  sc.target = target;
  sc.max_down = max_down;
  sc.max_up = max_up;
  sc.clip = clip;
  cudaStream_t st = m->d->stream;
  MK(m, cudaMemcpyAsync(m->X, in, sizeof(float) * kPropIn * (size_t)n, cudaMemcpyHostToDevice, st));
  mlp_eval_kernel<true><<<(n + kM - 1) / kM, kT, sizeof(EvalSmem), st>>>(m->P, n, m->X, sc, m->Y);
  MK(m, cudaGetLastError());
  MK(m, cudaMemcpyAsync(h2_out, m->Y, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost, st));
  MK(m, cudaStreamSynchronize(st));
  return SAPB_OK;
}

int sapb_mlp_gradient(sapb_mlp *m, int n, const float *x, const float *t, float *grad,
                      float *loss) {
  if (!m || n <= 0 || !x || !t) return sapb_fail(m ? m->d : nullptr, SAPB_EINVAL, "bad arguments");
  MK(m, cudaSetDevice(m->d->device));
  int rc = mlp_reserve(m, n);
  if (!rc) rc = mlp_reserve_part(m, n);
  if (rc) return rc;
  cudaStream_t st = m->d->stream;
  MK(m, cudaMemcpyAsync(m->X, x, sizeof(float) * kIn * (size_t)n, cudaMemcpyHostToDevice, st));
  MK(m, cudaMemcpyAsync(m->T, t, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, st));
  MK(m, mlp_step(m, n, nullptr, st));
  if (grad) MK(m, cudaMemcpyAsync(grad, m->G, sizeof(float) * kNP, cudaMemcpyDeviceToHost, st));
  float l = 0.f;
  MK(m, cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, st));
  MK(m, cudaStreamSynchronize(st));
  if (loss) *loss = l;
  return SAPB_OK;
}

int sapb_mlp_train(sapb_mlp *m, int n, const float *x, const float *t, int epochs, float lr,
                   float *loss) {
  if (!m || n <= 0 || epochs <= 0) return sapb_fail(m ? m->d : nullptr, SAPB_EINVAL, "bad arguments");
  MK(m, cudaSetDevice(m->d->device));
  int rc = mlp_reserve(m, n);
  if (!rc) rc = mlp_reserve_part(m, n);
  if (rc) return rc;
  cudaStream_t st = m->d->stream;
  MK(m, cudaMemcpyAsync(m->X, x, sizeof(float) * kIn * (size_t)n, cudaMemcpyHostToDevice, st));
  MK(m, cudaMemcpyAsync(m->T, t, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, st));
  for (int e = 0; e < epochs; e++) {
    const AdamStep a = adam_step(lr, ++m->steps);
    MK(m, mlp_step(m, n, &a, st));
  }
  float l = 0.f;
  MK(m, cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, st));
  MK(m, cudaStreamSynchronize(st));
  if (loss) *loss = l;  // loss before the last update
  return SAPB_OK;
}

}  // extern "C"
