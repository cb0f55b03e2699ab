// Truncated-DFT kernels of the Fourier layers (bdda_fno.cu): width 32, MD
// kept frequencies per axis (0 .. MD/2 - 1 and -MD/2 .. -1).
//
// All of them are bound by HBM when each activation is read once; the axis
// transform they replace read its input once per 8 outputs (z forward, 1.2 GB of
// useful bytes in 458 us at 45 x 55 x 70 cells and 16 samples; 0.36 GB in 133 us
// now) and formed all MD frequencies of real data where MD / 2 + 1 determine
// them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace bdda {
namespace {

constexpr int kWd = 32;   // channels

__device__ __forceinline__ float2 cfma2(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}

// The six axis tables, T[q][p]: forward z, y, x (q = cell, p = mode):
// exp(-2 pi i f n / N); inverse x, y, z (q = mode, p = cell): the conjugate.
// Evaluated in double and rounded, as the host did with long double (0.4 ms a
// call for 170 cells; the launch is 3 us).
struct TableArgs {
  float2* tab[6];
  int N[6];
  int md;
};
__global__ void fno_tables_kernel(TableArgs a) {
  const int t = blockIdx.y, N = a.N[t], md = a.md, h = md / 2;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N * md; e += gridDim.x * blockDim.x) {
    const bool inv = t >= 3;
    const int n = inv ? e % N : e / md, j = inv ? e / N : e % md;
    const int f = j < h ? j : N - (md - j);
    const int r = (int)((int64_t)f * n % N);
    double s, c;
    sincospi(2.0 * r / N, &s, &c);
    a.tab[t][e] = make_float2((float)c, (float)(inv ? s : -s));
  }
}

// z forward of a real field in[o][q][32] (q < Q): out[o][j][32] = scale sum_q in T[q][j].
// A warp takes LINES lines, a lane a channel; frequencies 0 .. MD/2 are summed,
// the others are their conjugates.
template <int MD, int LINES>
__global__ void __launch_bounds__(256) zfwd_kernel(const float* in, float2* out, const float2* T, int64_t O, int Q,
                                                   float scale) {
  constexpr int H = MD / 2;
  extern __shared__ float2 tsm[];   // [Q][H]: T[q][1 .. H]
  for (int e = threadIdx.x; e < Q * H; e += 256) {
    const int q = e / H;
    tsm[e] = T[q * MD + 1 + (e - q * H)];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int64_t o0 = (blockIdx.x * 8LL + (threadIdx.x >> 5)) * LINES; o0 < O; o0 += (int64_t)gridDim.x * 8 * LINES) {
    float re[LINES][H + 1], im[LINES][H + 1];
#pragma unroll
    for (int l = 0; l < LINES; ++l)
#pragma unroll
      for (int j = 0; j <= H; ++j) re[l][j] = im[l][j] = 0.f;
    const float* p[LINES];
#pragma unroll
    for (int l = 0; l < LINES; ++l) p[l] = in + min(o0 + l, O - 1) * Q * kWd + lane;
#pragma unroll 8
    for (int q = 0; q < Q; ++q) {
      float x[LINES];
#pragma unroll
      for (int l = 0; l < LINES; ++l) x[l] = p[l][q * kWd];
#pragma unroll
      for (int l = 0; l < LINES; ++l) re[l][0] += x[l];
#pragma unroll
      for (int j = 1; j <= H; ++j) {
        const float2 w = tsm[q * H + j - 1];
#pragma unroll
        for (int l = 0; l < LINES; ++l) {
          re[l][j] = fmaf(x[l], w.x, re[l][j]);
          im[l][j] = fmaf(x[l], w.y, im[l][j]);
        }
      }
    }
#pragma unroll
    for (int l = 0; l < LINES; ++l) {
      if (o0 + l >= O) continue;
      float2* d = out + (o0 + l) * MD * kWd + lane;
#pragma unroll
      for (int j = 0; j <= H; ++j) d[j * kWd] = make_float2(scale * re[l][j], scale * im[l][j]);
#pragma unroll
      for (int j = H + 1; j < MD; ++j) d[j * kWd] = make_float2(scale * re[l][MD - j], -scale * im[l][MD - j]);
    }
  }
}

// y / x forward of a complex field: out[o][p][i] = scale sum_{q<Q} in[o][q][i] T[q][p], p < MD.
// A thread takes one i and all p.
template <int MD>
__global__ void __launch_bounds__(256) cfwd_kernel(const float2* in, float2* out, const float2* T, int64_t O, int Q,
                                                   int I, float scale) {
  extern __shared__ float2 tsm[];   // [Q][MD]
  for (int e = threadIdx.x; e < Q * MD; e += 256) tsm[e] = T[e];
  __syncthreads();
  const int64_t n = O * I;
  for (int64_t t = blockIdx.x * 256LL + threadIdx.x; t < n; t += gridDim.x * 256LL) {
    const int64_t o = t / I;
    const int i = (int)(t - o * I);
    float2 a[MD];
#pragma unroll
    for (int p = 0; p < MD; ++p) a[p] = make_float2(0.f, 0.f);
    const float2* s = in + o * Q * I + i;
#pragma unroll 8
    for (int q = 0; q < Q; ++q) {
      const float2 x = s[(int64_t)q * I];
#pragma unroll
      for (int p = 0; p < MD; ++p) a[p] = cfma2(x, tsm[q * MD + p], a[p]);
    }
    float2* d = out + o * MD * I + i;
#pragma unroll
    for (int p = 0; p < MD; ++p) d[(int64_t)p * I] = make_float2(scale * a[p].x, scale * a[p].y);
  }
}

// x / y inverse: out[o][p][i] = sum_{q<MD} in[o][q][i] T[q][p], p < N, PCH of them per thread.
constexpr int kInvRows = 12;
template <int MD>
__global__ void __launch_bounds__(256) cinv_kernel(const float4* in, float4* out, const float2* T, int64_t O, int N,
                                                   int I2) {
  extern __shared__ float2 tsm[];   // [N][MD]
  for (int e = threadIdx.x; e < N * MD; e += 256) {
    const int q = e / N, p = e - q * N;
    tsm[p * MD + q] = T[e];
  }
  __syncthreads();
  const int chunks = (N + kInvRows - 1) / kInvRows;
  const int64_t n = O * chunks * I2;
  for (int64_t t = blockIdx.x * 256LL + threadIdx.x; t < n; t += gridDim.x * 256LL) {
    const int64_t oc = t / I2;
    const int i = (int)(t - oc * I2);
    const int64_t o = oc / chunks;
    const int p0 = (int)(oc - o * chunks) * kInvRows, p1 = min(N, p0 + kInvRows);
    float4 x[MD];
#pragma unroll
    for (int q = 0; q < MD; ++q) x[q] = in[(o * MD + q) * I2 + i];
    for (int p = p0; p < p1; ++p) {
      float2 a = make_float2(0.f, 0.f), b = a;
#pragma unroll
      for (int q = 0; q < MD; ++q) {
        const float2 w = tsm[p * MD + q];
        a = cfma2(make_float2(x[q].x, x[q].y), w, a);
        b = cfma2(make_float2(x[q].z, x[q].w), w, b);
      }
      out[(o * N + p) * I2 + i] = make_float4(a.x, a.y, b.x, b.y);
    }
  }
}

// z inverse, real part, as 2 H + 1 real coefficients of this lane's channel on
// the basis 1, (T_j.x, T_j.y) j = 1 .. H: two conjugate frequencies share one pair.
template <int MD> __device__ __forceinline__ void zinv_coefs(const float2* t1, int lane, float* u) {
  constexpr int H = MD / 2;
  u[0] = t1[lane].x;
#pragma unroll
  for (int j = 1; j < H; ++j) {
    const float2 a = t1[j * kWd + lane], b = t1[(MD - j) * kWd + lane];
    u[2 * j - 1] = a.x + b.x;
    u[2 * j] = b.y - a.y;
  }
  const float2 a = t1[H * kWd + lane];
  u[2 * H - 1] = a.x;
  u[2 * H] = -a.y;
}
// ---- spectral mixing, one CTA per mode k ---------------------------------------------
// S[b][k][o] = sum_i R[k][i][o] A[b][k][i]: a lane keeps column o of R_k in registers.
__global__ void __launch_bounds__(256) spec_mix_kernel(const float2* A, const float2* R, float2* S, int B, int K) {
  __shared__ float2 as[8][kWd];
  const int k = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float2 r[kWd];
#pragma unroll
  for (int i = 0; i < kWd; ++i) r[i] = R[((int64_t)k * kWd + i) * kWd + lane];
  for (int b = w; b < B; b += 8) {
    __syncwarp();
    as[w][lane] = A[((int64_t)b * K + k) * kWd + lane];
    __syncwarp();
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kWd; ++i) acc = cfma2(as[w][i], r[i], acc);
    S[((int64_t)b * K + k) * kWd + lane] = acc;
  }
}

// gA[b][k][i] = sum_o conj(R[k][i][o]) gS[b][k][o]: a lane keeps row i.  WIDE: R
// lies on a 16-byte boundary (parameters that are a slice of a larger array may
// not).  Two kernels, not a branch in one: with both forms in it, loss and
// gradients at 24 modes and 2 samples took 2.2 ms instead of 1.5.
template <bool WIDE>
__global__ void __launch_bounds__(256) spec_mix_bwd_data_kernel(const float2* gS, const float2* R, float2* gA, int B,
                                                                int K) {
  __shared__ float2 gs[8][kWd];
  const int k = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float2 r[kWd];
  const float2* row = R + ((int64_t)k * kWd + lane) * kWd;
  if constexpr (WIDE) {
#pragma unroll
    for (int o = 0; o < kWd / 2; ++o) {
      const float4 v = reinterpret_cast<const float4*>(row)[o];
      r[2 * o] = make_float2(v.x, -v.y);
      r[2 * o + 1] = make_float2(v.z, -v.w);
    }
  } else {
#pragma unroll
    for (int o = 0; o < kWd; ++o) r[o] = make_float2(row[o].x, -row[o].y);
  }
  for (int b = w; b < B; b += 8) {
    __syncwarp();
    gs[w][lane] = gS[((int64_t)b * K + k) * kWd + lane];
    __syncwarp();
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int o = 0; o < kWd; ++o) acc = cfma2(r[o], gs[w][o], acc);
    gA[((int64_t)b * K + k) * kWd + lane] = acc;
  }
}

// gR[k][i][o] += sum_b conj(A[b][k][i]) gS[b][k][o]: warp w takes i = 4 w .. 4 w + 3, a lane o.
__global__ void __launch_bounds__(256) spec_mix_bwd_weight_kernel(const float2* A, const float2* gS, float2* gR, int B,
                                                                  int K) {
  const int k = blockIdx.x, lane = threadIdx.x & 31, i0 = (threadIdx.x >> 5) * 4;
  float2 acc[4];
  float2* d = gR + ((int64_t)k * kWd + i0) * kWd + lane;
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = d[i * kWd];
#pragma unroll 4
  for (int b = 0; b < B; ++b) {
    const int64_t at = ((int64_t)b * K + k) * kWd;
    const float2 g = gS[at + lane];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = A[at + i0 + i];
      acc[i] = cfma2(make_float2(a.x, -a.y), g, acc[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i * kWd] = acc[i];
}

}  // namespace
}  // namespace bdda
