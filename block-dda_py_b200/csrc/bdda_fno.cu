// Fourier-neural-operator warm start for the block solvers: hand-written
// forward, backward, optimiser and inference kernels (no counterpart in the
// reference, whose solvers start from X0 = 0, bl_krylov.py:84-85,146).
//
// Network (per sample = one particle lattice x one orientation, B samples of
// one lattice per call), activations FP32, cell-major [B][Nx][Ny][Nz][C]:
//   lift      v0 = P x + p                      (cin -> width, pointwise)
//   layer l   v   = act(W_l v + b_l + K_l v)     (l = 0..layers-1, no act on the last)
//             K_l v = Re IDFT( R_l . DFT(v) ) on the `modes` lowest frequencies
//             per axis (|f| < modes/2), R_l one complex width x width matrix per mode
//   project   y = Q2 gelu(Q1 v + q1) + q2        (width -> proj -> cout)
// The truncated DFT is separable: three axis transforms, each a small complex
// matrix product over the kept modes (no full-length FFT is formed).  act =
// GELU (erf form).  Parameters are one flat FP32 array (layout below).
#include <cmath>
#include <cstring>

#include <algorithm>
#include <utility>

#include "bdda_fno_spec.cuh"
#include "bdda_internal.h"
#include "bdda_small.cuh"

namespace bdda {
namespace {

struct FnoCfg {
  int cin, width, cout, proj, layers, modes;
};

// Longest lattice axis the network runs on (its truncated-DFT tables hold
// kMaxAxis x modes entries per axis).
constexpr int kMaxAxis = 512;

// parameter offsets (floats)
struct FnoParams {
  size_t P, p, R[8], W[8], b[8], Q1, q1, Q2, q2, total;
};

FnoParams param_layout(const FnoCfg& c) {
  FnoParams o;
  const size_t K = (size_t)c.modes * c.modes * c.modes;
  size_t off = 0;
  o.P = off; off += (size_t)c.cin * c.width;
  o.p = off; off += c.width;
  for (int l = 0; l < c.layers; ++l) {
    o.R[l] = off; off += K * c.width * c.width * 2;
    o.W[l] = off; off += (size_t)c.width * c.width;
    o.b[l] = off; off += c.width;
  }
  o.Q1 = off; off += (size_t)c.width * c.proj;
  o.q1 = off; off += c.proj;
  o.Q2 = off; off += (size_t)c.proj * c.cout;
  o.q2 = off; off += c.cout;
  o.total = off;
  return o;
}

bool cfg_ok(const bdda_fno_config* c) {
  return c && c->cin >= 1 && c->cin <= 64 && c->width >= 1 && c->width <= 64 && c->cout >= 1 && c->cout <= 64 &&
         c->proj >= 1 && c->proj <= 128 && c->layers >= 1 && c->layers <= 8 && c->modes >= 2 && c->modes <= 32 &&
         (c->modes % 2) == 0;
}

FnoCfg to_cfg(const bdda_fno_config* c) { return FnoCfg{c->cin, c->width, c->cout, c->proj, c->layers, c->modes}; }

// 2^x: the unit's approximation (2 ulp) without exp2f's scaling around it for results below 2^-126, which flush to 0
__device__ __forceinline__ float pow2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// Two values at once: the packed FMA of sm_100 does both in one issue slot, with the same rounding.
typedef unsigned long long pair2;
__device__ __forceinline__ pair2 pack2(float x, float y) {
  pair2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(pair2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ pair2 both(float x) { return pack2(x, x); }
__device__ __forceinline__ pair2 fma2(pair2 a, pair2 b, pair2 c) {
  pair2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// Normal distribution function Phi(z) = erfc(-z / sqrt 2) / 2 without a branch:
// erfc(a) = 2^q(a) for a = |z| / sqrt 2 <= 6, q a polynomial of degree 12 with
// q(0) = 0 fitted to log2 erfc (weighted least squares, iterated towards the
// smallest largest error: 4.5e-9, and 1.5e-6 x max(erfc, 1e-3)).  In FP32 Phi is
// within 7e-8 (0.5 (1 + erff): 6.4e-8), for 17 instructions instead of about 40 (erff runs
// both of its branches in most warps; GELU was two thirds of the projection's
// instructions).
__device__ __forceinline__ float2 normal_cdf(float2 z) {
  const float ax = fminf(fabsf(z.x) * 0.70710678118654752f, 16.0f);
  const float ay = fminf(fabsf(z.y) * 0.70710678118654752f, 16.0f);
  const pair2 a = pack2(ax, ay);
  pair2 q = both(-8.052739808e-09f);
  q = fma2(q, a, both(2.966770865e-07f));
  q = fma2(q, a, both(-4.839806024e-06f));
  q = fma2(q, a, both(4.601462206e-05f));
  q = fma2(q, a, both(-2.808824938e-04f));
  q = fma2(q, a, both(1.121692010e-03f));
  q = fma2(q, a, both(-2.623979701e-03f));
  q = fma2(q, a, both(3.509852104e-04f));
  q = fma2(q, a, both(2.760771848e-02f));
  q = fma2(q, a, both(-1.482808441e-01f));
  q = fma2(q, a, both(-9.184457064e-01f));
  q = fma2(q, a, both(-1.627907157e+00f));
  const float2 v = unpack2(q);
  const float ex = 0.5f * pow2(v.x * ax), ey = 0.5f * pow2(v.y * ay);
  return make_float2(z.x < 0.f ? ex : 1.0f - ex, z.y < 0.f ? ey : 1.0f - ey);
}
// its derivative exp(-z^2 / 2) / sqrt(2 pi)
__device__ __forceinline__ float normal_pdf(float z) {
  return 0.39894228040143268f * pow2(-0.72134752044448170f * z * z);
}
__device__ __forceinline__ float2 gelu(float2 z) {
  const float2 c = normal_cdf(z);
  return make_float2(z.x * c.x, z.y * c.y);
}
__device__ __forceinline__ float2 gelu_grad(float2 z) {
  const float2 c = normal_cdf(z);
  return make_float2(fmaf(z.x, normal_pdf(z.x), c.x), fmaf(z.y, normal_pdf(z.y), c.y));
}

// ---- tensor-core pointwise layers --------------------------------------------------------------
// The 32 x 32 layers and the 32 x 64 projection run on the tensor cores:
// mma.sync m16n8k8 with TF32 operands and FP32 accumulation, each product
// split in three, a b ~ a_hi b_hi + a_hi b_lo + a_lo b_hi with a_hi = tf32(a),
// a_lo = tf32(a - a_hi), which keeps the accuracy of FP32 (the dropped a_lo b_lo
// is at most 2^-22 of a product, 2^-24 typically, an FP32 rounding 2^-24).  The unit's accumulator is cut, not rounded (a
// relative bias of -1.5e-7 after 32 columns), so each step of 8 columns starts from
// zero and is added in FP32: error 0.9e-7 rms, an FP32 chain's is 1.0e-7.
// Fragments of m16n8k8 (lane = 4 g + t):
// A (16 x 8) a0 (g, t), a1 (g + 8, t), a2 (g, t + 4), a3 (g + 8, t + 4);
// B (8 x 8) b0 (t, g), b1 (t + 4, g); D (16 x 8) d0 (g, 2t), d1 (g, 2t + 1),
// d2 (g + 8, 2t), d3 (g + 8, 2t + 1).  Each warp owns 16-row tiles of the
// activations, staged in shared memory by 16-byte loads.
//
// The layers are bound by HBM, so each kernel carries what is next to it: a
// forward layer evaluates its spectral branch's z inverse itself, the output
// projection runs both of its layers, and a backward layer takes the data
// gradient, the spectral branch's gradient, the previous activation's
// derivative and the weight gradient of one tile together.  One inference at
// 45 x 55 x 70 cells and 16 samples moves 4.9 GB that way, 12 GB with a kernel per
// step before (7.4 -> 3.0 ms).
__device__ __forceinline__ uint32_t tf32_of(float v) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ void split_tf32(float v, uint32_t& hi, uint32_t& lo) {
  hi = tf32_of(v);
  lo = tf32_of(v - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float* d, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// d += A B over K = 8 KS columns: A from a 16-row tile at `at` (row stride AS);
// B as split fragments, one 16-byte word per lane: (h of rows t, t + 4; l of the same)
template <int KS, int NS, int AS>
__device__ __forceinline__ void tile_mma(float (*acc)[4], const float* at, const uint4* frag, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
    uint32_t ah[4], al[4];
    split_tf32(at[g * AS + ks * 8 + t], ah[0], al[0]);
    split_tf32(at[(g + 8) * AS + ks * 8 + t], ah[1], al[1]);
    split_tf32(at[g * AS + ks * 8 + t + 4], ah[2], al[2]);
    split_tf32(at[(g + 8) * AS + ks * 8 + t + 4], ah[3], al[3]);
#pragma unroll
    for (int ns = 0; ns < NS; ++ns) {
      const uint4 f = frag[(ks * NS + ns) * 32 + lane];
      const uint32_t h[2] = {f.x, f.y}, l[2] = {f.z, f.w};
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      mma_tf32(d, al, h);
      mma_tf32(d, ah, l);
      mma_tf32(d, ah, h);
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[ns][q] += d[q];
    }
  }
}
// acc[mt][ns] += X^T G over the 16 rows of two tiles (X: 16 MT columns, row stride XS; G: 8 NS columns, row stride GS)
template <int MT, int NS, int XS, int GS>
__device__ __forceinline__ void tile_mma_t(float (*acc)[NS][4], const float* xt, const float* gt, int g, int t) {
#pragma unroll
  for (int k0 = 0; k0 < 16; k0 += 8) {
    uint32_t bh[NS][2], bl[NS][2];
#pragma unroll
    for (int ns = 0; ns < NS; ++ns) {
      split_tf32(gt[(k0 + t) * GS + ns * 8 + g], bh[ns][0], bl[ns][0]);
      split_tf32(gt[(k0 + t + 4) * GS + ns * 8 + g], bh[ns][1], bl[ns][1]);
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      uint32_t ah[4], al[4];   // A[i][m] = x[m][i]
      split_tf32(xt[(k0 + t) * XS + mt * 16 + g], ah[0], al[0]);
      split_tf32(xt[(k0 + t) * XS + mt * 16 + g + 8], ah[1], al[1]);
      split_tf32(xt[(k0 + t + 4) * XS + mt * 16 + g], ah[2], al[2]);
      split_tf32(xt[(k0 + t + 4) * XS + mt * 16 + g + 8], ah[3], al[3]);
#pragma unroll
      for (int ns = 0; ns < NS; ++ns) {
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        mma_tf32(d, al, bh[ns]);
        mma_tf32(d, ah, bl[ns]);
        mma_tf32(d, ah, bh[ns]);
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[mt][ns][q] += d[q];
      }
    }
  }
}
// component of B's fragments that holds element (k, n) of a matrix of 8 NS columns
template <int NS> __device__ __forceinline__ int frag_at(int k, int n) {
  return (((k >> 3) * NS + (n >> 3)) * 32 + (n & 7) * 4 + (k & 3)) * 4 + ((k >> 2) & 1);
}
// W (CI x CO, by rows) as the fragments of W or (TR) of its transpose
template <int CI, int CO, bool TR> __device__ __forceinline__ void split_weights(const float* W, uint4* frag) {
  uint32_t* f = reinterpret_cast<uint32_t*>(frag);
  for (int e = threadIdx.x; e < CI * CO; e += blockDim.x) {
    const int i = e / CO, o = e - i * CO, at = TR ? frag_at<CI / 8>(o, i) : frag_at<CO / 8>(i, o);
    split_tf32(W[e], f[at], f[at + 2]);
  }
}

// rows m0 .. m0 + 15 (below M) of a row-major (M x C) array, held by the warp in registers ...
template <int C> struct RowTile {
  float4 v[16 * C / 128];
  __device__ __forceinline__ void load(const float* src, int64_t m0, int64_t M, int lane) {
#pragma unroll
    for (int q = 0; q < 16 * C / 128; ++q) {
      const int e = lane + 32 * q, r = e / (C / 4), c4 = e - r * (C / 4);
      v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m0 + r < M) v[q] = *reinterpret_cast<const float4*>(src + (m0 + r) * C + 4 * c4);
    }
  }
  // ... and put into a tile of row stride TS
  template <int TS> __device__ __forceinline__ void put(float* tile, int lane) const {
#pragma unroll
    for (int q = 0; q < 16 * C / 128; ++q) {
      const int e = lane + 32 * q, r = e / (C / 4), c4 = e - r * (C / 4);
      *reinterpret_cast<float4*>(tile + r * TS + 4 * c4) = v[q];
    }
  }
};

// ---- lift: v = x P + p, 13 -> 32 --------------------------------------------------------
// A lane is an output channel; 32 rows of x are staged per warp (padded to 16
// columns) and broadcast.  One row per thread, as before, wrote 128 bytes a
// lane apart (468 us at 2.8 M rows; 115 now).
constexpr int kCin = 13, kW = 32, kCout = 6, kProj = 64;   // the shipped network

__global__ void __launch_bounds__(256) lift_kernel(const float* x, const float* P, const float* p, float* v, int64_t M) {
  __shared__ __align__(16) float xs[8][32 * 16];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float w[kCin];
#pragma unroll
  for (int i = 0; i < kCin; ++i) w[i] = P[i * kW + lane];
  const float b = p[lane];
  float* t = xs[warp];
  for (int64_t m0 = (blockIdx.x * 8LL + warp) * 32; m0 < M; m0 += gridDim.x * 256LL) {
    const int nr = (int)min((int64_t)32, M - m0);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kCin; ++q) {
      const int e = lane + 32 * q, r = e / kCin;
      if (r < nr) t[r * 16 + e - r * kCin] = x[m0 * kCin + e];
    }
    __syncwarp();
#pragma unroll 4
    for (int r = 0; r < nr; ++r) {
      const float4* row = reinterpret_cast<const float4*>(t + r * 16);
      const float4 a = row[0], c = row[1], d = row[2];
      float s = fmaf(a.x, w[0], b);
      s = fmaf(a.y, w[1], s); s = fmaf(a.z, w[2], s); s = fmaf(a.w, w[3], s);
      s = fmaf(c.x, w[4], s); s = fmaf(c.y, w[5], s); s = fmaf(c.z, w[6], s); s = fmaf(c.w, w[7], s);
      s = fmaf(d.x, w[8], s); s = fmaf(d.y, w[9], s); s = fmaf(d.z, w[10], s); s = fmaf(d.w, w[11], s);
      s = fmaf(t[r * 16 + 12], w[12], s);
      v[(m0 + r) * kW + lane] = s;
    }
  }
}

// gP += x^T gv, gp += column sums of gv (per-CTA sums, then one atomic each)
__global__ void __launch_bounds__(256) lift_bwd_kernel(const float* x, const float* gv, float* gP, float* gp, int64_t M) {
  __shared__ __align__(16) float xs[8][32 * 16];
  __shared__ float red[(kCin + 1) * kW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < (kCin + 1) * kW; e += 256) red[e] = 0.f;
  __syncthreads();
  float acc[kCin + 1];
#pragma unroll
  for (int i = 0; i <= kCin; ++i) acc[i] = 0.f;
  float* t = xs[warp];
  for (int64_t m0 = (blockIdx.x * 8LL + warp) * 32; m0 < M; m0 += gridDim.x * 256LL) {
    const int nr = (int)min((int64_t)32, M - m0);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kCin; ++q) {
      const int e = lane + 32 * q, r = e / kCin;
      if (r < nr) t[r * 16 + e - r * kCin] = x[m0 * kCin + e];
    }
    __syncwarp();
#pragma unroll 4
    for (int r = 0; r < nr; ++r) {
      const float g = gv[(m0 + r) * kW + lane];
#pragma unroll
      for (int i = 0; i < kCin; ++i) acc[i] = fmaf(t[r * 16 + i], g, acc[i]);
      acc[kCin] += g;
    }
  }
#pragma unroll
  for (int i = 0; i <= kCin; ++i) atomicAdd(&red[i * kW + lane], acc[i]);
  __syncthreads();
  for (int e = threadIdx.x; e < (kCin + 1) * kW; e += 256)
    atomicAdd(e < kCin * kW ? &gP[e] : &gp[e - kCin * kW], red[e]);
}

// ---- forward layer: z = v W + b + scale Re IDFT_z(t1), v' = act(z) ----------------------------
// A warp takes the lines (o) in turn, 16 rows of the line at a time.  The z
// inverse is part of the product: a row's basis values (bdda_fno_spec.cuh) are
// KU more columns of A, the line's coefficients KU more rows of B, split into
// fragments once per line.
template <int MD> struct ZInv {
  static constexpr int KU = (MD + 1 + 7) / 8 * 8;        // 2 H + 1 coefficients, padded
  static constexpr int frags = KU / 8 * (kW / 8) * 32;   // uint4 per warp
  static constexpr int row = KU + 4;                     // basis row stride (conflict-free A reads)
  static __host__ __device__ int rows(int N) { return (N + 15) / 16 * 16; }
  // the whole axis's basis is kept in shared memory: kMaxAxis cells at 32 modes are 90 KB
  static size_t basis_bytes(int N) { return (size_t)rows(N) * row * 4; }
};
// [rows(N)][row]: 1, T_j.x, T_j.y of cell n; zero past the coefficients and past N
template <int MD> __device__ __forceinline__ void zinv_basis_rows(float* bas, const float2* T, int N) {
  for (int e = threadIdx.x; e < ZInv<MD>::rows(N) * ZInv<MD>::row; e += blockDim.x) {
    const int n = e / ZInv<MD>::row, k = e - n * ZInv<MD>::row;
    float v = 0.f;
    if (n < N && k <= MD) {
      const float2 w = T[((k + 1) / 2) * N + n];
      v = k == 0 ? 1.f : (k & 1) ? w.x : w.y;
    }
    bas[e] = v;
  }
}
template <int MD> __device__ __forceinline__ void zinv_frags(const float2* t1, float scale, uint4* frag, int lane) {
  float u[MD + 1];
  zinv_coefs<MD>(t1, lane, u);
  uint32_t* f = reinterpret_cast<uint32_t*>(frag);
#pragma unroll
  for (int k = 0; k < ZInv<MD>::KU; ++k) {
    const int at = frag_at<kW / 8>(k, lane);
    if (k <= MD) split_tf32(scale * u[k], f[at], f[at + 2]);
    else f[at] = f[at + 2] = 0u;
  }
}

template <int MD>
__global__ void __launch_bounds__(256, 3) layer_fwd_kernel(const float* v, const float2* t1, const float2* T,
                                                           const float* Wt, const float* bias, float* z, float* y,
                                                           int64_t O, int N, float scale, int act) {
  typedef ZInv<MD> ZI;
  constexpr int XS = kW + 4;
  extern __shared__ __align__(16) unsigned char fsm[];
  uint4* wf = reinterpret_cast<uint4*>(fsm);                  // [4][4][32]
  uint4* uf = wf + 16 * 32;                                   // [8][frags]
  float* bs = reinterpret_cast<float*>(uf + 8 * ZI::frags);
  float* tiles = bs + kW;                                     // [8][16 XS]
  float* bas = tiles + 8 * 16 * XS;
  split_weights<kW, kW, false>(Wt, wf);
  for (int e = threadIdx.x; e < kW; e += 256) bs[e] = bias[e];
  zinv_basis_rows<MD>(bas, T, N);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float* xt = tiles + warp * 16 * XS;
  uint4* uw = uf + warp * ZI::frags;
  for (int64_t o = blockIdx.x * 8LL + warp; o < O; o += gridDim.x * 8LL) {
    const int64_t m1 = (o + 1) * N;
    RowTile<kW> next;
    next.load(v, o * N, m1, lane);
    __syncwarp();
    zinv_frags<MD>(t1 + o * MD * kW, scale, uw, lane);
    for (int n0 = 0; n0 < N; n0 += 16) {
      const int64_t m0 = o * N + n0;
      __syncwarp();
      next.put<XS>(xt, lane);
      if (n0 + 16 < N) next.load(v, m0 + 16, m1, lane);
      __syncwarp();
      float acc[kW / 8][4];
#pragma unroll
      for (int ns = 0; ns < kW / 8; ++ns) acc[ns][0] = acc[ns][1] = acc[ns][2] = acc[ns][3] = 0.f;
      tile_mma<kW / 8, kW / 8, XS>(acc, xt, wf, lane);
      tile_mma<ZI::KU / 8, kW / 8, ZI::row>(acc, bas + n0 * ZI::row, uw, lane);
#pragma unroll
      for (int ns = 0; ns < kW / 8; ++ns)
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
          const int c = ns * 8 + 2 * t;
          const int64_t m = m0 + g + 8 * hr;
          if (m >= m1) continue;
          const float z0 = acc[ns][2 * hr] + bs[c], z1 = acc[ns][2 * hr + 1] + bs[c + 1];
          if (z) *reinterpret_cast<float2*>(z + m * kW + c) = make_float2(z0, z1);
          *reinterpret_cast<float2*>(y + m * kW + c) = act ? gelu(make_float2(z0, z1)) : make_float2(z0, z1);
        }
    }
  }
}

// ---- projection: y = gelu(v Q1 + q1) Q2 + q2; the hidden pre-activation is kept for training ----
__global__ void __launch_bounds__(256, 2) proj_fwd_kernel(const float* v, const float* Q1, const float* q1,
                                                       const float* Q2, const float* q2, float* zq, float* y, int64_t M) {
  constexpr int XS = kW + 4;
  extern __shared__ __align__(16) unsigned char fsm[];
  uint4* wf = reinterpret_cast<uint4*>(fsm);   // [4][8][32]
  float* b1 = reinterpret_cast<float*>(wf + 32 * 32);
  float* w2 = b1 + kProj;                      // [kProj][8]
  float* tiles = w2 + kProj * 8;               // [8][16 XS]
  split_weights<kW, kProj, false>(Q1, wf);
  for (int e = threadIdx.x; e < kProj; e += 256) b1[e] = q1[e];
  for (int e = threadIdx.x; e < kProj * 8; e += 256) {
    const int i = e >> 3, o = e & 7;
    w2[e] = o < kCout ? Q2[i * kCout + o] : 0.f;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float* xt = tiles + warp * 16 * XS;
  const int64_t ntile = (M + 15) / 16, step = gridDim.x * 8LL;
  int64_t tile = blockIdx.x * 8LL + warp;
  RowTile<kW> next;
  if (tile < ntile) next.load(v, tile * 16, M, lane);
  for (; tile < ntile; tile += step) {
    const int64_t m0 = tile * 16;
    __syncwarp();
    next.put<XS>(xt, lane);
    if (tile + step < ntile) next.load(v, (tile + step) * 16, M, lane);
    __syncwarp();
    float acc[kProj / 8][4];
#pragma unroll
    for (int ns = 0; ns < kProj / 8; ++ns) acc[ns][0] = acc[ns][1] = acc[ns][2] = acc[ns][3] = 0.f;
    tile_mma<kW / 8, kProj / 8, XS>(acc, xt, wf, lane);
    float out[2][kCout];
#pragma unroll
    for (int hr = 0; hr < 2; ++hr)
#pragma unroll
      for (int o = 0; o < kCout; ++o) out[hr][o] = 0.f;
#pragma unroll
    for (int ns = 0; ns < kProj / 8; ++ns) {
      const int c = ns * 8 + 2 * t;
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        acc[ns][2 * hr] += b1[c];
        acc[ns][2 * hr + 1] += b1[c + 1];
        const int64_t m = m0 + g + 8 * hr;
        if (zq && m < M) *reinterpret_cast<float2*>(zq + m * kProj + c) = make_float2(acc[ns][2 * hr], acc[ns][2 * hr + 1]);
      }
      const float2 h2[2] = {gelu(make_float2(acc[ns][0], acc[ns][1])), gelu(make_float2(acc[ns][2], acc[ns][3]))};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float4 wa = *reinterpret_cast<const float4*>(w2 + (c + q) * 8);
        const float2 wb = *reinterpret_cast<const float2*>(w2 + (c + q) * 8 + 4);
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
          const float h = q ? h2[hr].y : h2[hr].x;
          out[hr][0] = fmaf(h, wa.x, out[hr][0]); out[hr][1] = fmaf(h, wa.y, out[hr][1]);
          out[hr][2] = fmaf(h, wa.z, out[hr][2]); out[hr][3] = fmaf(h, wa.w, out[hr][3]);
          out[hr][4] = fmaf(h, wb.x, out[hr][4]); out[hr][5] = fmaf(h, wb.y, out[hr][5]);
        }
      }
    }
#pragma unroll
    for (int hr = 0; hr < 2; ++hr) {
#pragma unroll
      for (int o = 0; o < kCout; ++o) {
        out[hr][o] += __shfl_xor_sync(0xffffffffu, out[hr][o], 1);
        out[hr][o] += __shfl_xor_sync(0xffffffffu, out[hr][o], 2);
      }
      const int64_t m = m0 + g + 8 * hr;
      if (m < M && t < 3) {
        const float a = t == 0 ? out[hr][0] : t == 1 ? out[hr][2] : out[hr][4];
        const float b = t == 0 ? out[hr][1] : t == 1 ? out[hr][3] : out[hr][5];
        *reinterpret_cast<float2*>(y + m * kCout + 2 * t) = make_float2(a + q2[2 * t], b + q2[2 * t + 1]);
      }
    }
  }
}

// Backward of the projection, one 16-row tile at a time: gzq = (gy Q2^T) gelu'(zq),
// gv = gzq Q1^T (times act'(zlast) when the last layer has one: it has none),
// gQ1 += v^T gzq, gq1 += gzq, gQ2 += gelu(zq)^T gy, gq2 += gy.
constexpr int kProjWarps = 4;
constexpr int kPvS = kW + 8, kPgS = kProj + 8, kPyS = 8;   // tile row strides: v, gzq, gy
__global__ void __launch_bounds__(32 * kProjWarps, 3) proj_bwd_kernel(const float* v, const float* zq, const float* gy,
                                                                  const float* Q1, const float* Q2, float* gv,
                                                                  float* gQ1, float* gq1, float* gQ2, float* gq2,
                                                                  int64_t M) {
  constexpr int NRED = kW * kProj + kProj + kProj * kCout + kCout;
  extern __shared__ __align__(16) unsigned char fsm[];
  uint4* wf = reinterpret_cast<uint4*>(fsm);   // Q1 transposed: [8][4][32]
  float* red = reinterpret_cast<float*>(wf + 32 * 32);
  float* tiles = red + (NRED + 3) / 4 * 4;
  constexpr int TILE = 16 * (kPvS + kPgS + kPyS);
  split_weights<kW, kProj, true>(Q1, wf);
  for (int e = threadIdx.x; e < NRED; e += blockDim.x) red[e] = 0.f;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float* vt = tiles + warp * TILE;
  float* gt = vt + 16 * kPvS;
  float* yt = gt + 16 * kPgS;
  pair2 w2[kCout], aq2[kCout];   // rows lane, lane + 32 of Q2 and of its gradient
  float b1[2] = {0.f, 0.f}, b2 = 0.f;
#pragma unroll
  for (int o = 0; o < kCout; ++o) {
    w2[o] = pack2(Q2[lane * kCout + o], Q2[(lane + 32) * kCout + o]);
    aq2[o] = both(0.f);
  }
  float aq1[2][kProj / 8][4];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int ns = 0; ns < kProj / 8; ++ns) aq1[mt][ns][0] = aq1[mt][ns][1] = aq1[mt][ns][2] = aq1[mt][ns][3] = 0.f;
  const int64_t ntile = (M + 15) / 16;
  for (int64_t tile = blockIdx.x * (int64_t)kProjWarps + warp; tile < ntile; tile += (int64_t)gridDim.x * kProjWarps) {
    const int64_t m0 = tile * 16;
    const int nr = (int)min((int64_t)16, M - m0);
    __syncwarp();
    RowTile<kW> vr;
    vr.load(v, m0, M, lane);
    for (int e = lane; e < 16 * kPyS; e += 32) {
      const int r = e / kPyS, o = e - r * kPyS;
      yt[e] = r < nr && o < kCout ? gy[(m0 + r) * kCout + o] : 0.f;
    }
    __syncwarp();
#pragma unroll 8
    for (int r = 0; r < 16; ++r) {
      pair2 y6[kCout], gh = both(0.f);
#pragma unroll
      for (int o = 0; o < kCout; ++o) y6[o] = both(yt[r * kPyS + o]);
      const float* zr = zq + (m0 + min(r, nr - 1)) * kProj + lane;   // rows past the end: gy is zero
      const float2 zz = make_float2(zr[0], zr[32]);
#pragma unroll
      for (int o = 0; o < kCout; ++o) gh = fma2(y6[o], w2[o], gh);
      const float2 cdf = normal_cdf(zz), gy2 = unpack2(gh);
      const pair2 h = pack2(zz.x * cdf.x, zz.y * cdf.y);
      const float gx = gy2.x * fmaf(zz.x, normal_pdf(zz.x), cdf.x);
      const float gw = gy2.y * fmaf(zz.y, normal_pdf(zz.y), cdf.y);
#pragma unroll
      for (int o = 0; o < kCout; ++o) aq2[o] = fma2(h, y6[o], aq2[o]);
      gt[r * kPgS + lane] = gx;
      gt[r * kPgS + lane + 32] = gw;
      b1[0] += gx;
      b1[1] += gw;
      if (lane < kCout) b2 += yt[r * kPyS + lane];
    }
    vr.put<kPvS>(vt, lane);
    __syncwarp();
    float acc[kW / 8][4];
#pragma unroll
    for (int ns = 0; ns < kW / 8; ++ns) acc[ns][0] = acc[ns][1] = acc[ns][2] = acc[ns][3] = 0.f;
    tile_mma<kProj / 8, kW / 8, kPgS>(acc, gt, wf, lane);
#pragma unroll
    for (int ns = 0; ns < kW / 8; ++ns)
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const int64_t m = m0 + g + 8 * hr;
        if (m < M)
          *reinterpret_cast<float2*>(gv + m * kW + ns * 8 + 2 * t) = make_float2(acc[ns][2 * hr], acc[ns][2 * hr + 1]);
      }
    tile_mma_t<2, kProj / 8, kPvS, kPgS>(aq1, vt, gt, g, t);
  }
  float* rq1 = red;
  float* rb1 = rq1 + kW * kProj;
  float* rq2 = rb1 + kProj;
  float* rb2 = rq2 + kProj * kCout;
#pragma unroll
  for (int q = 0; q < 2; ++q) atomicAdd(&rb1[lane + 32 * q], b1[q]);
  if (lane < kCout) atomicAdd(&rb2[lane], b2);
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int ns = 0; ns < kProj / 8; ++ns)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        atomicAdd(&rq1[(mt * 16 + g + 8 * (q >> 1)) * kProj + ns * 8 + 2 * t + (q & 1)], aq1[mt][ns][q]);
#pragma unroll
  for (int o = 0; o < kCout; ++o) {
    const float2 v = unpack2(aq2[o]);
    atomicAdd(&rq2[lane * kCout + o], v.x);
    atomicAdd(&rq2[(lane + 32) * kCout + o], v.y);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < kW * kProj; e += blockDim.x) atomicAdd(&gQ1[e], rq1[e]);
  for (int e = threadIdx.x; e < kProj; e += blockDim.x) atomicAdd(&gq1[e], rb1[e]);
  for (int e = threadIdx.x; e < kProj * kCout; e += blockDim.x) atomicAdd(&gQ2[e], rq2[e]);
  for (int e = threadIdx.x; e < kCout; e += blockDim.x) atomicAdd(&gq2[e], rb2[e]);
}

// Backward of a layer given gz (gradient of its z): gW += v^T gz, gb += gz, and the
// gradient of its input, gz W^T + Re IDFT_z(t1) (the spectral branch's, its x and
// y inverses done), times act'(zprev) of the layer below (null: the layer below has none).
constexpr int kLayerWarps = 4;
template <int MD>
__global__ void __launch_bounds__(32 * kLayerWarps, 4) layer_bwd_kernel(const float* gz, const float* v, const float2* t1,
                                                                    const float2* T, const float* Wt,
                                                                    const float* zprev, float* gout, float* gW,
                                                                    float* gb, int64_t O, int N) {
  typedef ZInv<MD> ZI;
  constexpr int TS = kW + 8;
  extern __shared__ __align__(16) unsigned char fsm[];
  uint4* wf = reinterpret_cast<uint4*>(fsm);                  // W transposed: [4][4][32]
  uint4* uf = wf + 16 * 32;                                   // [warps][frags]
  float* red = reinterpret_cast<float*>(uf + kLayerWarps * ZI::frags);
  float* tiles = red + kW * kW + kW;                          // [warps][2][16 TS]
  float* bas = tiles + kLayerWarps * 2 * 16 * TS;
  split_weights<kW, kW, true>(Wt, wf);
  zinv_basis_rows<MD>(bas, T, N);
  for (int e = threadIdx.x; e < kW * kW + kW; e += blockDim.x) red[e] = 0.f;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float* gt = tiles + warp * 2 * 16 * TS;
  float* vt = gt + 16 * TS;
  uint4* uw = uf + warp * ZI::frags;
  float aw[2][kW / 8][4], bsum = 0.f;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int ns = 0; ns < kW / 8; ++ns)
#pragma unroll
      for (int q = 0; q < 4; ++q) aw[mt][ns][q] = 0.f;
  for (int64_t o = blockIdx.x * (int64_t)kLayerWarps + warp; o < O; o += (int64_t)gridDim.x * kLayerWarps) {
    const int64_t m1 = (o + 1) * N;
    RowTile<kW> ng, nv;
    ng.load(gz, o * N, m1, lane);
    nv.load(v, o * N, m1, lane);
    __syncwarp();
    zinv_frags<MD>(t1 + o * MD * kW, 1.f, uw, lane);
    for (int n0 = 0; n0 < N; n0 += 16) {
      const int64_t m0 = o * N + n0;
      __syncwarp();
      ng.put<TS>(gt, lane);
      nv.put<TS>(vt, lane);
      if (n0 + 16 < N) {
        ng.load(gz, m0 + 16, m1, lane);
        nv.load(v, m0 + 16, m1, lane);
      }
      __syncwarp();
      float bt = 0.f;
#pragma unroll
      for (int r = 0; r < 16; ++r) bt += gt[r * TS + lane];
      bsum += bt;
      float acc[kW / 8][4];
#pragma unroll
      for (int ns = 0; ns < kW / 8; ++ns) acc[ns][0] = acc[ns][1] = acc[ns][2] = acc[ns][3] = 0.f;
      tile_mma<kW / 8, kW / 8, TS>(acc, gt, wf, lane);
      tile_mma<ZI::KU / 8, kW / 8, ZI::row>(acc, bas + n0 * ZI::row, uw, lane);
#pragma unroll
      for (int ns = 0; ns < kW / 8; ++ns)
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
          const int c = ns * 8 + 2 * t;
          const int64_t m = m0 + g + 8 * hr;
          if (m >= m1) continue;
          float a = acc[ns][2 * hr], b = acc[ns][2 * hr + 1];
          if (zprev) {
            const float2 zz = *reinterpret_cast<const float2*>(zprev + m * kW + c);
            const float2 dz = gelu_grad(zz);
            a *= dz.x;
            b *= dz.y;
          }
          *reinterpret_cast<float2*>(gout + m * kW + c) = make_float2(a, b);
        }
      tile_mma_t<2, kW / 8, TS, TS>(aw, vt, gt, g, t);
    }
  }
  atomicAdd(&red[kW * kW + lane], bsum);
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int ns = 0; ns < kW / 8; ++ns)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        atomicAdd(&red[(mt * 16 + g + 8 * (q >> 1)) * kW + ns * 8 + 2 * t + (q & 1)], aw[mt][ns][q]);
  __syncthreads();
  for (int e = threadIdx.x; e < kW * kW; e += blockDim.x) atomicAdd(&gW[e], red[e]);
  for (int e = threadIdx.x; e < kW; e += blockDim.x) atomicAdd(&gb[e], red[kW * kW + e]);
}

// ---- loss: masked relative squared error per sample -------------------------------------------
// L = (1/B) sum_b sum_m mask |y - t|^2 / sum_m mask |t|^2 ; gy = dL/dy
__global__ void loss_kernel(const float* y, const float* t, const float* mask, int64_t ncell, int C, int B,
                            const double* den, float* gy, double* loss) {
  const int64_t n = (int64_t)B * ncell * C;
  double local = 0.0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t bm = e / C;
    const int b = (int)(bm / ncell);
    const int64_t m = bm - (int64_t)b * ncell;
    const float w = mask[m];
    const float d = y[e] - t[e];
    const double s = 1.0 / (den[b] * B);
    gy[e] = (float)(2.0 * s * w * d);
    local += s * w * d * d;
  }
  for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, local);
}

// ---- Adam -------------------------------------------------------------------------------------
__global__ void adam_kernel(float* p, const float* g, float* m, float* v, int64_t n, float lr, float b1, float b2,
                            float eps, float c1, float c2, float wd) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = g[i] + wd * p[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// ---- features and warm start ---------------------------------------------------------------------
// scale[b] = sqrt(mean_r |B[r][b] / diag[r]|^2): column sums of a row-major
// block, so a CTA takes a range of rows with a lane per column (one CTA per column,
// reading every L-th value: 503 us at 235,000 rows x 16); the CTAs' sums are
// added in order by the second kernel.
constexpr int kScaleBlocks = 296;
__global__ void __launch_bounds__(256) jacobi_scale_kernel(const double2* diag, const double2* B, int64_t rows, int L,
                                                           double* partial) {
  __shared__ double red[256];
  const int lanes = L < 256 ? 256 / L : 1;   // rows side by side
  const int64_t per = (rows + gridDim.x - 1) / gridDim.x;
  const int64_t r0 = blockIdx.x * per, r1 = min(rows, r0 + per);
  for (int b0 = 0; b0 < L; b0 += 256) {
    const int cols = min(L - b0, 256);
    const int row = threadIdx.x / cols, b = threadIdx.x - row * cols;
    double local = 0.0;
    if (row < lanes)
      for (int64_t r = r0 + row; r < r1; r += lanes) {
        const double2 j = zdiv(B[r * L + b0 + b], diag[r]);
        local += j.x * j.x + j.y * j.y;
      }
    red[threadIdx.x] = local;
    __syncthreads();
    if (threadIdx.x < cols) {
      double s = 0.0;
      for (int q = 0; q < lanes; ++q) s += red[q * cols + threadIdx.x];
      partial[(int64_t)blockIdx.x * L + b0 + threadIdx.x] = s;
    }
    __syncthreads();
  }
}
__global__ void __launch_bounds__(256) jacobi_scale_sum_kernel(const double* partial, int nblk, int64_t rows, int L,
                                                               double* scale) {
  __shared__ double red[256];
  const int b = blockIdx.x;
  double s = 0.0;
  for (int q = threadIdx.x; q < nblk; q += 256) s += partial[(int64_t)q * L + b];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) scale[b] = sqrt(red[0] / (double)rows) + 1e-300;
}

// The lattice is walked in blocks of kCellTile cells x up to kColTile samples:
// a dipole's rows of B and X are read as runs over the samples, the cell-major
// fields of a sample as runs over the cells, and the two meet in shared memory.
// (One cell of one sample per thread: 16-byte reads a row apart.)
constexpr int kCellTile = 32, kColTile = 16;

// x[b][cell][:] = (mask, Re/Im chi_x, chi_y, chi_z, Re/Im J_x, J_y, J_z / scale) with
// J = B / diag the Jacobi guess of orientation b; zero outside the particle
__global__ void __launch_bounds__(256) features_kernel(const int32_t* cell_map, int64_t ncell, int n_occ, int L,
                                                       const double2* diag, const double2* B, const double* chi,
                                                       const double* scale, float* x, float* mask) {
  __shared__ float js[kColTile][kCellTile][6];
  __shared__ float ch[6];
  __shared__ int map[kCellTile];
  const int64_t tiles = (ncell + kCellTile - 1) / kCellTile;
  const int64_t c0 = blockIdx.x % tiles * kCellTile;
  const int b0 = (int)(blockIdx.x / tiles) * kColTile;
  const int nc = (int)min((int64_t)kCellTile, ncell - c0), nb = min(kColTile, L - b0);
  if (threadIdx.x < nc) {
    const int m = cell_map[c0 + threadIdx.x];
    map[threadIdx.x] = m >= 0 && m < n_occ ? m : -1;
    if (b0 == 0) mask[c0 + threadIdx.x] = m >= 0 ? 1.f : 0.f;
  }
  if (threadIdx.x >= 32 && threadIdx.x < 38) ch[threadIdx.x - 32] = (float)chi[threadIdx.x - 32];
  __syncthreads();
  for (int e = threadIdx.x; e < nc * 3 * nb; e += 256) {
    const int ca = e / nb, b = e - ca * nb, c = ca / 3, a = ca - 3 * c;
    float re = 0.f, im = 0.f;
    if (map[c] >= 0) {
      const int64_t r = 3 * (int64_t)map[c] + a;
      const double2 j = zdiv(B[r * L + b0 + b], diag[r]);
      const double s = 1.0 / scale[b0 + b];
      re = (float)(j.x * s);
      im = (float)(j.y * s);
    }
    js[b][c][2 * a] = re;
    js[b][c][2 * a + 1] = im;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nb * nc * kCin; e += 256) {
    const int b = e / (nc * kCin), q = e - b * (nc * kCin), c = q / kCin, i = q - c * kCin;
    float v = 0.f;
    if (map[c] >= 0) v = i == 0 ? 1.f : i < 7 ? ch[i - 1] : js[b][c][i - 7];
    x[((int64_t)(b0 + b) * ncell + c0) * kCin + q] = v;
  }
}

// X0[3m + a][b] = J + scale[b] (y_re + i y_im) at the occupied cells
__global__ void __launch_bounds__(256) warm_start_kernel(const int32_t* cell_map, int64_t ncell, int n_occ, int L,
                                                         const double2* diag, const double2* B, const double* scale,
                                                         const float* y, double2* X0) {
  __shared__ float ys[kColTile][kCellTile * 6 + 1];
  __shared__ int map[kCellTile];
  const int64_t tiles = (ncell + kCellTile - 1) / kCellTile;
  const int64_t c0 = blockIdx.x % tiles * kCellTile;
  const int b0 = (int)(blockIdx.x / tiles) * kColTile;
  const int nc = (int)min((int64_t)kCellTile, ncell - c0), nb = min(kColTile, L - b0);
  if (threadIdx.x < nc) {
    const int m = cell_map[c0 + threadIdx.x];
    map[threadIdx.x] = m >= 0 && m < n_occ ? m : -1;
  }
  for (int e = threadIdx.x; e < nb * nc * 6; e += 256) {
    const int b = e / (nc * 6), q = e - b * (nc * 6);
    ys[b][q] = y[((int64_t)(b0 + b) * ncell + c0) * 6 + q];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nc * 3 * nb; e += 256) {
    const int ca = e / nb, b = e - ca * nb, c = ca / 3, a = ca - 3 * c;
    if (map[c] < 0) continue;
    const int64_t r = 3 * (int64_t)map[c] + a, i = r * L + b0 + b;
    const double2 j = zdiv(B[i], diag[r]);
    const double s = scale[b0 + b];
    X0[i] = make_double2(j.x + s * ys[b][c * 6 + 2 * a], j.y + s * ys[b][c * 6 + 2 * a + 1]);
  }
}

// target t[b][cell][:] = (X - J) / scale at occupied cells, 0 elsewhere, and den[b] += sum |t|^2
__global__ void __launch_bounds__(256) target_kernel(const int32_t* cell_map, int64_t ncell, int n_occ, int L,
                                                     const double2* diag, const double2* B, const double2* X,
                                                     const double* scale, float* t6, double* den) {
  __shared__ float ts[kColTile][kCellTile * 6 + 1];
  __shared__ int map[kCellTile];
  const int64_t tiles = (ncell + kCellTile - 1) / kCellTile;
  const int64_t c0 = blockIdx.x % tiles * kCellTile;
  const int b0 = (int)(blockIdx.x / tiles) * kColTile;
  const int nc = (int)min((int64_t)kCellTile, ncell - c0), nb = min(kColTile, L - b0);
  if (threadIdx.x < nc) {
    const int m = cell_map[c0 + threadIdx.x];
    map[threadIdx.x] = m >= 0 && m < n_occ ? m : -1;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nc * 3 * nb; e += 256) {
    const int ca = e / nb, b = e - ca * nb, c = ca / 3, a = ca - 3 * c;
    float re = 0.f, im = 0.f;
    if (map[c] >= 0) {
      const int64_t r = 3 * (int64_t)map[c] + a, i = r * L + b0 + b;
      const double2 j = zdiv(B[i], diag[r]), x = X[i];
      const double s = 1.0 / scale[b0 + b];
      re = (float)((x.x - j.x) * s);
      im = (float)((x.y - j.y) * s);
    }
    ts[b][c * 6 + 2 * a] = re;
    ts[b][c * 6 + 2 * a + 1] = im;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nb * nc * 6; e += 256) {
    const int b = e / (nc * 6), q = e - b * (nc * 6);
    t6[((int64_t)(b0 + b) * ncell + c0) * 6 + q] = ts[b][q];
  }
  // a warp per sample in turn; cells outside the particle add zero
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b = warp; b < nb; b += 8) {
    double s = 0.0;
    for (int q = lane; q < nc * 6; q += 32) s += (double)ts[b][q] * ts[b][q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0 && s != 0.0) atomicAdd(&den[b0 + b], s);
  }
}

// ---- host orchestration -----------------------------------------------------------------------------
#define BDDA_TRY_F(expr)           \
  do {                             \
    int s_ = (expr);               \
    if (s_ != BDDA_OK) return s_;  \
  } while (0)

int grid_for(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16)); }

struct FnoWork {
  size_t x, v[9], z[9], zq, y, A[8], S, t1, t2, gv, gv2, part, gS, gA, tabs, mask, tgt, gy, den, chi, loss, total;
};

struct Shape {
  int B, n[3];
  int64_t ncell, M;    // cells, rows = B * ncell
  int K;               // modes^3
};

FnoWork work_layout(const FnoCfg& c, const Shape& s) {
  FnoWork w;
  size_t off = 0;
  auto take = [&](size_t bytes) { const size_t o = off; off = (off + bytes + 255) & ~(size_t)255; return o; };
  const int64_t M = s.M;
  const int Wd = c.width, md = c.modes;
  w.x = take(M * c.cin * 4);
  for (int l = 0; l <= c.layers; ++l) w.v[l] = take(M * Wd * 4);
  for (int l = 0; l < c.layers; ++l) w.z[l] = take(M * Wd * 4);
  w.zq = take(M * c.proj * 4);
  w.y = take(M * c.cout * 4);
  for (int l = 0; l < c.layers; ++l) w.A[l] = take((size_t)s.B * s.K * Wd * 8);
  w.S = take((size_t)s.B * s.K * Wd * 8);
  // axis intermediates: after z: B Nx Ny md Wd; after y: B Nx md md Wd (complex)
  const size_t t1 = (size_t)s.B * s.n[0] * s.n[1] * md * Wd * 8;
  const size_t t2 = (size_t)s.B * s.n[0] * md * md * Wd * 8;
  w.t1 = take(t1);
  w.t2 = take(t2);
  w.gv = take(M * Wd * 4);
  w.gv2 = take(M * Wd * 4);
  w.part = take((size_t)kScaleBlocks * s.B * 8);
  w.gS = take((size_t)s.B * s.K * Wd * 8);
  w.gA = take((size_t)s.B * s.K * Wd * 8);
  w.tabs = take((size_t)6 * kMaxAxis * 32 * 8);
  w.mask = take(s.ncell * 4);
  w.tgt = take(M * c.cout * 4);
  w.gy = take(M * c.cout * 4);
  w.den = take((size_t)s.B * 8);
  w.chi = take(6 * 8);
  w.loss = take(64);
  w.total = off;
  return w;
}

struct Ctx {
  FnoCfg c;
  FnoParams pl;
  Shape s;
  FnoWork wl;
  unsigned char* w;
  const float* prm;
  float* grad;
  cudaStream_t st;
  float2* tab[6];   // fwd z, y, x; inv x, y, z
};

template <typename Tp>
Tp* at(Ctx& x, size_t off) { return reinterpret_cast<Tp*>(x.w + off); }

int write_tables(Ctx& x) {
  const int ax_of[6] = {2, 1, 0, 0, 1, 2};
  TableArgs a;
  a.md = x.c.modes;
  int most = 1;
  for (int t = 0; t < 6; ++t) {
    a.tab[t] = x.tab[t];
    a.N[t] = x.s.n[ax_of[t]];
    most = std::max(most, a.N[t]);
  }
  fno_tables_kernel<<<dim3((most * a.md + 255) / 256, 6), 256, 0, x.st>>>(a);
  count_launch();
  BDDA_CUDA_TRY(cudaGetLastError());
  return BDDA_OK;
}

template <typename K> int raise_smem(K k, size_t smem) {
  if (smem > 48 * 1024)
    BDDA_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  return BDDA_OK;
}

// The kernels that know the number of modes.
template <int MD> struct Spectral {
  static constexpr int I2y = MD * kWd / 2, I2x = MD * MD * kWd / 2;
  static int cfwd(Ctx& x, const float2* in, float2* out, const float2* T, int64_t O, int Q, int I2, float scale) {
    const size_t smem = (size_t)Q * MD * sizeof(float2);
    BDDA_TRY_F(raise_smem(cfwd_kernel<MD>, smem));
    cfwd_kernel<MD><<<grid_for(O * 2 * I2), 256, smem, x.st>>>(in, out, T, O, Q, 2 * I2, scale);
    count_launch();
    BDDA_CUDA_TRY(cudaGetLastError());
    return BDDA_OK;
  }
  static int cinv(Ctx& x, const float2* in, float2* out, const float2* T, int64_t O, int N, int I2) {
    const size_t smem = (size_t)N * MD * sizeof(float2);
    BDDA_TRY_F(raise_smem(cinv_kernel<MD>, smem));
    cinv_kernel<MD><<<grid_for(O * I2 * ((N + kInvRows - 1) / kInvRows)), 256, smem, x.st>>>(
        reinterpret_cast<const float4*>(in), reinterpret_cast<float4*>(out), T, O, N, I2);
    count_launch();
    BDDA_CUDA_TRY(cudaGetLastError());
    return BDDA_OK;
  }
  // truncated forward DFT of a real [B][Nx][Ny][Nz][32] field into A [B][md^3][32] (scale s)
  static int dft_fwd(Ctx& x, const float* v, float2* A, float scale) {
    const int B = x.s.B, Nx = x.s.n[0], Ny = x.s.n[1], Nz = x.s.n[2];
    float2* t1 = at<float2>(x, x.wl.t1);
    float2* t2 = at<float2>(x, x.wl.t2);
    constexpr int LINES = MD <= 16 ? 2 : 1;
    const int64_t O = (int64_t)B * Nx * Ny;
    const size_t smem = (size_t)Nz * (MD / 2) * sizeof(float2);
    BDDA_TRY_F(raise_smem(zfwd_kernel<MD, LINES>, smem));
    zfwd_kernel<MD, LINES><<<(int)std::min<int64_t>(148 * 16, (O + 8 * LINES - 1) / (8 * LINES)), 256, smem, x.st>>>(
        v, t1, x.tab[0], O, Nz, 1.f);
    count_launch();
    BDDA_CUDA_TRY(cudaGetLastError());
    BDDA_TRY_F(cfwd(x, t1, t2, x.tab[1], (int64_t)B * Nx, Ny, I2y, 1.f));
    return cfwd(x, t2, A, x.tab[2], B, Nx, I2x, scale);
  }
  // x and y inverses of S [B][md^3][32] into t1 [B][Nx][Ny][md][32]; the z inverse is the next layer kernel's
  static int dft_inv_xy(Ctx& x, const float2* S) {
    const int B = x.s.B, Nx = x.s.n[0], Ny = x.s.n[1];
    float2* t2 = at<float2>(x, x.wl.t2);
    BDDA_TRY_F(cinv(x, S, t2, x.tab[3], B, Nx, I2x));
    return cinv(x, t2, at<float2>(x, x.wl.t1), x.tab[4], (int64_t)B * Nx, Ny, I2y);
  }
  static int layer_fwd(Ctx& x, const float* v, const float* W, const float* b, float* z, float* y, float scale, int act) {
    const int N = x.s.n[2];
    const int64_t O = (int64_t)x.s.B * x.s.n[0] * x.s.n[1];
    const size_t smem = ((size_t)(16 * 32 + 8 * ZInv<MD>::frags) * 4 + kW + 8 * 16 * (kW + 4)) * 4 +
                        ZInv<MD>::basis_bytes(N);
    BDDA_TRY_F(raise_smem(layer_fwd_kernel<MD>, smem));
    layer_fwd_kernel<MD><<<(int)std::min<int64_t>(148 * 3, (O + 7) / 8), 256, smem, x.st>>>(
        v, at<float2>(x, x.wl.t1), x.tab[5], W, b, z, y, O, N, scale, act);
    count_launch();
    BDDA_CUDA_TRY(cudaGetLastError());
    return BDDA_OK;
  }
  static int layer_bwd(Ctx& x, const float* gz, const float* v, const float* W, const float* zprev, float* gout,
                       float* gW, float* gb) {
    const int N = x.s.n[2];
    const int64_t O = (int64_t)x.s.B * x.s.n[0] * x.s.n[1];
    const size_t smem =
        ((size_t)(16 * 32 + kLayerWarps * ZInv<MD>::frags) * 4 + kW * kW + kW + kLayerWarps * 2 * 16 * (kW + 8)) * 4 +
        ZInv<MD>::basis_bytes(N);
    BDDA_TRY_F(raise_smem(layer_bwd_kernel<MD>, smem));
    layer_bwd_kernel<MD><<<(int)std::min<int64_t>(148 * 4, (O + kLayerWarps - 1) / kLayerWarps), 32 * kLayerWarps, smem,
                           x.st>>>(gz, v, at<float2>(x, x.wl.t1), x.tab[5], W, zprev, gout, gW, gb, O, N);
    count_launch();
    BDDA_CUDA_TRY(cudaGetLastError());
    return BDDA_OK;
  }

  static int forward(Ctx& x, bool train) {
    const FnoCfg& c = x.c;
    const float* P = x.prm;
    const float inv = 1.f / (float)x.s.ncell;
    lift_kernel<<<(int)std::min<int64_t>(148 * 8, (x.s.M + 255) / 256), 256, 0, x.st>>>(
        at<float>(x, x.wl.x), P + x.pl.P, P + x.pl.p, at<float>(x, x.wl.v[0]), x.s.M);
    count_launch();
    for (int l = 0; l < c.layers; ++l) {
      float* vl = at<float>(x, x.wl.v[l]);
      float2* A = at<float2>(x, x.wl.A[train ? l : 0]);
      float2* S = at<float2>(x, x.wl.S);
      BDDA_TRY_F(dft_fwd(x, vl, A, 1.f));
      spec_mix_kernel<<<x.s.K, 256, 0, x.st>>>(A, reinterpret_cast<const float2*>(P + x.pl.R[l]), S, x.s.B, x.s.K);
      count_launch();
      BDDA_TRY_F(dft_inv_xy(x, S));
      BDDA_TRY_F(layer_fwd(x, vl, P + x.pl.W[l], P + x.pl.b[l], train ? at<float>(x, x.wl.z[l]) : nullptr,
                           at<float>(x, x.wl.v[l + 1]), inv, l + 1 < c.layers ? 1 : 0));
    }
    const size_t smem = (size_t)(32 * 32 * 4 + kProj + kProj * 8 + 8 * 16 * (kW + 4)) * 4;
    BDDA_TRY_F(raise_smem(proj_fwd_kernel, smem));
    proj_fwd_kernel<<<(int)std::min<int64_t>(148 * 4, (x.s.M + 127) / 128), 256, smem, x.st>>>(
        at<float>(x, x.wl.v[c.layers]), P + x.pl.Q1, P + x.pl.q1, P + x.pl.Q2, P + x.pl.q2,
        train ? at<float>(x, x.wl.zq) : nullptr, at<float>(x, x.wl.y), x.s.M);
    count_launch();
    BDDA_CUDA_TRY(cudaGetLastError());
    return BDDA_OK;
  }

  // gradient of the loss w.r.t. every parameter, given the gradient gy of the output
  static int backward(Ctx& x, const float* gy) {
    const FnoCfg& c = x.c;
    const float* P = x.prm;
    float* G = x.grad;
    float* gz = at<float>(x, x.wl.gv);    // gradient of the current layer's z ...
    float* gn = at<float>(x, x.wl.gv2);   // ... and of the one below
    const float inv = 1.f / (float)x.s.ncell;
    constexpr int NRED = (kW * kProj + kProj + kProj * kCout + kCout + 3) / 4 * 4;
    const size_t smem = (size_t)(32 * 32 * 4 + NRED + kProjWarps * 16 * (kPvS + kPgS + kPyS)) * 4;
    BDDA_TRY_F(raise_smem(proj_bwd_kernel, smem));
    const int64_t tiles = (x.s.M + 15) / 16;
    proj_bwd_kernel<<<(int)std::min<int64_t>(148 * 3, (tiles + kProjWarps - 1) / kProjWarps), 32 * kProjWarps, smem, x.st>>>(
        at<float>(x, x.wl.v[c.layers]), at<float>(x, x.wl.zq), gy, P + x.pl.Q1, P + x.pl.Q2, gz, G + x.pl.Q1, G + x.pl.q1,
        G + x.pl.Q2, G + x.pl.q2, x.s.M);   // the last layer has no activation: gv is its gz
    count_launch();
    BDDA_CUDA_TRY(cudaGetLastError());
    for (int l = c.layers - 1; l >= 0; --l) {
      // spectral branch: s = inv Re IDFT(S): gS = inv DFT(gz); gA = R^H gS; gR += conj(A) gS; its part
      // of the input's gradient is Re IDFT(gA)
      float2* gS = at<float2>(x, x.wl.gS);
      float2* gA = at<float2>(x, x.wl.gA);
      BDDA_TRY_F(dft_fwd(x, gz, gS, inv));
      const float2* R = reinterpret_cast<const float2*>(P + x.pl.R[l]);
      if ((reinterpret_cast<uintptr_t>(R) & 15) == 0)
        spec_mix_bwd_data_kernel<true><<<x.s.K, 256, 0, x.st>>>(gS, R, gA, x.s.B, x.s.K);
      else
        spec_mix_bwd_data_kernel<false><<<x.s.K, 256, 0, x.st>>>(gS, R, gA, x.s.B, x.s.K);
      spec_mix_bwd_weight_kernel<<<x.s.K, 256, 0, x.st>>>(at<float2>(x, x.wl.A[l]), gS,
                                                          reinterpret_cast<float2*>(G + x.pl.R[l]), x.s.B, x.s.K);
      count_launch(2);
      BDDA_CUDA_TRY(cudaGetLastError());
      BDDA_TRY_F(dft_inv_xy(x, gA));
      BDDA_TRY_F(layer_bwd(x, gz, at<float>(x, x.wl.v[l]), P + x.pl.W[l], l > 0 ? at<float>(x, x.wl.z[l - 1]) : nullptr,
                           gn, G + x.pl.W[l], G + x.pl.b[l]));
      std::swap(gz, gn);
    }
    lift_bwd_kernel<<<(int)std::min<int64_t>(148 * 4, (x.s.M + 255) / 256), 256, 0, x.st>>>(
        at<float>(x, x.wl.x), gz, G + x.pl.P, G + x.pl.p, x.s.M);
    count_launch();
    BDDA_CUDA_TRY(cudaGetLastError());
    return BDDA_OK;
  }
};

bool shipped(const FnoCfg& c) { return c.cin == kCin && c.width == kW && c.cout == kCout && c.proj == kProj; }

#define BDDA_FNO_MODES(F) F(2) F(4) F(6) F(8) F(10) F(12) F(14) F(16) F(18) F(20) F(22) F(24) F(26) F(28) F(30) F(32)
int forward(Ctx& x, bool train) {
  switch (x.c.modes) {
#define BDDA_FNO_CASE(MD) case MD: return Spectral<MD>::forward(x, train);
    BDDA_FNO_MODES(BDDA_FNO_CASE)
#undef BDDA_FNO_CASE
    default: return BDDA_BAD_ARG;
  }
}
int backward(Ctx& x, const float* gy) {
  switch (x.c.modes) {
#define BDDA_FNO_CASE(MD) case MD: return Spectral<MD>::backward(x, gy);
    BDDA_FNO_MODES(BDDA_FNO_CASE)
#undef BDDA_FNO_CASE
    default: return BDDA_BAD_ARG;
  }
}

// CTAs of the kernels that walk cells x samples
unsigned cell_blocks(const Ctx& x) {
  return (unsigned)(((x.s.ncell + kCellTile - 1) / kCellTile) * ((x.s.B + kColTile - 1) / kColTile));
}

// tables: write the axis DFT tables into the workspace (bdda_fno_features
// does; the other entry points use the tables it left there)
int make_ctx(Ctx& x, const bdda_fno_config* cfg, int B, const int n[3], void* work, size_t work_bytes,
             const float* params, float* grads, cudaStream_t st, bool tables = false) {
  if (!cfg_ok(cfg) || B < 1 || !n) return BDDA_BAD_ARG;
  x.c = to_cfg(cfg);
  if (!shipped(x.c)) return BDDA_BAD_ARG;
  x.pl = param_layout(x.c);
  x.s.B = B;
  for (int a = 0; a < 3; ++a) {
    if (n[a] < x.c.modes || n[a] > kMaxAxis) return BDDA_BAD_ARG;
    x.s.n[a] = n[a];
  }
  x.s.ncell = (int64_t)n[0] * n[1] * n[2];
  x.s.M = x.s.ncell * B;
  x.s.K = x.c.modes * x.c.modes * x.c.modes;
  x.wl = work_layout(x.c, x.s);
  if (!work || work_bytes < x.wl.total) return BDDA_NO_WORKSPACE;
  x.w = static_cast<unsigned char*>(work);
  x.prm = params;
  x.grad = grads;
  x.st = st;
  float2* base = at<float2>(x, x.wl.tabs);
  for (int t = 0; t < 6; ++t) x.tab[t] = base + (size_t)t * kMaxAxis * 32;
  return tables ? write_tables(x) : BDDA_OK;
}

}  // namespace
}  // namespace bdda

using namespace bdda;

extern "C" {

size_t bdda_fno_param_count(const bdda_fno_config* cfg) {
  if (!cfg_ok(cfg)) return 0;
  return param_layout(to_cfg(cfg)).total;
}

size_t bdda_fno_workspace_bytes(const bdda_fno_config* cfg, int B, const int n[3]) {
  if (!cfg_ok(cfg) || B < 1 || !n) return 0;
  Shape s;
  s.B = B;
  for (int a = 0; a < 3; ++a) s.n[a] = n[a];
  s.ncell = (int64_t)n[0] * n[1] * n[2];
  s.M = s.ncell * B;
  s.K = cfg->modes * cfg->modes * cfg->modes;
  return work_layout(to_cfg(cfg), s).total;
}

int bdda_fno_features(const bdda_fno_config* cfg, const int n[3], int n_occ, int L, const int32_t* cell_map,
                      const void* diag, const void* B, const double chi[6], double* scale, void* work,
                      size_t work_bytes, void* stream) {
  if (!cfg_ok(cfg) || !n || n_occ < 1 || L < 1 || !cell_map || !diag || !B || !chi || !scale) return BDDA_BAD_ARG;
  Ctx x;
  const int s = make_ctx(x, cfg, L, n, work, work_bytes, nullptr, nullptr, static_cast<cudaStream_t>(stream), true);
  if (s != BDDA_OK) return s;
  double* tmp = at<double>(x, x.wl.chi);
  BDDA_CUDA_TRY(cudaMemcpyAsync(tmp, chi, 6 * sizeof(double), cudaMemcpyHostToDevice, x.st));
  double* partial = at<double>(x, x.wl.part);
  const int nblk = (int)std::min<int64_t>(kScaleBlocks, 3 * (int64_t)n_occ);
  jacobi_scale_kernel<<<nblk, 256, 0, x.st>>>(static_cast<const double2*>(diag), static_cast<const double2*>(B),
                                              3 * (int64_t)n_occ, L, partial);
  jacobi_scale_sum_kernel<<<L, 256, 0, x.st>>>(partial, nblk, 3 * (int64_t)n_occ, L, scale);
  features_kernel<<<cell_blocks(x), 256, 0, x.st>>>(cell_map, x.s.ncell, n_occ, L, static_cast<const double2*>(diag),
                                                    static_cast<const double2*>(B), tmp, scale, at<float>(x, x.wl.x),
                                                    at<float>(x, x.wl.mask));
  count_launch(3);
  BDDA_CUDA_TRY(cudaGetLastError());
  return BDDA_OK;
}

int bdda_fno_forward(const bdda_fno_config* cfg, int B, const int n[3], const float* params, int train, void* work,
                     size_t work_bytes, void* stream) {
  Ctx x;
  const int s = make_ctx(x, cfg, B, n, work, work_bytes, params, nullptr, static_cast<cudaStream_t>(stream));
  if (s != BDDA_OK) return s;
  if (!params) return BDDA_BAD_ARG;
  return forward(x, train != 0);
}

int bdda_fno_loss(const bdda_fno_config* cfg, int B, const int n[3], int n_occ, const int32_t* cell_map,
                  const void* diag, const void* Bm, const void* X, const double* scale, double* loss, void* work,
                  size_t work_bytes, void* stream) {
  Ctx x;
  const int s = make_ctx(x, cfg, B, n, work, work_bytes, nullptr, nullptr, static_cast<cudaStream_t>(stream));
  if (s != BDDA_OK) return s;
  if (!cell_map || !diag || !Bm || !X || !scale || !loss) return BDDA_BAD_ARG;
  float* tgt = at<float>(x, x.wl.tgt);
  double* den = at<double>(x, x.wl.den);
  double* dl = at<double>(x, x.wl.loss);
  BDDA_CUDA_TRY(cudaMemsetAsync(den, 0, (size_t)B * sizeof(double), x.st));
  BDDA_CUDA_TRY(cudaMemsetAsync(dl, 0, sizeof(double), x.st));
  target_kernel<<<cell_blocks(x), 256, 0, x.st>>>(cell_map, x.s.ncell, n_occ, B, static_cast<const double2*>(diag),
                                                  static_cast<const double2*>(Bm), static_cast<const double2*>(X), scale,
                                                  tgt, den);
  loss_kernel<<<grid_for(x.s.M * kCout), 256, 0, x.st>>>(at<float>(x, x.wl.y), tgt, at<float>(x, x.wl.mask),
                                                         x.s.ncell, kCout, B, den, at<float>(x, x.wl.gy), dl);
  count_launch(2);
  BDDA_CUDA_TRY(cudaGetLastError());
  BDDA_CUDA_TRY(cudaMemcpyAsync(loss, dl, sizeof(double), cudaMemcpyDeviceToHost, x.st));
  return BDDA_OK;
}

int bdda_fno_backward(const bdda_fno_config* cfg, int B, const int n[3], const float* params, const float* grad_out,
                      float* grads, void* work, size_t work_bytes, void* stream) {
  Ctx x;
  const int s = make_ctx(x, cfg, B, n, work, work_bytes, params, grads, static_cast<cudaStream_t>(stream));
  if (s != BDDA_OK) return s;
  if (!params || !grads) return BDDA_BAD_ARG;
  const float* gy = grad_out ? grad_out : at<float>(x, x.wl.gy);
  return backward(x, gy);
}

int bdda_fno_adam(float* params, const float* grads, float* m, float* v, size_t n, float lr, float beta1, float beta2,
                  float eps, float weight_decay, int step, void* stream) {
  if (!params || !grads || !m || !v || n == 0 || step < 1) return BDDA_BAD_ARG;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  adam_kernel<<<grid_for((int64_t)n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      params, grads, m, v, (int64_t)n, lr, beta1, beta2, eps, c1, c2, weight_decay);
  count_launch();
  BDDA_CUDA_TRY(cudaGetLastError());
  return BDDA_OK;
}

int bdda_fno_warm_start(const bdda_fno_config* cfg, const int n[3], int n_occ, int L, const int32_t* cell_map,
                        const void* diag, const void* B, const double* scale, void* X0, void* work,
                        size_t work_bytes, void* stream) {
  Ctx x;
  const int s = make_ctx(x, cfg, L, n, work, work_bytes, nullptr, nullptr, static_cast<cudaStream_t>(stream));
  if (s != BDDA_OK) return s;
  if (!cell_map || !diag || !B || !scale || !X0) return BDDA_BAD_ARG;
  warm_start_kernel<<<cell_blocks(x), 256, 0, x.st>>>(cell_map, x.s.ncell, n_occ, L, static_cast<const double2*>(diag),
                                                      static_cast<const double2*>(B), scale, at<float>(x, x.wl.y),
                                                      static_cast<double2*>(X0));
  count_launch();
  BDDA_CUDA_TRY(cudaGetLastError());
  return BDDA_OK;
}

size_t bdda_fno_buffer_offset(const bdda_fno_config* cfg, int B, const int n[3], int which) {
  if (!cfg_ok(cfg) || B < 1 || !n) return (size_t)-1;
  Shape s;
  s.B = B;
  for (int a = 0; a < 3; ++a) s.n[a] = n[a];
  s.ncell = (int64_t)n[0] * n[1] * n[2];
  s.M = s.ncell * B;
  s.K = cfg->modes * cfg->modes * cfg->modes;
  const FnoWork w = work_layout(to_cfg(cfg), s);
  switch (which) {
    case 0: return w.x;
    case 1: return w.y;
    case 2: return w.mask;
    case 3: return w.gy;
    case 4: return w.tgt;
    default: return (size_t)-1;
  }
}

size_t bdda_fno_offset(const bdda_fno_config* cfg, int what, int layer) {
  if (!cfg_ok(cfg)) return (size_t)-1;
  const FnoParams p = param_layout(to_cfg(cfg));
  if (layer < 0 || layer >= cfg->layers) layer = 0;
  switch (what) {
    case 0: return p.P;
    case 1: return p.p;
    case 2: return p.R[layer];
    case 3: return p.W[layer];
    case 4: return p.b[layer];
    case 5: return p.Q1;
    case 6: return p.q1;
    case 7: return p.Q2;
    case 8: return p.q2;
    default: return (size_t)-1;
  }
}

}  // extern "C"
