// One-CTA dense algebra on L x L complex matrices (L <= 64) in shared memory.
//
// These replace the reference's numpy.linalg calls on the small block
// matrices (bl_krylov/bl_krylov.py:92,101,104,113,167,184): LU with partial
// pivoting for solve(), and a Cholesky-based QR for qr().  All threads of
// the CTA must call each routine; matrices are row-major double2.
#pragma once
#include <cuda_runtime.h>

namespace bdda {

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zmulc(double2 a, double2 b) {   // conj(a) * b
  return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zdiv(double2 a, double2 b) {
  // Smith's algorithm
  if (fabs(b.x) >= fabs(b.y)) {
    const double r = b.y / b.x, d = b.x + r * b.y;
    return make_double2((a.x + a.y * r) / d, (a.y - a.x * r) / d);
  }
  const double r = b.x / b.y, d = b.y + r * b.x;
  return make_double2((a.x * r + a.y) / d, (a.y * r - a.x) / d);
}
__device__ __forceinline__ bool zfinite(double2 a) { return isfinite(a.x) && isfinite(a.y); }

__device__ __forceinline__ void block_copy(double2* dst, const double2* src, int n) {
  for (int e = threadIdx.x; e < n; e += blockDim.x) dst[e] = src[e];
}

// ---- L <= 32: elimination without divisions -----------------------------------------
// One dependent FP64 operation takes about 40 cycles here and a division ten
// times that, so a factorisation step is bound by the chain pivot search ->
// division -> scaling -> update, not by its arithmetic.  These routines
// eliminate without dividing: the rows below a pivot d become
// (d x - c u) 2^-e, 2^e the power of two above d.  That scales all remaining rows (and
// right-hand sides) by the same factor d 2^-e of modulus 0.5 to 1.4, so pivots are chosen as
// partial pivoting chooses them and the solution is the same; the only
// divisions, by the L pivots, run side by side before the back substitution.
// Rows are not moved: perm[k] is the pivot row of step k; every warp finds it
// by itself, so a step has one barrier.  Equal rows give an exactly zero row
// (both products are formed by the same operations), hence a singular matrix
// that LAPACK's LU finds singular by equal rows is found here too.
// bicg_alpha_kernel, B200: L = 10 24 -> 9 us, L = 32 90 -> 40 us.  Above 32
// columns the CTA-wide routines below are as good (their trailing updates
// outweigh the chain).
constexpr int kElimMax = 32;
__host__ __device__ constexpr int elim_pitch(int ncol) { return ncol | 1; }   // odd: column reads without bank conflicts

// 2^-(exponent + 1) of the larger component: the scaled value lies in [1/2, 1)
// in it, so the rows do not grow with the steps: entries up to about 1e304 at
// 32 columns (2^-exponent, values in [1, 2), overflowed there).
__device__ __forceinline__ double pow2_below(double2 d) {
  const int hx = __double2hiint(fabs(d.x)) >> 20, hy = __double2hiint(fabs(d.y)) >> 20;
  const int e = min(max(max(hx, hy), 1), 2044);
  return __hiloint2double((2045 - e) << 20, 0);
}
__device__ __forceinline__ double2 elim_mul(double2 a, double2 b) {   // the same operations for any operands
  return make_double2(fma(a.x, b.x, -__dmul_rn(a.y, b.y)), fma(a.x, b.y, __dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 elim_step(double2 ds, double2 x, double2 cs, double2 u) {
  const double2 p = elim_mul(ds, x), q = elim_mul(cs, u);
  return make_double2(__dsub_rn(p.x, q.x), __dsub_rn(p.y, q.y));
}

// w (L rows of `pitch`): A in the columns [0, L), ncol right-hand sides after
// it.  *bad as lu_factor's.
static __device__ void elim_factor(double2* w, int pitch, int L, int ncol, int* perm, int* bad) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned used = 0;
  for (int k = 0; k < L; ++k) {
    long long key = -1;   // |re| + |im| as an integer: non-negative doubles order as their bits
    if (lane < L && !((used >> lane) & 1)) {
      const double2 v = w[lane * pitch + k];
      key = __double_as_longlong(fabs(v.x) + fabs(v.y));
    }
    const int hi = (int)(key >> 32);
    const int mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = hi == mh ? (unsigned)key : 0u;
    const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
    const int p = __ffs(__ballot_sync(0xffffffffu, hi == mh && lo == ml)) - 1;
    if (threadIdx.x == 0) {
      const double best = __hiloint2double(mh, (int)ml);
      perm[k] = p;
      if (!isfinite(best)) *bad = 2;
      else if (!(best > 0.0) && *bad == 0) *bad = 1;
    }
    used |= 1u << p;
    const double2 d = w[p * pitch + k];
    const double s = pow2_below(d);
    const double2 ds = make_double2(d.x * s, d.y * s);
    for (int i = warp; i < L; i += nw) {
      if ((used >> i) & 1) continue;
      const double2 c = w[i * pitch + k];
      const double2 cs = make_double2(c.x * s, c.y * s);
      for (int j = k + 1 + lane; j < L + ncol; j += 32)
        w[i * pitch + j] = elim_step(ds, w[i * pitch + j], cs, w[p * pitch + j]);
    }
    __syncthreads();
  }
}

// The same steps on new right-hand sides (columns [L, L + ncol)) of a factored w.
static __device__ void elim_replay(double2* w, int pitch, int L, int ncol, const int* perm) {
  __shared__ int rank[kElimMax];
  if (threadIdx.x < L) rank[perm[threadIdx.x]] = threadIdx.x;
  __syncthreads();
  const int r = threadIdx.x & 7, per = blockDim.x >> 3;
  for (int c0 = 0; c0 < ncol; c0 += per) {
    const int c = L + c0 + (threadIdx.x >> 3);
    const bool on = c < L + ncol;
    for (int k = 0; k < L; ++k) {
      const int p = perm[k];
      const double2 d = w[p * pitch + k];
      const double s = pow2_below(d);
      const double2 ds = make_double2(d.x * s, d.y * s);
      if (on) {
        const double2 u = w[p * pitch + c];
        for (int i = r; i < L; i += 8)
          if (rank[i] > k) {
            const double2 v = w[i * pitch + k];
            w[i * pitch + c] = elim_step(ds, w[i * pitch + c], make_double2(v.x * s, v.y * s), u);
          }
      }
      __syncwarp();
    }
  }
  __syncthreads();
}

// Back substitution: unknown k of right-hand side c ends in row perm[k], column c.
static __device__ void elim_back(double2* w, int pitch, int L, int ncol, const int* perm) {
  __shared__ double2 inv[kElimMax];
  if (threadIdx.x < L) inv[threadIdx.x] = zdiv(make_double2(1.0, 0.0), w[perm[threadIdx.x] * pitch + threadIdx.x]);
  __syncthreads();
  const int r = threadIdx.x & 7, per = blockDim.x >> 3;
  for (int c0 = 0; c0 < ncol; c0 += per) {
    const int c = L + c0 + (threadIdx.x >> 3);
    const bool on = c < L + ncol;
    for (int k = L - 1; k >= 0; --k) {
      const int p = perm[k];
      double2 xk = make_double2(0.0, 0.0);
      if (on) xk = elim_mul(w[p * pitch + c], inv[k]);
      __syncwarp();
      if (on) {
        if (r == 0) w[p * pitch + c] = xk;
        for (int i = r; i < k; i += 8) {
          double2* x = w + perm[i] * pitch;
          x[c] = make_double2(fma(-x[k].x, xk.x, fma(x[k].y, xk.y, x[c].x)), fma(-x[k].x, xk.y, fma(-x[k].y, xk.x, x[c].y)));
        }
      }
      __syncwarp();
    }
  }
  __syncthreads();
}

// Hermitian positive definite g -> upper R with R^H R = g, and x <- R^-1 (both
// by rows, lower parts zero), L <= 32.  The same idea: the trailing matrix
// after step k is the Schur complement times c_k = prod d 2^-e, so
// R(k, j) = g(k, j) / sqrt(c_k d_k), all square roots and divisions at the end,
// side by side (cholqr_step_kernel, L = 8: 16 -> 6 us).
static __device__ void elim_chol_inv(double2* g, int L, double2* x, int* bad) {
  __shared__ double dk[kElimMax], ck[kElimMax], rs[kElimMax];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double c = 1.0;
  for (int k = 0; k < L; ++k) {
    const double d = g[k * L + k].x;
    const double s = pow2_below(make_double2(d, 0.0)), ds = d * s;
    if (threadIdx.x == 0) {
      if (!isfinite(d)) *bad = 2;
      else if (!(d > 0.0) && *bad == 0) *bad = 1;
      dk[k] = d;
      ck[k] = c;
    }
    c *= ds;
    for (int i = k + 1 + warp; i < L; i += nw) {
      const double2 v = g[k * L + i];
      const double2 u = make_double2(v.x * s, v.y * s);
      const int j = k + 1 + lane;
      if (j >= i && j < L) {
        const double2 t = zmulc(u, g[k * L + j]);
        g[i * L + j] = make_double2(ds * g[i * L + j].x - t.x, ds * g[i * L + j].y - t.y);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x < L) rs[threadIdx.x] = 1.0 / sqrt(fmax(ck[threadIdx.x] * dk[threadIdx.x], 0.0));
  __syncthreads();
  for (int e = threadIdx.x; e < L * L; e += blockDim.x) {
    const int i = e / L, j = e - i * L;
    const double2 v = g[e];
    g[e] = i < j ? make_double2(v.x * rs[i], v.y * rs[i]) : make_double2(i == j ? dk[i] * rs[i] : 0.0, 0.0);
    x[e] = make_double2(i == j ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  const int r = threadIdx.x & 7;
  const int col = threadIdx.x >> 3;
  for (int k = L - 1; k >= 0; --k) {   // 1 / R(k, k) = c_k / sqrt(c_k d_k)
    double2 xk = make_double2(0.0, 0.0);
    if (col < L) {
      const double q = ck[k] * rs[k];
      xk = x[k * L + col];
      xk = make_double2(xk.x * q, xk.y * q);
    }
    __syncwarp();
    if (col < L) {
      if (r == 0) x[k * L + col] = xk;
      for (int i = r; i < k; i += 8) x[i * L + col] = zsub(x[i * L + col], zmul(g[i * L + k], xk));
    }
    __syncwarp();
  }
  __syncthreads();
}

// w <- A (L x L) and B (L x ncol) side by side, B scaled by sign
__device__ __forceinline__ void elim_load(double2* w, int pitch, const double2* a, const double2* b, int L, double sign) {
  for (int e = threadIdx.x; e < L * L; e += blockDim.x) {
    const int i = e / L, j = e - i * L;
    w[i * pitch + j] = a[e];
    w[i * pitch + L + j] = make_double2(sign * b[e].x, sign * b[e].y);
  }
}

// out (L x L, by rows) <- A^-1 B, L <= 32, in w (L rows of elim_pitch(2 L));
// all threads; the result is visible to the CTA after a barrier
static __device__ void elim_solve(double2* w, const double2* a, const double2* b, int L, int* perm, int* bad,
                                  double2* out) {
  const int pitch = elim_pitch(2 * L);
  elim_load(w, pitch, a, b, L, 1.0);
  __syncthreads();
  elim_factor(w, pitch, L, L, perm, bad);
  elim_back(w, pitch, L, L, perm);
  for (int e = threadIdx.x; e < L * L; e += blockDim.x) {
    const int i = e / L, j = e - i * L;
    out[e] = w[perm[i] * pitch + L + j];
  }
}

// dynamic shared memory of the small kernels, in double2: two or three
// matrices, with the padding of an elimination's rows
__host__ __device__ constexpr int small_elems(int L, int mats) { return mats * L * L + L; }

// In-place LU with partial pivoting (row interchanges recorded in piv, in
// order).  Pivot choice as LAPACK's izamax: largest |re| + |im|, first on
// ties.  *bad becomes 1 for an exactly zero pivot (singular) and 2 for a
// non-finite one (the matrix holds NaN/Inf).
static __device__ void lu_factor(double2* a, int L, int* piv, int* bad) {
  __shared__ double sbest[32];
  __shared__ int sidx[32];
  for (int k = 0; k < L; ++k) {
    if (threadIdx.x < 32) {
      double best = -1.0;
      int bi = k;
      for (int i = k + threadIdx.x; i < L; i += 32) {
        const double2 v = a[i * L + k];
        const double m = fabs(v.x) + fabs(v.y);
        if (m > best || (m != m)) { best = (m != m) ? INFINITY : m; bi = i; }
      }
      sbest[threadIdx.x] = best;
      sidx[threadIdx.x] = bi;
      __syncwarp();
      if (threadIdx.x == 0) {
        double b = -1.0;
        int id = k;
        for (int w = 0; w < 32; ++w)
          if (sbest[w] > b || (sbest[w] == b && sidx[w] < id)) { b = sbest[w]; id = sidx[w]; }
        piv[k] = id;
        if (!isfinite(b)) *bad = 2;
        else if (!(b > 0.0) && *bad == 0) *bad = 1;
      }
    }
    __syncthreads();
    const int p = piv[k];
    if (p != k)
      for (int j = threadIdx.x; j < L; j += blockDim.x) {
        const double2 t = a[k * L + j];
        a[k * L + j] = a[p * L + j];
        a[p * L + j] = t;
      }
    __syncthreads();
    const double2 d = a[k * L + k];
    if (!(*bad))
      for (int i = k + 1 + threadIdx.x; i < L; i += blockDim.x) a[i * L + k] = zdiv(a[i * L + k], d);
    __syncthreads();
    const int m = L - k - 1;
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
      const int i = k + 1 + e / m, j = k + 1 + e % m;
      a[i * L + j] = zsub(a[i * L + j], zmul(a[i * L + k], a[k * L + j]));
    }
    __syncthreads();
  }
}

// b (L x ncol) <- A^-1 b from lu_factor's output
static __device__ void lu_solve(const double2* lu, const int* piv, int L, double2* b, int ncol) {
  for (int k = 0; k < L; ++k) {
    const int p = piv[k];
    if (p != k)
      for (int j = threadIdx.x; j < ncol; j += blockDim.x) {
        const double2 t = b[k * ncol + j];
        b[k * ncol + j] = b[p * ncol + j];
        b[p * ncol + j] = t;
      }
    __syncthreads();
  }
  for (int k = 0; k < L; ++k) {            // unit lower
    const int m = L - k - 1;
    for (int e = threadIdx.x; e < m * ncol; e += blockDim.x) {
      const int i = k + 1 + e / ncol, j = e % ncol;
      b[i * ncol + j] = zsub(b[i * ncol + j], zmul(lu[i * L + k], b[k * ncol + j]));
    }
    __syncthreads();
  }
  for (int k = L - 1; k >= 0; --k) {       // upper
    const double2 d = lu[k * L + k];
    for (int j = threadIdx.x; j < ncol; j += blockDim.x) b[k * ncol + j] = zdiv(b[k * ncol + j], d);
    __syncthreads();
    for (int e = threadIdx.x; e < k * ncol; e += blockDim.x) {
      const int i = e / ncol, j = e % ncol;
      b[i * ncol + j] = zsub(b[i * ncol + j], zmul(lu[i * L + k], b[k * ncol + j]));
    }
    __syncthreads();
  }
}

// Hermitian positive definite g -> upper R with R^H R = g (lower part zeroed).
static __device__ void chol_upper(double2* g, int L, int* bad) {
  for (int k = 0; k < L; ++k) {
    if (threadIdx.x == 0) {
      const double d = g[k * L + k].x;
      if (!isfinite(d)) *bad = 2;
      else if (!(d > 0.0) && *bad == 0) *bad = 1;
      g[k * L + k] = make_double2(sqrt(fmax(d, 0.0)), 0.0);
    }
    __syncthreads();
    const double rkk = g[k * L + k].x;
    if (!(*bad))
      for (int j = k + 1 + threadIdx.x; j < L; j += blockDim.x)
        g[k * L + j] = make_double2(g[k * L + j].x / rkk, g[k * L + j].y / rkk);
    __syncthreads();
    const int m = L - k - 1;
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
      const int i = k + 1 + e / m, j = k + 1 + e % m;
      if (j >= i) g[i * L + j] = zsub(g[i * L + j], zmulc(g[k * L + i], g[k * L + j]));
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < L * L; e += blockDim.x)
    if (e / L > e % L) g[e] = make_double2(0.0, 0.0);
  __syncthreads();
}

// x <- R^-1 for upper-triangular R (x must not alias r)
static __device__ void tri_upper_inv(const double2* r, int L, double2* x) {
  for (int e = threadIdx.x; e < L * L; e += blockDim.x)
    x[e] = make_double2((e / L == e % L) ? 1.0 : 0.0, 0.0);
  __syncthreads();
  for (int k = L - 1; k >= 0; --k) {
    const double2 d = r[k * L + k];
    for (int j = threadIdx.x; j < L; j += blockDim.x) x[k * L + j] = zdiv(x[k * L + j], d);
    __syncthreads();
    for (int e = threadIdx.x; e < k * L; e += blockDim.x) {
      const int i = e / L, j = e % L;
      x[i * L + j] = zsub(x[i * L + j], zmul(r[i * L + k], x[k * L + j]));
    }
    __syncthreads();
  }
}

// c = op(a) b with op = transpose (TA) or identity; c must not alias a or b
template <bool TA>
static __device__ void small_matmul(const double2* a, const double2* b, double2* c, int L) {
  for (int e = threadIdx.x; e < L * L; e += blockDim.x) {
    const int i = e / L, j = e % L;
    double2 s = make_double2(0.0, 0.0);
    for (int m = 0; m < L; ++m) s = zadd(s, zmul(TA ? a[m * L + i] : a[i * L + m], b[m * L + j]));
    c[e] = s;
  }
  __syncthreads();
}

}  // namespace bdda
