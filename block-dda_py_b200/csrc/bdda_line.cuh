// Pencil passes of one axis length M = A * B in two register stages, with the
// half of the pencil that is structurally zero (or cropped) left out.
//
// On the doubled grid at most M / 2 rows of a pencil hold data: a forward pass
// reads rows below n_in <= M / 2, an inverse pass writes rows below
// n_out <= M / 2.  With A even, A = 2 H, j < B, q < H, k = 2 k' + h:
//   X[k + A k2] = sum_j w_B^(j k2) w_M^(j k) sum_{q<H} (x[j + B q] w_A^(q h)) w_H^(q k')
// so stage 1 is two H-point transforms of the same H values (even and odd
// k), not an A-point one of which half the inputs are zero; stage 2 is a
// B-point transform.  The inverse runs the same steps backwards and adds the
// two halves.  Against the plan's radix sequence (three or four stages of
// radix <= 10, run-time strides in the generic kernel) that is one
// shared-memory round trip instead of two or three, no zero row loaded or
// multiplied, and every index division by a constant.
//
// Spectra stay in the plan's digit-reversed order in HBM: row and Green's
// entries are addressed through the plan's frequency -> position table.
//
// Columns.  The Z and Y passes act on every column of a row alone, so their
// tiles are W consecutive entries of the flattened (p1, column) index: a block
// width L that is odd or below the tile width wastes nothing.  The X pass couples
// the three components: its tile is R right-hand sides of one pencil, or,
// when L < R, the L right-hand sides of R / L neighbouring pencils.
//
// Bound.  Z and Y passes: memory latency, hence small tiles, one job per
// thread, as many CTAs as the registers allow (4.2-6.1 of the 6.56 TB/s copy
// rate in complex128).  X pass in complex128: the FP64 pipe (66 instructions a
// grid value at 90 points, 56 % of its peak by the counters): a CTA works through
// the column tiles of one pencil with the pencil's Green's entries staged once in
// shared memory, and asks for the next tile's rows before it computes.  In
// complex64: issue (69 % of the slots at 192 points) and shared memory (52 % of its
// wavefronts).  One product on a B200, the
// run-time-radix kernels -> these (time of the bytes at the copy rate):
//   17 x 17 x 17    L = 10  complex128   105 -> 45 us     (11)
//   52 x 60 x 71    L = 1   complex128   534 -> 141 us    (71)
//   61 x 47 x 85    L = 11  complex128  2.25 -> 1.08 ms   (0.58)
//   45 x 55 x 83    L = 32  complex128  3.82 -> 1.97 ms   (1.28)
//                           complex64   2.53 -> 1.17 ms   (0.64)
//   105 x 98 x 92   L = 60  complex128  34.8 -> 20.4 ms   (11.1)
//   93 x 112 x 174  L = 64  complex64   28.2 -> 20.3 ms   (11.0; the first
//                           kernels specialised for its radices before)
#pragma once
#include <atomic>

#include "bdda_fixed.cuh"

namespace bdda {

// ---- length -> split, tile width, threads: the same rules for every length ------
constexpr bool line_radix(int r) {
  return (r >= 2 && r <= 10) || r == 12 || r == 14 || r == 15 || r == 16 || r == 18 || r == 20 || r == 21 || r == 25;
}
// stage-1 half radices: H-point transforms of 2 H outputs
constexpr bool line_half(int h) { return (h >= 1 && h <= 10) || h == 12 || h == 14 || h == 15 || h == 16; }

// Forward / inverse passes: the most balanced split (the smaller the larger
// factor, the fewer registers a job holds), A even; ties to the larger A,
// whose stage holds H inputs at a time.  0: no split.
constexpr int line_split(int M) {
  int best = 0, key = 1 << 30;
  for (int A = 2; A <= 32; A += 2) {
    if (M % A || !line_half(A / 2)) continue;
    const int B = M / A;
    if (B < 2 || !line_radix(B)) continue;
    const int k = 2 * (A > B ? A : B) - (A > B ? 1 : 0);
    if (k < key) { key = k; best = A; }
  }
  return best;
}
// X pass: a middle job holds 3 B frequencies, so B weighs 2.5 times, and is
// at most 10.
constexpr int conv_split(int M) {
  int best = 0, key = 1 << 30;
  for (int A = 2; A <= 32; A += 2) {
    if (M % A || !line_half(A / 2)) continue;
    const int B = M / A;
    if (B < 2 || B > 10) continue;
    const int k = 2 * A > 5 * B ? 2 * A : 5 * B;
    if (k < key) { key = k; best = A; }
  }
  return best;
}

// Threads per CTA: the multiple of 32 from `least` to 256 whose rounds of jobs
// (n1 of A-point work, n2 of B-point work) leave the fewest lanes idle; ties
// to the larger, whose loads are all in flight at once.
constexpr int line_threads(int n1, int a, int n2, int b, int least) {
  int best = 256, key = 1 << 30;
  for (int nt = 256; nt >= 64; nt -= 32) {
    if (nt < least) break;
    const int spent = ((n1 + nt - 1) / nt) * nt * a + ((n2 + nt - 1) / nt) * nt * b;
    if (spent < key) { key = spent; best = nt; }
  }
  return best;
}
constexpr int at_least(int x, int lo) { return x < lo ? lo : x; }

// Forward and inverse passes are bound by memory latency, so tiles are small
// (W columns: 128-byte rows) and CTAs many.  An inverse pass keeps one stage-2
// job per thread where that takes at most 256, so that its epilogue's operands
// can be fetched ahead.
template <typename T, int M, int KIND> struct LineShape {
  static constexpr int A = line_split(M), B = A ? M / A : 2, H = A / 2;
  static constexpr int W = 128 / (int)sizeof(T);
  static constexpr int NT = A ? line_threads(B * W, A, A * W, B, KIND == K_INV && B * W <= 256 ? B * W : 64) : 128;
  static constexpr int wide = B > A ? B : A;
  static constexpr int regs = sizeof(T) == 8 ? (wide <= 16 ? 64 : 80) : wide <= 12 ? 80 : wide <= 16 ? 100 : 128;
  static constexpr int smem = M * W * (int)sizeof(T) + M * (int)sizeof(T) + 2 * M;
  static constexpr int by_regs = 65536 / (NT * regs), by_smem = 227 * 1024 / (smem + 1024);
  static constexpr int MINB = at_least(by_regs < by_smem ? by_regs : by_smem, 1);
};
// X pass.  A middle job holds 3 B complex values, so few CTAs fit the
// register file, and what a CTA waits for (its loads, the barriers between its
// stages) has to be covered by the others: as many CTAs as shared memory and
// the jobs' registers allow.  55 of the 200 kernels spill to get there, most of them
// 20 bytes a thread or less (the most, 168, complex64 at 200 points).
template <typename T, int M> struct ConvShape {
  static constexpr int A = conv_split(M), B = A ? M / A : 0, H = A / 2;
  static constexpr bool C128 = sizeof(T) == 16;
  static constexpr int per_row = 31 * (int)sizeof(T);   // tile of 24 columns, Green's entries, twiddle
  static constexpr bool small = M * per_row <= (C128 ? 75 : 38) * 1024 && B <= 7;
  static constexpr bool big = M * per_row > (C128 ? 113 : 56) * 1024;
  static constexpr int R = C128 && big ? 4 : 8;          // right-hand sides per tile (three columns each)
  static constexpr int NT = small || (C128 && big) ? 128 : big ? 256 : 192;
  static constexpr int MINB = small ? (C128 ? 3 : 5) : C128 || big ? 2 : 4;
};

// ---- register transforms ------------------------------------------------------------
template <int R, bool INV, typename T> __device__ __forceinline__ void line_dft(T* v);

// Good-Thomas on registers for coprime A, B: with n = B n1 + A n2 (mod R) and
// k = k1 (mod A) = k2 (mod B), w_R^(nk) = w_A^(n1 k1) w_B^(n2 k2), so the A- and
// B-point transforms need no twiddles between them; both index maps are
// compile-time register permutations.
template <int A, int B, bool INV, typename T> __device__ __forceinline__ void dft_pfa(T* v) {
  constexpr int R = A * B;
  T u[R];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
    T t[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) t[n1] = v[(B * n1 + A * n2) % R];
    line_dft<A, INV>(t);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) u[k1 * B + n2] = t[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    T t[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) t[n2] = u[k1 * B + n2];
    line_dft<B, INV>(t);
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (k % A == k1) v[k] = t[k % B];
  }
}

template <int R, bool INV, typename T> __device__ __forceinline__ void line_dft(T* v) {
  if constexpr (R == 1) return;
  else if constexpr (R == 6) dft_pfa<2, 3, INV>(v);
  else if constexpr (R == 10) dft_pfa<2, 5, INV>(v);
  else if constexpr (R == 12) dft_pfa<4, 3, INV>(v);
  else if constexpr (R == 14) dft_pfa<2, 7, INV>(v);
  else if constexpr (R == 15) dft_pfa<3, 5, INV>(v);
  else if constexpr (R == 18) dft_pfa<2, 9, INV>(v);
  else if constexpr (R == 20) dft_pfa<4, 5, INV>(v);
  else if constexpr (R == 21) dft_pfa<3, 7, INV>(v);
  else if constexpr (R == 25) dft_ab<5, 5, INV>(v);
  else dft<R, INV>(v);
}

// Fields a pass reads beyond PassArgs.
struct LineArgs {
  PassArgs p;
  int ncol;                 // line passes: flattened columns P1 * C
  // X pass: right-hand sides per tile of one pencil, pencils per tile, tiles per
  // pencil, tiles a CTA works through, CTAs per pencil
  int lt, pp, ltile, per, split;
  int tiles;                // CTAs per p0
};

__device__ __forceinline__ int line_comp(int c, int L) { return (c >= L) + (c >= 2 * L); }

// x[q] *= w_A^q (conj for the inverse), q < H: constants after unrolling
template <int A, bool INV, typename T> __device__ __forceinline__ void half_twiddle(T* x) {
#pragma unroll
  for (int q = 1; q < A / 2; ++q) x[q] = twiddle_const<A, INV>(x[q], q);
}

// a b + c, four fused operations
__device__ __forceinline__ double2 line_fma(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ float2 line_fma(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}

template <typename T> __device__ __forceinline__ T czero() { return mkc<T>(0, 0); }

// ---- forward / inverse pass --------------------------------------------------------
// FULL: the forward pass of a pencil with data in its upper half too, the images
// of the rows below (the Green's tensor; PassArgs.mirror): the even half
// transforms x[q] + x[q + H], the odd one their difference.
template <typename T, int KIND, int M, bool FULL>
__global__ void __launch_bounds__(LineShape<T, M, KIND>::NT, LineShape<T, M, KIND>::MINB) line_kernel(const __grid_constant__ LineArgs la) {
  typedef LineShape<T, M, KIND> S;
  constexpr int A = S::A, B = S::B, H = S::H, W = S::W, NT = S::NT;
  const PassArgs& a = la.p;
  if (a.live && *a.live == 0) return;
  extern __shared__ __align__(128) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);              // [M][W]
  T* tw = sm + M * W;                               // [M]
  uint16_t* pos = reinterpret_cast<uint16_t*>(tw + M);
  for (int i = threadIdx.x; i < M; i += NT) {
    tw[i] = static_cast<const T*>(a.tw)[i];
    pos[i] = a.pos[i];
  }
  const int tile = blockIdx.x % la.tiles, p0 = blockIdx.x / la.tiles;
  const int C = (int)a.C;
  // this thread's column: the same in every round (W divides NT)
  static_assert(NT % W == 0, "a thread keeps its column");
  const int s = threadIdx.x % W;
  const int g = tile * W + s;
  const bool col = g < la.ncol;
  const int p1 = col ? g / C : 0, c = col ? g - p1 * C : 0;
  const T* src = static_cast<const T*>(a.src) + p0 * a.src_p0 + p1 * a.src_p1 + c;
  T* dst = static_cast<T*>(a.dst) + p0 * a.dst_p0 + p1 * a.dst_p1 + c;
  const int32_t* cmap = a.cell_map ? a.cell_map + p0 * a.cell_p0 + p1 * a.cell_p1 : nullptr;
  if constexpr (KIND == K_FWD) {
    __syncthreads();   // tw, pos
#pragma unroll 1
    for (int j = threadIdx.x / W; j < B; j += NT / W) {
      T x[H], t[H];
      if constexpr (!FULL) {
        if (cmap) {
          int m[H];
#pragma unroll
          for (int q = 0; q < H; ++q) m[q] = col && j + B * q < a.n_in ? cmap[j + B * q] : -1;
#pragma unroll
          for (int q = 0; q < H; ++q) {
            x[q] = czero<T>();
            if (m[q] >= 0) {
              const int64_t i = (int64_t)m[q] * C + c;
              if constexpr (std::is_same<T, float2>::value) x[q] = a.wide ? narrow_at(a.S, i) : static_cast<const T*>(a.S)[i];
              else x[q] = static_cast<const T*>(a.S)[i];
            }
          }
        } else {
#pragma unroll
          for (int q = 0; q < H; ++q)
            x[q] = col && j + B * q < a.n_in ? src[(int64_t)(j + B * q) * a.src_row] : czero<T>();
        }
#pragma unroll
        for (int q = 0; q < H; ++q) t[q] = x[q];
      } else {
#pragma unroll
        for (int q = 0; q < H; ++q) {
          // row r, and row r + M / 2, the image of row M / 2 - r
          const int r = j + B * q, i = M / 2 - r;
          const T lo = col && r < a.n_in ? src[(int64_t)r * a.src_row] : czero<T>();
          T hi = col && i < a.n_in ? src[(int64_t)i * a.src_row] : czero<T>();
          if ((a.mirror >> c) & 1) {
            hi.x = -hi.x;
            hi.y = -hi.y;
          }
          t[q] = cadd(lo, hi);
          x[q] = csub(lo, hi);
        }
      }
      line_dft<H, false>(t);
      sm[j * W + s] = t[0];
#pragma unroll
      for (int k = 1; k < H; ++k) sm[(j + B * 2 * k) * W + s] = cmul(t[k], tw[j * 2 * k]);
      half_twiddle<A, false>(x);
      line_dft<H, false>(x);
#pragma unroll
      for (int k = 0; k < H; ++k) sm[(j + B * (2 * k + 1)) * W + s] = cmul(x[k], tw[j * (2 * k + 1)]);
    }
    __syncthreads();
#pragma unroll 1
    for (int k = threadIdx.x / W; k < A; k += NT / W) {
      T v[B];
#pragma unroll
      for (int j = 0; j < B; ++j) v[j] = sm[(j + B * k) * W + s];
      line_dft<B, false>(v);
      if (col) {
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) dst[(int64_t)pos[k + A * k2] * a.dst_row] = v[k2];
      }
    }
  } else {
    // The epilogue's dipole numbers, and the lines of S it will read, are
    // fetched first: they arrive while the transforms run.
    constexpr bool once = B * W <= NT;   // one stage-2 job per thread
    int m[H];
    if (once && cmap) {
      const int j = threadIdx.x / W;
#pragma unroll
      for (int q = 0; q < H; ++q) m[q] = col && j < B && j + B * q < a.n_out ? cmap[j + B * q] : -1;
    }
    __syncthreads();
#pragma unroll 1
    for (int k = threadIdx.x / W; k < A; k += NT / W) {
      T v[B];
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k2] = col ? src[(int64_t)pos[k + A * k2] * a.src_row] : czero<T>();
      line_dft<B, true>(v);
      sm[B * k * W + s] = v[0];
#pragma unroll
      for (int j = 1; j < B; ++j) sm[(j + B * k) * W + s] = cmulc(v[j], tw[j * k]);
    }
    if (once && cmap) {
      const char* sp = static_cast<const char*>(a.S) + c * (a.wide ? 16 : (int)sizeof(T));
#pragma unroll
      for (int q = 0; q < H; ++q)
        if (m[q] >= 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(sp + (int64_t)m[q] * C * (a.wide ? 16 : (int)sizeof(T))));
    }
    __syncthreads();
    typedef typename real_of<T>::type F;
    const F sc = F(a.scale);
    const int L = a.L;
#pragma unroll 1
    for (int j = threadIdx.x / W; j < B; j += NT / W) {
      if (!once && cmap) {
#pragma unroll
        for (int q = 0; q < H; ++q) m[q] = col && j + B * q < a.n_out ? cmap[j + B * q] : -1;
      }
      T e[H], o[H];
#pragma unroll
      for (int k = 0; k < H; ++k) e[k] = sm[(j + B * 2 * k) * W + s];
      line_dft<H, true>(e);
#pragma unroll
      for (int k = 0; k < H; ++k) o[k] = sm[(j + B * (2 * k + 1)) * W + s];
      line_dft<H, true>(o);
      half_twiddle<A, true>(o);
#pragma unroll
      for (int q = 0; q < H; ++q) e[q] = cscale(cadd(e[q], o[q]), sc);
      if (cmap) {   // crop + gather + diagonal + Jacobi: (diag S + y) jpre (bl_krylov.py:55)
        const int comp = line_comp(c, L);
#pragma unroll
        for (int q = 0; q < H; ++q) {
          if (m[q] >= 0) {
            const int64_t r3 = 3 * (int64_t)m[q] + comp, i = (int64_t)m[q] * C + c;
            const T d = static_cast<const T*>(a.diag)[r3], jp = static_cast<const T*>(a.jpre)[r3];
            if constexpr (std::is_same<T, float2>::value) {
              if (a.wide) {
                widen_to(a.dst, i, cmul(cadd(cmul(d, narrow_at(a.S, i)), e[q]), jp));
                continue;
              }
            }
            static_cast<T*>(a.dst)[i] = cmul(cadd(cmul(d, static_cast<const T*>(a.S)[i]), e[q]), jp);
          }
        }
      } else if (col) {
#pragma unroll
        for (int q = 0; q < H; ++q)
          if (j + B * q < a.n_out) dst[(int64_t)(j + B * q) * a.dst_row] = e[q];
      }
    }
  }
}

// ---- X pass -------------------------------------------------------------------------
// GS: the pencil's Green's entries are staged in shared memory, in natural
// frequency order (tiles of one pencil); otherwise the middle reads them from
// global memory, each entry once per tile.
template <typename T, int M, bool GS>
__global__ void __launch_bounds__(ConvShape<T, M>::NT, ConvShape<T, M>::MINB) conv_kernel(const __grid_constant__ LineArgs la) {
  typedef ConvShape<T, M> S;
  constexpr int A = S::A, B = S::B, H = S::H, R = S::R, W = 3 * R, NT = S::NT;
  const PassArgs& a = la.p;
  if (a.live && *a.live == 0) return;
  extern __shared__ __align__(128) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);               // [M][W], column comp * R + r
  T* tw = sm + M * W;                                // [M]
  uint16_t* pos = reinterpret_cast<uint16_t*>(tw + M);
  int* off = reinterpret_cast<int*>(pos + (M + 7) / 8 * 8);   // [R]: offset of right-hand side r's x component
  T* gs = reinterpret_cast<T*>(off + 8);                      // [M][6] (GS)
  const int item = blockIdx.x % la.tiles, p0 = blockIdx.x / la.tiles;
  const int lt = la.lt, L = a.L, C = (int)a.C;
  // right-hand side r of a tile: pencil p1 + r / lt, column l0 + r % lt
  const int p1 = la.pp > 1 ? item * la.pp : item / la.split;
  const int t0 = la.pp > 1 ? 0 : (item - p1 * la.split) * la.per, t1 = min(la.ltile, t0 + la.per);
  if (threadIdx.x < R) {
    const int r = threadIdx.x;
    off[r] = r / lt * C + r % lt;
  }
  const int64_t base = p0 * a.src_p0 + (int64_t)p1 * a.src_p1;   // src_p1 = dst_p1 = C
  const T* gh = static_cast<const T*>(a.ghat) + ((int64_t)p0 * a.P1 + p1) * (M * 6);
  if constexpr (GS) {
    constexpr int CH = 6 * (int)sizeof(T) / 16;   // 16-byte chunks per frequency
    for (int i = threadIdx.x; i < M * CH; i += NT) {
      const int f = i / CH, part = i - f * CH;
      cp_async16(reinterpret_cast<char*>(gs + f * 6) + 16 * part,
                 reinterpret_cast<const char*>(gh + a.pos[f] * 6) + 16 * part);
    }
    cp_async_commit();
  }
  for (int i = threadIdx.x; i < M; i += NT) {
    tw[i] = static_cast<const T*>(a.tw)[i];
    if constexpr (!GS) pos[i] = a.pos[i];
  }
  for (int tile = t0; tile < t1; ++tile) {
  const int l0 = tile * lt;
  const int nr = la.pp > 1 ? min(la.pp, a.P1 - p1) * lt : min(lt, L - l0);
  const float by_nr = 1.f / nr;   // (int)((x + 0.5f) * by_nr) = x / nr for the job counts here (x < 2^12)
  const T* src = static_cast<const T*>(a.src) + base + l0;
  T* dst = static_cast<T*>(a.dst) + base + l0;
  if (tile + 1 < t1) {   // the next tile's rows into L2 while this one computes
    for (int i = threadIdx.x; i < 3 * a.n_in; i += NT) {
      const int row = i / 3, comp = i - 3 * row;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(src + (int64_t)row * a.src_row + comp * L + lt));
    }
  }
  __syncthreads();
  // stage 1, forward
#pragma unroll 1
  for (int job = threadIdx.x; job < 3 * B * nr; job += NT) {
    const int t3 = (int)((job + 0.5f) * by_nr), j = t3 / 3, comp = t3 - 3 * j, r = job - t3 * nr, s = comp * R + r;
    const T* p = src + (off[r] + comp * L);
    T x[H], t[H];
#pragma unroll
    for (int q = 0; q < H; ++q) x[q] = j + B * q < a.n_in ? p[(int64_t)(j + B * q) * a.src_row] : czero<T>();
#pragma unroll
    for (int q = 0; q < H; ++q) t[q] = x[q];
    line_dft<H, false>(t);
    sm[j * W + s] = t[0];
#pragma unroll
    for (int k = 1; k < H; ++k) sm[(j + B * 2 * k) * W + s] = cmul(t[k], tw[j * 2 * k]);
    half_twiddle<A, false>(x);
    line_dft<H, false>(x);
#pragma unroll
    for (int k = 0; k < H; ++k) sm[(j + B * (2 * k + 1)) * W + s] = cmul(x[k], tw[j * (2 * k + 1)]);
  }
  if constexpr (GS) cp_async_wait<0>();
  __syncthreads();
  // middle: B-point transforms of the three components, the Green multiply, back
#pragma unroll 1
  for (int job = threadIdx.x; job < A * nr; job += NT) {
    const int k = (int)((job + 0.5f) * by_nr), r = job - k * nr;
    const T* gp = gh + (int64_t)(la.pp > 1 ? r / lt : 0) * (M * 6);
    T y[3][B];
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
#pragma unroll
      for (int j = 0; j < B; ++j) y[comp][j] = sm[(j + B * k) * W + comp * R + r];
      line_dft<B, false>(y[comp]);
    }
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) {
      const T* g = GS ? gs + (k + A * k2) * 6 : gp + pos[k + A * k2] * 6;
      T gv[6];
      if constexpr (GS) {
#pragma unroll
        for (int i = 0; i < 6; ++i) gv[i] = g[i];
      } else if constexpr (std::is_same<T, float2>::value) {
        const float4* g4 = reinterpret_cast<const float4*>(g);
        const float4 u = __ldg(g4), v = __ldg(g4 + 1), w = __ldg(g4 + 2);
        gv[0] = lo2(u); gv[1] = hi2(u); gv[2] = lo2(v); gv[3] = hi2(v); gv[4] = lo2(w); gv[5] = hi2(w);
      } else {
#pragma unroll
        for (int i = 0; i < 6; ++i) gv[i] = __ldg(g + i);
      }
      const T v0 = y[0][k2], v1 = y[1][k2], v2 = y[2][k2];
      y[0][k2] = line_fma(gv[0], v0, line_fma(gv[1], v1, cmul(gv[2], v2)));
      y[1][k2] = line_fma(gv[1], v0, line_fma(gv[3], v1, cmul(gv[4], v2)));
      y[2][k2] = line_fma(gv[2], v0, line_fma(gv[4], v1, cmul(gv[5], v2)));
    }
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
      line_dft<B, true>(y[comp]);
#pragma unroll
      for (int j = 0; j < B; ++j) sm[(j + B * k) * W + comp * R + r] = y[comp][j];
    }
  }
  __syncthreads();
  // stage 1, inverse: rows below n_out
#pragma unroll 1
  for (int job = threadIdx.x; job < 3 * B * nr; job += NT) {
    const int t3 = (int)((job + 0.5f) * by_nr), j = t3 / 3, comp = t3 - 3 * j, r = job - t3 * nr, s = comp * R + r;
    T* p = dst + (off[r] + comp * L);
    T e[H], o[H];
    e[0] = sm[j * W + s];
#pragma unroll
    for (int k = 1; k < H; ++k) e[k] = cmulc(sm[(j + B * 2 * k) * W + s], tw[j * 2 * k]);
    line_dft<H, true>(e);
#pragma unroll
    for (int k = 0; k < H; ++k) o[k] = cmulc(sm[(j + B * (2 * k + 1)) * W + s], tw[j * (2 * k + 1)]);
    line_dft<H, true>(o);
    half_twiddle<A, true>(o);
#pragma unroll
    for (int q = 0; q < H; ++q)
      if (j + B * q < a.n_out) p[(int64_t)(j + B * q) * a.dst_row] = cadd(e[q], o[q]);
  }
  }
}

// ---- launch ---------------------------------------------------------------------------
// Raises a kernel's dynamic shared-memory limit once per device (the
// attribute is per function and device; repeating it is harmless).
template <typename K> int line_smem_limit(K kern, size_t smem, std::atomic<uint64_t>& done) {
  int dev = 0;
  BDDA_CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
  if (!bit || !(done.load(std::memory_order_acquire) & bit)) {
    BDDA_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    done.fetch_or(bit, std::memory_order_release);
  }
  return BDDA_OK;
}

template <typename T, int KIND, int M, bool FULL>
int line_launch(const PassArgs& a, int64_t P0, cudaStream_t st) {
  typedef LineShape<T, M, KIND> S;
  static std::atomic<uint64_t> done{0};
  LineArgs la;
  la.p = a;
  const int64_t ncol = (int64_t)a.P1 * a.C;
  if (ncol > 0x7fffffff) return BDDA_BAD_ARG;
  la.ncol = (int)ncol;
  la.lt = la.pp = la.ltile = la.per = la.split = 0;
  la.tiles = (la.ncol + S::W - 1) / S::W;
  const int64_t nblk = P0 * la.tiles;
  if (nblk <= 0) return BDDA_OK;
  if (nblk > 0x7fffffff) return BDDA_BAD_ARG;
  const size_t smem = S::smem;
  auto kern = line_kernel<T, KIND, M, FULL>;
  const int s = line_smem_limit(kern, smem, done);
  if (s != BDDA_OK) return s;
  kern<<<(unsigned)nblk, S::NT, smem, st>>>(la);
  BDDA_CUDA_TRY(cudaGetLastError());
  count_launch();
  return BDDA_OK;
}

template <typename T, int M>
int conv_launch(const PassArgs& a, int64_t P0, cudaStream_t st) {
  typedef ConvShape<T, M> S;
  static std::atomic<uint64_t> done[2];
  LineArgs la;
  la.p = a;
  la.ncol = 0;
  if (a.L >= S::R) {   // near-equal column tiles of one pencil
    la.pp = 1;
    la.ltile = (a.L + S::R - 1) / S::R;
    la.lt = (a.L + la.ltile - 1) / la.ltile;
  } else {             // every column of R / L pencils
    la.pp = S::R / a.L;
    la.ltile = 1;
    la.lt = a.L;
  }
  la.per = la.ltile;
  while (la.per > 1 && P0 * a.P1 * ((la.ltile + la.per - 1) / la.per) < 148 * 16) la.per = (la.per + 1) / 2;
  la.split = (la.ltile + la.per - 1) / la.per;
  la.tiles = la.pp > 1 ? (a.P1 + la.pp - 1) / la.pp : a.P1 * la.split;
  const int64_t nblk = P0 * la.tiles;
  if (nblk <= 0) return BDDA_OK;
  if (nblk > 0x7fffffff) return BDDA_BAD_ARG;
  const size_t smem = (size_t)M * 3 * S::R * sizeof(T) + M * sizeof(T) + (M + 7) / 8 * 16 + 32;
  if (la.pp == 1) {
    auto kern = conv_kernel<T, M, true>;
    const size_t gsm = smem + (size_t)M * 6 * sizeof(T);
    const int s = line_smem_limit(kern, gsm, done[0]);
    if (s != BDDA_OK) return s;
    kern<<<(unsigned)nblk, S::NT, gsm, st>>>(la);
  } else {
    auto kern = conv_kernel<T, M, false>;
    const int s = line_smem_limit(kern, smem, done[1]);
    if (s != BDDA_OK) return s;
    kern<<<(unsigned)nblk, S::NT, smem, st>>>(la);
  }
  BDDA_CUDA_TRY(cudaGetLastError());
  count_launch();
  return BDDA_OK;
}

template <typename T, int KIND, int M, bool FULL>
constexpr LineLaunchFn line_entry() {
  if constexpr (line_split(M) != 0) return &line_launch<T, KIND, M, FULL>;
  else return nullptr;
}
template <typename T, int M>
constexpr LineLaunchFn conv_entry() {
  if constexpr (conv_split(M) != 0) return &conv_launch<T, M>;
  else return nullptr;
}

// The even 7-smooth lengths from 16 to 540 (a side of 270 cells) that have a split:
// all but 486 and 490.  The X pass has kernels of the first two lists, except 250;
// 294, in the third, has no split for it either.
#define BDDA_LINE_SHORT(F)                                                                              \
  F(16) F(18) F(20) F(24) F(28) F(30) F(32) F(36) F(40) F(42) F(48) F(50) F(54) F(56) F(60) F(64) F(70) \
  F(72) F(80) F(84) F(90) F(96) F(98) F(100) F(108) F(112) F(120) F(126) F(128)
#define BDDA_LINE_MID(F)                                                                       \
  F(140) F(144) F(150) F(160) F(162) F(168) F(180) F(192) F(196) F(200) F(210) F(216) F(224) F(240) F(250) \
  F(252) F(256) F(270) F(280) F(288) F(300) F(320)
#define BDDA_LINE_LONG(F)                                                                      \
  F(294) F(324) F(336) F(350) F(360) F(378) F(384) F(392) F(400) F(420) F(432) F(448) F(450) F(480) F(500) \
  F(504) F(512) F(540)

}  // namespace bdda
