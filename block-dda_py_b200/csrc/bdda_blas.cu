// Tall-skinny block kernels: Gram products, fused block updates, dots.
#include <climits>
#include <type_traits>

#include "bdda_blas.cuh"
#include "bdda_blas_dev.cuh"
#include "bdda_internal.h"

namespace bdda {

// L-specialised Gram / update kernels on (tests switch them off to compare).
static int g_fixed_blas = 1;

// ---- Gram: G_k[i][j] = sum_r op(A[r][i]) B_k[r][j], any L <= 64 ---------------
// The L x L tile is padded to LP = NT TM columns and computed by NT x NT
// threads with TM x TM elements each (rows ty + NT i, columns tx + NT j, so a warp
// reads consecutive words); narrow blocks leave room for GROUPS = 256 / NT^2
// such thread grids, which take the rows of a chunk in turn and are added at
// the end.  Chunks are double-buffered with cp.async.  The kernel before
// (one thread grid whatever L, no prefetch) ran L = 1 with one thread of 256
// busy: 97 us for 3 x 105,000 rows and two products, 9 us now.
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

template <int NT, int TM> struct GramShape {
  static constexpr int LP = NT * TM, GROUPS = 256 / (NT * NT);
  // rows per chunk: 512 / LP for narrow blocks, 16 for wide ones
  static constexpr int RCH = 512 / LP > 16 ? 512 / LP : 16;
};

template <typename T, bool CONJ, int NT, int TM, int NB>
__global__ void __launch_bounds__(256) gram_kernel(GramArgs g) {
  typedef GramShape<NT, TM> S;
  constexpr int LP = S::LP, GROUPS = S::GROUPS, RCH = S::RCH, CH = RCH * LP;
  extern __shared__ __align__(16) unsigned char gsh[];
  T* buf = reinterpret_cast<T*>(gsh);   // [2][1 + NB][RCH][LP]
  const int L = g.L, t = threadIdx.x;
  const int grp = t / (NT * NT), tt = t - grp * (NT * NT), ty = tt / NT, tx = tt - ty * NT;
  const float by_l = 1.f / L;
  T zero;
  zero.x = 0;
  zero.y = 0;
  for (int e = t; e < 2 * (1 + NB) * CH; e += 256) buf[e] = zero;   // the columns at or past L stay zero
  __syncthreads();
  double2 acc[NB][TM][TM];
#pragma unroll
  for (int k = 0; k < NB; ++k)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TM; ++j) acc[k][i][j] = make_double2(0.0, 0.0);
  const int64_t nchunks = (g.n + RCH - 1) / RCH;
  const int64_t per = (nchunks + gridDim.x - 1) / gridDim.x;
  const int64_t c0 = blockIdx.x * per, c1 = min(nchunks, c0 + per);
  const T* src[1 + NB];
  src[0] = static_cast<const T*>(g.A);
#pragma unroll
  for (int k = 0; k < NB; ++k) src[1 + k] = static_cast<const T*>(g.B[k]);
  auto stage = [&](int64_t ck, int slot) {
    const int64_t r0 = ck * RCH;
    const int valid = (int)min((int64_t)RCH, g.n - r0) * L;
    for (int e = t; e < RCH * L; e += 256) {
      const int r = (int)((e + 0.5f) * by_l), c = e - r * L;
#pragma unroll
      for (int m = 0; m < 1 + NB; ++m) {
        T* d = buf + (slot * (1 + NB) + m) * CH + r * LP + c;
        if (e < valid) cp_async_elem<(int)sizeof(T)>(d, src[m] + r0 * L + e);
        else *d = zero;
      }
    }
  };
  if (c0 < c1) stage(c0, 0);
  cp_async_commit_g();
  for (int64_t ck = c0; ck < c1; ++ck) {
    const int slot = (int)((ck - c0) & 1);
    if (ck + 1 < c1) stage(ck + 1, slot ^ 1);
    cp_async_commit_g();
    cp_async_wait_g<1>();
    __syncthreads();
    const T* sA = buf + slot * (1 + NB) * CH;
#pragma unroll 2
    for (int r = grp; r < RCH; r += GROUPS) {
      double2 a[TM], b[NB][TM];
#pragma unroll
      for (int ii = 0; ii < TM; ++ii) {
        a[ii] = to_d2(sA[r * LP + ty + NT * ii]);
        if (CONJ) a[ii].y = -a[ii].y;
      }
#pragma unroll
      for (int k = 0; k < NB; ++k)
#pragma unroll
        for (int jj = 0; jj < TM; ++jj) b[k][jj] = to_d2(sA[(1 + k) * CH + r * LP + tx + NT * jj]);
#pragma unroll
      for (int k = 0; k < NB; ++k)
#pragma unroll
        for (int ii = 0; ii < TM; ++ii)
#pragma unroll
          for (int jj = 0; jj < TM; ++jj) acc[k][ii][jj] = cfma(a[ii], b[k][jj], acc[k][ii][jj]);
    }
    __syncthreads();
  }
  cp_async_wait_g<0>();
  double2* out = g.partial + (int64_t)blockIdx.x * NB * L * L;
  if constexpr (GROUPS == 1) {
#pragma unroll
    for (int k = 0; k < NB; ++k)
#pragma unroll
      for (int ii = 0; ii < TM; ++ii)
#pragma unroll
        for (int jj = 0; jj < TM; ++jj) {
          const int i = ty + NT * ii, j = tx + NT * jj;
          if (i < L && j < L) out[(k * L + i) * L + j] = acc[k][ii][jj];
        }
  } else {   // TM = 1: add the thread grids (rows of the chunk modulo GROUPS) in order
    double2* red = reinterpret_cast<double2*>(gsh);   // [GROUPS][NB][NT][NT]: 512 elements at most
#pragma unroll
    for (int k = 0; k < NB; ++k) red[(grp * NB + k) * (NT * NT) + tt] = acc[k][0][0];
    __syncthreads();
    if (grp < NB && ty < L && tx < L) {
      double2 s = make_double2(0.0, 0.0);
      for (int q = 0; q < GROUPS; ++q) {
        const double2 v = red[(q * NB + grp) * (NT * NT) + tt];
        s.x += v.x;
        s.y += v.y;
      }
      out[(grp * L + ty) * L + tx] = s;
    }
  }
}

__global__ void gram_reduce_kernel(const double2* partial, int nblk, int width, double2* out) {
  gram_reduce_body(partial, nblk, width, out, blockIdx.x * kReduceOut);
}

template <typename T, bool CONJ, int L, int NB>
__global__ void __launch_bounds__(256) gram_fixed_kernel(GramArgs g) {
  extern __shared__ __align__(16) unsigned char gfs[];
  gram_fixed_body<T, CONJ, L, NB>(g, blockIdx.x, gridDim.x, gfs);
}

template <typename T, bool CONJ, int L>
static int gram_fixed(const GramArgs& g, double2* out, cudaStream_t st) {
  const size_t smem = (size_t)2 * (1 + g.nB) * 16 * L * sizeof(T);
  if (g.nB == 1) {
    auto k = gram_fixed_kernel<T, CONJ, L, 1>;
    BDDA_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k<<<kRedBlocks, 256, smem, st>>>(g);
  } else {
    auto k = gram_fixed_kernel<T, CONJ, L, 2>;
    BDDA_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k<<<kRedBlocks, 256, smem, st>>>(g);
  }
  BDDA_CUDA_TRY(cudaGetLastError());
  const int width = g.nB * L * L;
  gram_reduce_kernel<<<(width + kReduceOut - 1) / kReduceOut, 256, 0, st>>>(g.partial, kRedBlocks, width, out);
  BDDA_CUDA_TRY(cudaGetLastError());
  count_launch(2);
  return BDDA_OK;
}

template <typename T, bool CONJ, int NT, int TM, int NB>
static int gram_launch(const GramArgs& g, cudaStream_t st) {
  typedef GramShape<NT, TM> S;
  const size_t stages = (size_t)2 * (1 + NB) * S::RCH * S::LP * sizeof(T), groups = (size_t)NB * 256 * sizeof(double2);
  const size_t smem = stages > groups ? stages : groups;
  auto k = gram_kernel<T, CONJ, NT, TM, NB>;
  BDDA_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k<<<kRedBlocks, 256, smem, st>>>(g);
  BDDA_CUDA_TRY(cudaGetLastError());
  return BDDA_OK;
}
template <typename T, bool CONJ, int NT, int TM>
static int gram_tm(const GramArgs& g, double2* out, cudaStream_t st) {
  const int s = g.nB == 1 ? gram_launch<T, CONJ, NT, TM, 1>(g, st) : gram_launch<T, CONJ, NT, TM, 2>(g, st);
  if (s != BDDA_OK) return s;
  const int width = g.nB * g.L * g.L;
  gram_reduce_kernel<<<(width + kReduceOut - 1) / kReduceOut, 256, 0, st>>>(g.partial, kRedBlocks, width, out);
  BDDA_CUDA_TRY(cudaGetLastError());
  count_launch(2);
  return BDDA_OK;
}
// the smallest padded width that holds L
template <typename T, bool CONJ>
static int gram_any(const GramArgs& g, double2* out, cudaStream_t st) {
  if (g.L == 1) return gram_tm<T, CONJ, 1, 1>(g, out, st);
  if (g.L == 2) return gram_tm<T, CONJ, 2, 1>(g, out, st);
  if (g.L <= 4) return gram_tm<T, CONJ, 4, 1>(g, out, st);
  if (g.L <= 8) return gram_tm<T, CONJ, 8, 1>(g, out, st);
  if (g.L <= 16) return gram_tm<T, CONJ, 16, 1>(g, out, st);
  if (g.L <= 32) return gram_tm<T, CONJ, 16, 2>(g, out, st);
  if (g.L <= 48) return gram_tm<T, CONJ, 16, 3>(g, out, st);
  return gram_tm<T, CONJ, 16, 4>(g, out, st);
}

template <typename T>
int gram(const GramArgs& g, bool conj, double2* out, cudaStream_t st) {
  if (g.L < 1 || g.L > kMaxL || g.nB < 1 || g.nB > 2) return BDDA_BAD_ARG;
  const bool aligned = ((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B[0]) |
                         reinterpret_cast<uintptr_t>(g.nB > 1 ? g.B[1] : g.B[0])) & 15) == 0;
  if (aligned && g_fixed_blas) {
#define BDDA_GRAM_L(LL) \
  if (g.L == LL) return conj ? gram_fixed<T, true, LL>(g, out, st) : gram_fixed<T, false, LL>(g, out, st);
    BDDA_GRAM_L(8) BDDA_GRAM_L(16) BDDA_GRAM_L(32) BDDA_GRAM_L(64)
#undef BDDA_GRAM_L
  }
  return conj ? gram_any<T, true>(g, out, st) : gram_any<T, false>(g, out, st);
}

// ---- fused block update, any L <= 64 ----------------------------------------------
// out = a0*Y0 + a1*Y1 + (X1 + c2*X2) M, arithmetic in A (double2 for c128,
// float2 for c64 vectors), optional per-CTA partial of ||out||_F^2.  NCG x NRG
// threads; a thread owns two rows and the columns cg + NCG j (consecutive lanes
// read consecutive words of M, padded to NCG TC columns).
template <typename T, typename A, int NCG, int TC>
__global__ void __launch_bounds__(256) update_kernel(UpdateArgs u) {
  constexpr int LP = NCG * TC, NRG = 256 / NCG, TR = 2, RB = NRG * TR;
  const int L = u.L;
  extern __shared__ __align__(16) unsigned char ush[];
  A* sM = reinterpret_cast<A*>(ush);           // [L][LP]
  A* sX = sM + (u.M ? L * LP : 0);             // [RB][L]
  const int t = threadIdx.x;
  const int rg = t / NCG, cg = t - rg * NCG;
  const A one = conv_acc<A>(make_double2(1.0, 0.0)), zero = conv_acc<A>(make_double2(0.0, 0.0));
  const A a0 = u.a0 ? conv_acc<A>(*u.a0) : one;
  const A a1 = u.a1 ? conv_acc<A>(*u.a1) : one;
  const A c2 = u.c2 ? conv_acc<A>(*u.c2) : one;
  const T* Y0 = static_cast<const T*>(u.Y0);
  const T* Y1 = static_cast<const T*>(u.Y1);
  const T* X1 = static_cast<const T*>(u.X1);
  const T* X2 = static_cast<const T*>(u.X2);
  T* out = static_cast<T*>(u.out);
  if (u.M)
    for (int e = t; e < L * LP; e += 256) {
      const int r = e / LP, c = e - r * LP;
      sM[e] = c < L ? conv_acc<A>(u.M[r * L + c]) : zero;
    }
  double nrm = 0.0;
  for (int64_t rb = (int64_t)blockIdx.x * RB; rb < u.n; rb += (int64_t)gridDim.x * RB) {
    if (u.M) {
      __syncthreads();
      const int64_t left = (u.n - rb) * L;
      for (int e = t; e < RB * L; e += 256) {
        A v = zero;
        if (e < left) {
          v = ld_as<A>(X1, rb * L + e);
          if (X2) v = cfma(c2, ld_as<A>(X2, rb * L + e), v);
        }
        sX[e] = v;
      }
      __syncthreads();
    }
    A acc[TR][TC];
#pragma unroll
    for (int ii = 0; ii < TR; ++ii) {
      const int64_t row = rb + rg + NRG * ii;
#pragma unroll
      for (int jj = 0; jj < TC; ++jj) {
        const int c = cg + NCG * jj;
        acc[ii][jj] = zero;
        if (row < u.n && c < L) {
          if (Y0) acc[ii][jj] = cfma(a0, ld_as<A>(Y0, row * L + c), acc[ii][jj]);
          if (Y1) acc[ii][jj] = cfma(a1, ld_as<A>(Y1, row * L + c), acc[ii][jj]);
        }
      }
    }
    if (u.M) {
#pragma unroll 4
      for (int i = 0; i < L; ++i) {
        A x[TR], m[TC];
#pragma unroll
        for (int ii = 0; ii < TR; ++ii) x[ii] = sX[(rg + NRG * ii) * L + i];
#pragma unroll
        for (int jj = 0; jj < TC; ++jj) m[jj] = sM[i * LP + cg + NCG * jj];
#pragma unroll
        for (int ii = 0; ii < TR; ++ii)
#pragma unroll
          for (int jj = 0; jj < TC; ++jj) acc[ii][jj] = cfma(x[ii], m[jj], acc[ii][jj]);
      }
    }
#pragma unroll
    for (int ii = 0; ii < TR; ++ii) {
      const int64_t row = rb + rg + NRG * ii;
#pragma unroll
      for (int jj = 0; jj < TC; ++jj) {
        const int c = cg + NCG * jj;
        if (row < u.n && c < L) {
          const T v = st_as<T>(acc[ii][jj]);
          out[row * L + c] = v;
          const double2 vd = to_d2(v);
          nrm += vd.x * vd.x + vd.y * vd.y;
        }
      }
    }
  }
  if (u.norm_partial) {
    const double s = block_sum(nrm);
    if (threadIdx.x == 0) u.norm_partial[blockIdx.x] = s;
  }
}

// CTAs of an update: kRedBlocks where the norm's partials are counted on,
// else up to eight per SM (an update moves three or four vectors and little
// else, so it needs the bytes in flight: 143 -> 107 us for 280,000 rows at L = 32).
static int update_grid(const UpdateArgs& u, int rb) {
  if (u.norm_partial) return kRedBlocks;
  const int64_t b = (u.n + rb - 1) / rb;
  return (int)(b < 1 ? 1 : b < 4 * kRedBlocks ? b : 4 * kRedBlocks);
}

template <typename T, typename A, int L>
__global__ void __launch_bounds__(256) update_fixed_kernel(UpdateArgs u) {
  extern __shared__ __align__(16) unsigned char ufs[];
  update_fixed_body<T, A, L>(u, blockIdx.x, gridDim.x, ufs);
}

template <typename T, typename A, int L>
static int update_fixed(const UpdateArgs& u, cudaStream_t st) {
  constexpr int TC = L >= 64 ? 4 : (L >= 32 ? 2 : 1);
  constexpr int RB = (256 / (L / TC)) * 2;
  const size_t smem = u.M ? ((size_t)L * L + (size_t)RB * L) * sizeof(A) : 0;
  auto k = update_fixed_kernel<T, A, L>;
  BDDA_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k<<<update_grid(u, RB), 256, smem, st>>>(u);
  BDDA_CUDA_TRY(cudaGetLastError());
  count_launch();
  return BDDA_OK;
}

template <typename T, typename A, int NCG, int TC>
static int update_tn(const UpdateArgs& u, cudaStream_t st) {
  constexpr int RB = 256 / NCG * 2;
  const size_t smem = u.M ? ((size_t)u.L * NCG * TC + (size_t)RB * u.L) * sizeof(A) : 0;
  auto k = update_kernel<T, A, NCG, TC>;
  BDDA_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k<<<update_grid(u, RB), 256, smem, st>>>(u);
  BDDA_CUDA_TRY(cudaGetLastError());
  count_launch();
  return BDDA_OK;
}

template <typename T>
int update(const UpdateArgs& u, cudaStream_t st) {
  if (u.L < 1 || u.L > kMaxL || !u.out) return BDDA_BAD_ARG;
  typedef typename std::conditional<std::is_same<T, float2>::value, float2, double2>::type A;
  if (g_fixed_blas) {
    if (u.L == 64) return update_fixed<T, A, 64>(u, st);
    if (u.L == 32) return update_fixed<T, A, 32>(u, st);
    if (u.L == 16) return update_fixed<T, A, 16>(u, st);
    if (u.L == 8) return update_fixed<T, A, 8>(u, st);
  }
  if (u.L == 1) return update_tn<T, A, 1, 1>(u, st);
  if (u.L == 2) return update_tn<T, A, 2, 1>(u, st);
  if (u.L <= 4) return update_tn<T, A, 4, 1>(u, st);
  if (u.L <= 8) return update_tn<T, A, 8, 1>(u, st);
  if (u.L <= 16) return update_tn<T, A, 16, 1>(u, st);
  if (u.L <= 32) return update_tn<T, A, 16, 2>(u, st);
  if (u.L <= 48) return update_tn<T, A, 16, 3>(u, st);
  return update_tn<T, A, 16, 4>(u, st);
}

template <typename T>
__global__ void __launch_bounds__(256) dots_kernel(DotArgs d) {
  dots_body<T>(d, blockIdx.x, gridDim.x);
}

template <typename T>
int dots(const DotArgs& d, cudaStream_t st) {
  dots_kernel<T><<<kRedBlocks, 256, 0, st>>>(d);
  BDDA_CUDA_TRY(cudaGetLastError());
  count_launch();
  return BDDA_OK;
}

__global__ void reduce_partials_kernel(const double* partial, int nblk, int width, double* out) {
  for (int w = 0; w < width; ++w) {
    double s = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) s += partial[(int64_t)b * width + w];
    s = block_sum(s);
    if (threadIdx.x == 0) out[w] = s;
    __syncthreads();
  }
}

int reduce_partials(const double* partial, int nblk, int width, double* out, cudaStream_t st) {
  reduce_partials_kernel<<<1, 256, 0, st>>>(partial, nblk, width, out);
  BDDA_CUDA_TRY(cudaGetLastError());
  count_launch();
  return BDDA_OK;
}

void set_fixed_blas(int on) { g_fixed_blas = on ? 1 : 0; }

template int gram<double2>(const GramArgs&, bool, double2*, cudaStream_t);
template int gram<float2>(const GramArgs&, bool, double2*, cudaStream_t);
template int update<double2>(const UpdateArgs&, cudaStream_t);
template int update<float2>(const UpdateArgs&, cudaStream_t);
template int dots<double2>(const DotArgs&, cudaStream_t);
template int dots<float2>(const DotArgs&, cudaStream_t);

}  // namespace bdda
