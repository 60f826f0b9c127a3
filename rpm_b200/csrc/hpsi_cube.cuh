// Device pieces of the general cube form of H psi (see hpsi.cu), shared by its
// tiled passes and by the one-block Lanczos kernel of small states (batched.cu).
#pragma once

#include "common.cuh"
#include "hpsi.cuh"

namespace rpm {

// ---------------------------------------------------------------------------
// Cube form
// ---------------------------------------------------------------------------
// Complex multiply-accumulate of the cube kernels: four FMAs per complex
// product in the state precision (FP32 for complex64, FP64 for complex128).
template <class T> struct CubeArith;

template <>
struct CubeArith<double2> {
  using Coef = double2;
  using R = double;
  __device__ static double2 prep(double2 x) { return x; }
  __device__ static double2 mac(const double2& c, double2 x, double2, double2 acc) { return cfma(c, x, acc); }
  __device__ static double2 rmac(double d, double2 x, double2 acc) {
    acc.x = fma(d, x.x, acc.x);
    acc.y = fma(d, x.y, acc.y);
    return acc;
  }
  __device__ static double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
  __device__ static double2 from_complex(double2 v) { return v; }
  __device__ static double re(const double2& c) { return c.x; }
};

template <>
struct CubeArith<float2> {
  using Coef = float2;
  using R = float;
  __device__ static float2 prep(float2 x) { return x; }
  __device__ static float2 mac(const float2& c, float2 x, float2, float2 acc) { return cfma(c, x, acc); }
  __device__ static float2 rmac(float d, float2 x, float2 acc) {
    acc.x = fmaf(d, x.x, acc.x);
    acc.y = fmaf(d, x.y, acc.y);
    return acc;
  }
  __device__ static float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
  __device__ static float2 from_complex(float2 v) { return v; }
  __device__ static float re(const float2& c) { return c.x; }
};

// Per outer index o (all group digits except the NI inner ones), built once
// per CTA in shared memory: the outer digits packed 4 bits each and the
// diagonal / electron-flip coefficients merged over Z and the outer digits.
// Group index g = e * half + C * o + i  (C = 2^NI, i = inner digits).
template <class T>
struct OuterRec {
  typename CubeArith<T>::Coef f[2];
  typename CubeArith<T>::R d[2];
  unsigned lo, hi;
};

__device__ __forceinline__ int align16(int bytes) { return (bytes + 15) & ~15; }

// Asynchronous global -> shared copy of one complex element (cp.async).
template <class T>
__device__ __forceinline__ void async_copy(T* smem_dst, const T* gmem_src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  if constexpr (sizeof(T) == 16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem_src) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem_src) : "memory");
  }
}
__device__ __forceinline__ void async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// Copy one group's CubeSide and its coefficient table into shared memory.
template <class Coef>
__device__ __forceinline__ void load_side(const CubeSide& src, const Coef* tab_src, CubeSide& side, Coef* tab) {
  const int* s = reinterpret_cast<const int*>(&src);
  int* d = reinterpret_cast<int*>(&side);
  for (int k = threadIdx.x; k < (int)(sizeof(CubeSide) / sizeof(int)); k += blockDim.x) d[k] = s[k];
  __syncthreads();
  for (int k = threadIdx.x; k < side.ntab; k += blockDim.x) tab[k] = tab_src[k];
}

template <class T, int NI>
__device__ __forceinline__ void build_outer(const CubeSide& side, const typename CubeArith<T>::Coef* tab,
                                            OuterRec<T>* otab, int n_outer) {
  using A = CubeArith<T>;
  const int nout = side.K - NI;
  for (int o = threadIdx.x; o < n_outer; o += blockDim.x) {
    OuterRec<T> rec;
    rec.d[0] = A::re(tab[0]);
    rec.d[1] = A::re(tab[1]);
    rec.f[0] = tab[2];
    rec.f[1] = tab[3];
    int rem = o;
    unsigned lo = 0, hi = 0;
    for (int k = nout - 1; k >= 0; --k) {
      const int d = side.dim[k];
      const int m = rem % d;
      rem /= d;
      if (k < 8) lo |= (unsigned)m << (4 * k);
      else hi |= (unsigned)m << (4 * (k - 8));
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        rec.d[e] += A::re(tab[side.offD[k] + e * d + m]);
        rec.f[e] = A::add(rec.f[e], tab[side.offF[k] + e * d + m]);
      }
    }
    rec.lo = lo;
    rec.hi = hi;
    otab[o] = rec;
  }
}

// Diagonal and electron-flip coefficients contributed by the inner digits:
// the same for every cube of a CTA, so computed once per thread.
template <class T, int NI>
struct InnerConst {
  typename CubeArith<T>::R d[2][1 << NI];
  typename CubeArith<T>::Coef f[2][1 << NI];
  __device__ InnerConst(const CubeSide& side, const typename CubeArith<T>::Coef* tab) {
    using A = CubeArith<T>;
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int i = 0; i < (1 << NI); ++i) {
        // first inner digit, then the others
        typename A::Coef fl = tab[side.offF[side.K - NI] + e * 2 + ((i >> (NI - 1)) & 1)];
        typename A::R dg = A::re(tab[side.offD[side.K - NI] + e * 2 + ((i >> (NI - 1)) & 1)]);
#pragma unroll
        for (int q = 1; q < NI; ++q) {
          const int k = side.K - NI + q;
          const int bit = (i >> (NI - 1 - q)) & 1;
          dg += A::re(tab[side.offD[k] + e * 2 + bit]);
          fl = A::add(fl, tab[side.offF[k] + e * 2 + bit]);
        }
        d[e][i] = dg;
        f[e][i] = fl;
      }
  }
};

// Register-cube update shared by both passes.  `at(e, i, delta)` returns the
// element (electron e, inner i) of the cube whose outer index is shifted by
// `delta` (delta = 0: the thread's own cube).
template <class T, int NI, class At>
__device__ __forceinline__ void cube_apply(const CubeSide& side, const typename CubeArith<T>::Coef* tab,
                                           const InnerConst<T, NI>& ic, const OuterRec<T>& rec,
                                           const typename CubeArith<T>::R (&dout)[2],
                                           const typename CubeArith<T>::Coef (&fout)[2], const T (&x)[2][1 << NI],
                                           T (&acc)[2][1 << NI], At at) {
  using A = CubeArith<T>;
  constexpr int C = 1 << NI;
  const int K = side.K;
  T xs[2][C];
#pragma unroll
  for (int e = 0; e < 2; ++e)
#pragma unroll
    for (int i = 0; i < C; ++i) xs[e][i] = A::prep(x[e][i]);
#pragma unroll
  for (int e = 0; e < 2; ++e)
#pragma unroll
    for (int i = 0; i < C; ++i) {
      acc[e][i] = A::rmac(dout[e] + ic.d[e][i], x[e][i], acc[e][i]);
      acc[e][i] = A::mac(A::add(fout[e], ic.f[e][i]), x[1 - e][i], xs[1 - e][i], acc[e][i]);
    }
#pragma unroll
  for (int q = 0; q < NI; ++q) {
    const typename A::Coef* X = tab + side.offX[K - NI + q];
#pragma unroll
    for (int i = 0; i < C; ++i) {
      const int bit = (i >> (NI - 1 - q)) & 1;
      const int ip = i ^ (1 << (NI - 1 - q));
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        acc[e][i] = A::mac(X[(e * 2 + bit) * 4 + (1 - bit)], x[0][ip], xs[0][ip], acc[e][i]);
        acc[e][i] = A::mac(X[(e * 2 + bit) * 4 + 2 + (1 - bit)], x[1][ip], xs[1][ip], acc[e][i]);
      }
    }
  }
  const int nout = K - NI;
  for (int k = 0; k < nout; ++k) {
    const int d = side.dim[k];
    const int m = (int)(((k < 8) ? (rec.lo >> (4 * k)) : (rec.hi >> (4 * (k - 8)))) & 15u);
    const int ostride = side.gs[k] >> NI;
    const typename A::Coef* X = tab + side.offX[k] + (size_t)m * 2 * d;
    for (int mp = 0; mp < d; ++mp) {
      if (mp == m) continue;
      const int delta = (mp - m) * ostride;
      T y[2][C];
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int i = 0; i < C; ++i) y[e][i] = at(e, i, delta);
#pragma unroll
      for (int ep = 0; ep < 2; ++ep) {
        // coefficients of output electron e from input electron ep
        const typename A::Coef c0 = X[(0 * d) * 2 * d + ep * d + mp];
        const typename A::Coef c1 = X[(1 * d) * 2 * d + ep * d + mp];
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const T ys = A::prep(y[ep][i]);
          acc[0][i] = A::mac(c0, y[ep][i], ys, acc[0][i]);
          acc[1][i] = A::mac(c1, y[ep][i], ys, acc[1][i]);
        }
      }
    }
  }
}

}  // namespace rpm
