// The project's Euclidean column norm on one warp (in place of the BLAS xNRM2 that the
// reference's dnorm2_/znorm2_ call, src/dnorm2.c:12), with the bit helpers it shares with
// the SVD kernels. Device code that needs only vj_fp.cuh, threadIdx.x and the warp
// shuffles, so that a host harness can run it lane by lane.
#pragma once
#include "vj_fp.cuh"

namespace vj {

template <typename T> __device__ __forceinline__ T bitst(unsigned long long u)
{
  return fp<T>::val((typename fp<T>::U)u);
}
template <typename T> __device__ __forceinline__ unsigned long long absbits(T x)
{
  return (unsigned long long)(fp<T>::bits(x) & ~fp<T>::SIGN);
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v)
{
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = (w > v) ? w : v;
  }
  return v;
}

// the warp's largest value, on every lane
#ifdef __CUDA_ARCH__
__device__ __forceinline__ unsigned warp_max_bits(unsigned v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long v)
{
  const unsigned h = (unsigned)(v >> 32), hm = __reduce_max_sync(0xffffffffu, h);
  const unsigned lm = __reduce_max_sync(0xffffffffu, (h == hm) ? (unsigned)v : 0u);
  return ((unsigned long long)hm << 32) | lm;
}
#else
template <typename U> __device__ U warp_max_bits(U v) { return (U)warp_max_u64((unsigned long long)v); }
#endif

// The second pass of the project's column norm: the sum of squares of x scaled by the power of
// two of its largest magnitude (mx: that magnitude's bits), for one warp; every lane returns
// the same value. Blocks of four elements per lane that scale to normal values (all of a
// column but its smallest entries) run as straight-line code, so that their loads and
// exponent adds overlap the accumulator's FMAs.
template <typename T> __device__ T warp_nrm2_scaled(const T *x, long long m, unsigned long long mx)
{
  using F = fp<T>;
  const int lane = threadIdx.x & 31;
  const T a = bitst<T>(mx);
  if (!visfinite(a))
    return visnan(a) ? F::qnan() : a;
  if (mx == 0ull)
    return (T)0;
  const int k = ilogb_(a), mm = (int)m;
  T acc = (T)0;
  int i = lane;
  for (; i + 96 < mm; i += 128) {
    T y[4];
    bool fast = true;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      y[u] = x[i + 32 * u];
      const int be = (int)((F::bits(y[u]) & ~F::SIGN) >> F::MB);
      fast = fast && (be > 0) && (be - k > 0);  // (|x| <= 2^(k+1): no overflow)
    }
    if (fast) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        y[u] = F::val(F::bits(y[u]) + ((typename F::U)(long long)(-k) << F::MB));
    }
    else {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        y[u] = scale2(y[u], -k);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      acc = F::fma_(y[u], y[u], acc);
  }
  for (; i < mm; i += 32) {
    const T y = scale2(x[i], -k);
    acc = F::fma_(y, y, acc);
  }
#pragma unroll
  for (int w = 16; w >= 1; w >>= 1)
    acc = acc + __shfl_down_sync(0xffffffffu, acc, w);
  acc = __shfl_sync(0xffffffffu, acc, 0);
  return scale2(F::sqrt_(acc), k);
}

// The project's column norm (two-pass power-of-two scaling, 32 lanes, halving tree) for
// one warp; every lane returns the same value.
template <typename T> __device__ T warp_nrm2(const T *x, long long m)
{
  const int lane = threadIdx.x & 31;
  typename fp<T>::U mx = 0;
  for (long long i = lane; i < m; i += 32) {
    const typename fp<T>::U a = fp<T>::bits(x[i]) & ~fp<T>::SIGN;
    mx = (a > mx) ? a : mx;
  }
  return warp_nrm2_scaled(x, m, warp_max_u64((unsigned long long)mx));
}

// The sums of squares of two columns, each scaled by 2^-k with k the exponent of its largest
// magnitude (mx, my: that magnitude's bits; zero or not finite: the sum is not used), in the
// project's norm order (svd_norm.cuh) for one warp, on its lane 0.
template <typename T>
__device__ void pair_sumsq(int m, const T *x, const T *y, typename fp<T>::U mx, typename fp<T>::U my, T &ax, T &ay)
{
  using F = fp<T>;
  const int lane = (int)(threadIdx.x & 31u);
  const T vx = F::val(mx), vy = F::val(my);
  const int kx = (mx && visfinite(vx)) ? -ilogb_(vx) : 0, ky = (my && visfinite(vy)) ? -ilogb_(vy) : 0;
  ax = ay = (T)0;
  if (sizeof(T) == 4 && kx >= 1 - F::BIAS && kx <= F::BIAS && ky >= 1 - F::BIAS && ky <= F::BIAS) {
    // (the product by a normal power of two is scale2's value)
    const T px = pow2<T>(kx), py = pow2<T>(ky);
#pragma unroll 4
    for (int i = lane; i < m; i += 32) {
      const T a = x[i] * px, b = y[i] * py;
      ax = F::fma_(a, a, ax);
      ay = F::fma_(b, b, ay);
    }
  }
  else {
    // four rows of a lane at a time, rows past the end as zeros (which add nothing)
    auto scaled = [](T v, int k, bool &fast) {
      const int e = (int)((F::bits(v) & ~F::SIGN) >> F::MB);
      if ((F::bits(v) & ~F::SIGN) != 0)
        fast = fast && (e > 0) && (e + k > 0) && (e + k <= F::EMAXB);
      return (e == 0) ? (T)0 : F::val(F::bits(v) + ((typename F::U)(long long)k << F::MB));
    };
    for (int i = lane; i < m; i += 128) {
      T a[4], b[4], sa[4], sb[4];
      bool fast = true;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool in = i + 32 * u < m;
        a[u] = in ? x[i + 32 * u] : (T)0;
        b[u] = in ? y[i + 32 * u] : (T)0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        sa[u] = scaled(a[u], kx, fast);
        sb[u] = scaled(b[u], ky, fast);
      }
      if (!fast) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          sa[u] = scale2(a[u], kx);
          sb[u] = scale2(b[u], ky);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (u == 0 || i + 32 * u < m) {
          ax = F::fma_(sa[u], sa[u], ax);
          ay = F::fma_(sb[u], sb[u], ay);
        }
    }
  }
#pragma unroll
  for (int w = 16; w >= 1; w >>= 1) {
    ax = ax + __shfl_down_sync(0xffffffffu, ax, w);
    ay = ay + __shfl_down_sync(0xffffffffu, ay, w);
  }
}

}  // namespace vj
