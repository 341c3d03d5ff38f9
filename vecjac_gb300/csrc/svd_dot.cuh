// The SVD's scaled compensated dot products in the reference's lane order (src/ddpscl.c,
// src/zdpscl.c): the per-precision constants, 2Sum, the lanes' halving-tree sum, the
// 8/16-lane form (pair_nu: the batched kernel; pair_dot: its quotient) and the FP64 form with
// one accumulator chain per warp (chain_dot: the check of a whole sweep's pairs; the step kernel,
// jsvd.cu, splits products and chains between warps itself). Device code that needs only
// vj_fp.cuh, threadIdx.x and __shfl_down_sync, so that a host harness can run it lane by
// lane.
#pragma once
#include <cfloat>

#include "vj_fp.cuh"

namespace vj {

template <typename T> struct svdc;
template <> struct svdc<double> {
  static constexpr int LANES = 8;
  static constexpr double EPS = DBL_EPSILON;
  static constexpr int ROT_R = 1022, ROT_C = 1021;
  static constexpr double MAX_FIN_EXP = 1023.0;
  static constexpr double RMAX = DBL_MAX;
};
template <> struct svdc<float> {
  static constexpr int LANES = 16;
  static constexpr float EPS = FLT_EPSILON;
  static constexpr int ROT_R = 126, ROT_C = 125;
  static constexpr float MAX_FIN_EXP = 127.0f;
  static constexpr float RMAX = FLT_MAX;
};

// 2Sum (src/d2sum.h)
template <typename T> __device__ __forceinline__ void two_sum(T a, T b, T &s, T &t)
{
  const T s_ = a + b;
  T a_ = s_ - b;
  T b_ = s_ - a_;
  a_ = a - a_;
  b_ = b - b_;
  s = s_;
  t = a_ + b_;
}

// halving tree over the LANES lanes of warp 0 (GCC's _mm512_reduce_add order); lane 0 has it
template <int LANES, typename T> __device__ __forceinline__ T hsum(T v)
{
#pragma unroll
  for (int w = LANES / 2; w >= 1; w >>= 1)
    v = __shfl_down_sync(0xffffffffu, v, w) + v;
  return v;
}

// scaled compensated dot products (src/ddpscl.c / src/zdpscl.c) by LANES lanes; x = G_q,
// y = G_p. Only the two (four for complex data) 2Sum accumulations carry a dependency from
// one element to the next; the loads, the power-of-two scaling and the exact product split
// (round-down product and its error by an FMA) of the elements of a block are independent
// of it, and blocks of normal values run as straight-line code so that their latency
// overlaps the accumulator chains.
template <typename T, bool CPLX> struct DotTerms {
  T pd[CPLX ? 4 : 1], dn[CPLX ? 4 : 1];
};

// One step of a 2Sum recurrence, (s, t) := (RN(s + b), s + b - RN(s + b)) with b = p + t.
// FP64: Dekker's Fast2Sum on the operands ordered by their high words. Fast2Sum's error is
// exact when the first operand's exponent is not below the second's (T. J. Dekker, "A
// floating-point technique for extending the available precision", Numer. Math. 18, 1971),
// which is 2Sum's error too, and the error of an addition is unique. That is 3 instead of 6
// FP64 operations after p + t; the comparison and the four selects run on the integer pipes
// while the FP64 unit forms s + b. Measured on one warp: 331 clocks per step against 448
// (2Sum), and 342 against 533 with one warp on each sub-partition. (An infinite s + b leaves
// t infinite or NaN and the dot product not finite, as with 2Sum.) FP32, where an addition
// costs no more than a select, keeps 2Sum.
// the high word's exponent and fraction of |b| above those of |s|; on the device as FP32 values,
// whose comparison takes the absolute values for free (28 clocks less on the recurrence than
// masking the words; the order is that of the words below 2^1017, and the scaled values
// accumulated here are below 4 m)
__device__ __forceinline__ bool hi_larger(double b, double s)
{
#ifdef __CUDA_ARCH__
  return fabsf(__int_as_float(__double2hiint(b))) > fabsf(__int_as_float(__double2hiint(s)));
#else
  return ((unsigned)(fp<double>::bits(b) >> 32) << 1) > ((unsigned)(fp<double>::bits(s) >> 32) << 1);
#endif
}
template <typename T> __device__ __forceinline__ void sum_step(const FpOps<T> &o, T p, T &s, T &t)
{
  const T b = o.add(p, t);
  if constexpr (sizeof(T) == 8) {
    const T r = o.add(s, b);
    const bool sw = hi_larger(b, s);
    const T h = sw ? b : s, l = sw ? s : b;
    t = o.sub(l, o.sub(r, h));
    s = r;
  }
  else
    two_sum(s, b, s, t);
}

template <typename T>
__device__ __forceinline__ void dot_acc(const FpOps<T> &o, T pd, T dn, T &s, T &t, T &s_, T &t_)
{
  sum_step(o, pd, s, t);
  sum_step(o, dn, s_, t_);
}

#ifdef __CUDACC__
// Two FP32 values in one register pair and the packed operations on them (each half rounded
// like the scalar operation): half the instructions of two recurrences that run in step.
struct F32x2 {
  unsigned long long v;
};
__device__ __forceinline__ F32x2 f2_make(float a, float b)
{
  F32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_get(F32x2 x, float &a, float &b)
{
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F32x2 f2_add(F32x2 a, F32x2 b)
{
  F32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F32x2 f2_mul(F32x2 a, F32x2 b)
{
  F32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F32x2 f2_fma(F32x2 a, F32x2 b, F32x2 c)
{
  F32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// pair_nu below for real FP32 columns whose scale factors 2^nx, 2^ny are normal: the scaling
// is a product (scale2's value for every x), the pd and dn recurrences share packed
// instructions: 13 instructions per row of a lane instead of about 36.
__device__ __forceinline__ void pair_nu_f32(int m, const float *x, const float *y, int nx, int ny, bool live, float &sr,
                                            float &tr, float &sr_, float &tr_)
{
  constexpr int L = svdc<float>::LANES, D = 4;
  const int lane = (int)(threadIdx.x & 31u) % L;
  const float px = pow2<float>(nx), py = pow2<float>(ny);
  const F32x2 neg = f2_make(-1.0f, -1.0f);
  F32x2 s = f2_make(0.0f, 0.0f), t = s;
  auto step = [&](float a, float b) {
    a *= px;
    b *= py;
    const float pd = __fmul_rd(a, b), dn = __fmaf_rn(a, b, -pd);
    const F32x2 q = f2_add(f2_make(pd, dn), t);
    const F32x2 r = f2_add(s, q);
    F32x2 u = f2_fma(q, neg, r);  // 2Sum, as two_sum above
    F32x2 w = f2_fma(u, neg, r);
    u = f2_fma(u, neg, s);
    w = f2_fma(w, neg, q);
    s = r;
    t = f2_add(u, w);
  };
  if (live) {
    // (every lane has m / L rows)
    const int rows = m / L;
    x += lane;
    y += lane;
    int r = 0;
    if (rows >= D) {
      float a[D], b[D];
#pragma unroll
      for (int d = 0; d < D; ++d) {
        a[d] = x[L * d];
        b[d] = y[L * d];
      }
      for (; r + 2 * D <= rows; r += D) {
        x += L * D;
        y += L * D;
        float a1[D], b1[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
          a1[d] = x[L * d];
          b1[d] = y[L * d];
        }
#pragma unroll
        for (int d = 0; d < D; ++d)
          step(a[d], b[d]);
#pragma unroll
        for (int d = 0; d < D; ++d) {
          a[d] = a1[d];
          b[d] = b1[d];
        }
      }
#pragma unroll
      for (int d = 0; d < D; ++d)
        step(a[d], b[d]);
      r += D;
      x += L * D;
      y += L * D;
    }
    for (; r < rows; ++r, x += L, y += L)
      step(*x, *y);
  }
  f2_get(s, sr, sr_);
  f2_get(t, tr, tr_);
}
#endif

// the dot product before its division by fx fy, on lane 0 of every group of LANES lanes
template <typename T, bool CPLX>
__device__ void pair_nu(long long m, const T *xr, const T *xi, const T *yr, const T *yi, T ex, T ey, bool live, T &zr,
                        T &zi)
{
  using F = fp<T>;
  constexpr int L = svdc<T>::LANES;
  constexpr int NV = CPLX ? 4 : 2;  // values loaded per element
  constexpr int D = 4;              // elements per block (the next block's loads in flight)
  const int lane = (threadIdx.x & 31) % L;
  const int nx = -(int)ex, ny = -(int)ey;
  const FpOps<T> o = FpOps<T>::make();
  T sr = 0, tr = 0, sr_ = 0, tr_ = 0, si = 0, ti = 0, si_ = 0, ti_ = 0;
  auto load = [&](long long i, T (&v)[NV]) {
    if (i < m) {
      v[0] = xr[i];
      v[1] = yr[i];
      if (CPLX) {
        v[2] = xi[i];
        v[3] = yi[i];
      }
    }
  };
  // products of one element from its scaled values; (negations are written as FP
  // negations: the FMA folds them, with the same bits)
  auto products = [&](T xri, T yri, T xii, T yii, DotTerms<T, CPLX> &d) {
    if (CPLX) {
      const T xs[4] = {xri, xii, xri, -xii}, ys[4] = {yri, yii, yii, yri};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        d.pd[k] = o.mul_rd(xs[k], ys[k]);
        d.dn[k] = F::fma_(xs[k], ys[k], -d.pd[k]);
      }
    }
    else {
      d.pd[0] = o.mul_rd(xri, yri);
      d.dn[0] = F::fma_(xri, yri, -d.pd[0]);
    }
  };
  auto accumulate = [&](const DotTerms<T, CPLX> &c) {
    if (CPLX) {
      dot_acc(o, c.pd[0], c.dn[0], sr, tr, sr_, tr_);
      dot_acc(o, c.pd[1], c.dn[1], sr, tr, sr_, tr_);
      dot_acc(o, c.pd[2], c.dn[2], si, ti, si_, ti_);
      dot_acc(o, c.pd[3], c.dn[3], si, ti, si_, ti_);
    }
    else
      dot_acc(o, c.pd[0], c.dn[0], sr, tr, sr_, tr_);
  };
  auto normal_after = [&](T w, int n) {
    const int be = (int)((F::bits(w) & ~F::SIGN) >> F::MB);
    return (be > 0) && (be <= F::EMAXB) && (be + n > 0) && (be + n <= F::EMAXB);
  };
  auto fscale = [&](T w, int n) { return F::val(F::bits(w) + ((typename F::U)(long long)n << F::MB)); };
#ifdef __CUDA_ARCH__
  bool done = false;
  if constexpr (sizeof(T) == 4 && !CPLX) {
    done = !live || (nx >= 1 - F::BIAS && nx <= F::BIAS && ny >= 1 - F::BIAS && ny <= F::BIAS);
    if (done)
      pair_nu_f32((int)m, xr, yr, nx, ny, live, sr, tr, sr_, tr_);
  }
#else
  const bool done = false;
#endif
  if (live && !done && lane < m) {
    T cur[D][NV], nxt[D][NV];
#pragma unroll
    for (int d = 0; d < D; ++d)
      load(lane + (long long)L * d, cur[d]);
    for (long long i0 = lane; i0 < m; i0 += (long long)L * D) {
#pragma unroll
      for (int d = 0; d < D; ++d)
        load(i0 + (long long)L * (D + d), nxt[d]);
      // a full block of values that scale to normal values: straight-line code (the
      // exponent add of scale2's fast path), so that the products of later elements can
      // fill the latency of the earlier elements' 2Sum recurrences
      bool fast = (i0 + (long long)L * (D - 1) < m);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        fast = fast && normal_after(cur[d][0], nx) && normal_after(cur[d][1], ny);
        if (CPLX)
          fast = fast && normal_after(cur[d][2], nx) && normal_after(cur[d][3], ny);
      }
      if (fast) {
        DotTerms<T, CPLX> tm[D];
#pragma unroll
        for (int d = 0; d < D; ++d)
          products(fscale(cur[d][0], nx), fscale(cur[d][1], ny), CPLX ? fscale(cur[d][2], nx) : (T)0,
                   CPLX ? fscale(cur[d][3], ny) : (T)0, tm[d]);
#pragma unroll
        for (int d = 0; d < D; ++d)
          accumulate(tm[d]);
      }
      else {
#pragma unroll
        for (int d = 0; d < D; ++d)
          if (i0 + (long long)L * d < m) {
            DotTerms<T, CPLX> tm;
            products(scale2(cur[d][0], nx), scale2(cur[d][1], ny), CPLX ? scale2(cur[d][2], nx) : (T)0,
                     CPLX ? scale2(cur[d][3], ny) : (T)0, tm);
            accumulate(tm);
          }
      }
#pragma unroll
      for (int d = 0; d < D; ++d)
#pragma unroll
        for (int k = 0; k < NV; ++k)
          cur[d][k] = nxt[d][k];
    }
  }
  zr = hsum<L>(sr) + (hsum<L>(tr) + (hsum<L>(sr_) + hsum<L>(tr_)));
  zi = 0;
  if (CPLX)
    zi = hsum<L>(si) + (hsum<L>(ti) + (hsum<L>(si_) + hsum<L>(ti_)));
}

template <typename T, bool CPLX>
__device__ void pair_dot(long long m, const T *xr, const T *xi, const T *yr, const T *yi, T ex, T ey, T fx, T fy,
                         bool live, T &zr, T &zi)
{
  pair_nu<T, CPLX>(m, xr, xi, yr, yi, ex, ey, live, zr, zi);
  const T de = fx * fy;
  zr = fp<T>::div(zr, de);
  zi = CPLX ? fp<T>::div(zi, de) : (T)0;
}

// The same scaled compensated dot products (FP64 only) with the independent accumulator
// chains of one lane in different warps. The reference keeps, per lane, two 2Sum
// recurrences (round-down products pd and their exact errors dn; src/ddpscl.c:46-60) for
// real data and four for complex data (real and imaginary parts; src/zdpscl.c:58-80).
// Chain C (bit 0: dn instead of pd, bit 1: imaginary part) of pairs 0..3 runs on one warp,
// pair j on lanes [8j, 8j+8): every lane keeps the reference's element order and
// recurrence, the chains of a lane just run side by side on different sub-partitions,
// each warp with one instruction stream (no per-thread selects: on GB300 an FP64 result
// that goes through the integer pipes costs hundreds of cycles). Elements are loaded a
// block (8 real, 4 complex) ahead of their accumulation, so that L2 latency (columns not
// staged in shared memory) overlaps the recurrence, and a block of normal values is
// accumulated by straight-line code whose products the scheduler can interleave with the
// recurrence. Returns the 8-lane halving-tree sums of s and t on lane 8j.
template <typename T, bool CPLX, int C>
__device__ void chain_dot(long long m, const T *xr, const T *xi, const T *yr, const T *yi, T ex, T ey, bool live,
                          int l8, T &S, T &Tt)
{
  static_assert(sizeof(T) == 8, "the chain-split dot product is the FP64 form");
  using F = fp<T>;
  constexpr bool DN = (C & 1) != 0, IM = (C & 2) != 0;
  constexpr int NV = CPLX ? 4 : 2;  // values loaded per element
  constexpr int NT = CPLX ? 2 : 1;  // terms accumulated per element
  constexpr int D = CPLX ? 4 : 8;   // elements per block: the next block's loads are in flight
                                    // while this block is accumulated (hides L2 latency)
  const int nx = -(int)ex, ny = -(int)ey;
  const FpOps<T> o = FpOps<T>::make();
  T s = 0, t = 0;
  auto load = [&](long long i, T (&v)[NV]) {
    if (i < m) {
      v[0] = xr[i];
      v[1] = yr[i];
      if (CPLX) {
        v[2] = xi[i];
        v[3] = yi[i];
      }
    }
  };
  // the term(s) of element i from its scaled values: real part xr yr, xi yi; imaginary part
  // xr yi, xi (-yr) (= (-xi) yr exactly)
  auto terms = [&](T xr_, T yr_, T xi_, T yi_, T (&v)[NT]) {
    const T a0 = xr_, b0 = (CPLX && IM) ? yi_ : yr_;
    const T q0 = o.mul_rd(a0, b0);
    v[0] = DN ? F::fma_(a0, b0, -q0) : q0;
    if (CPLX) {
      const T a1 = xi_, b1 = IM ? -yr_ : yi_;
      const T q1 = o.mul_rd(a1, b1);
      v[NT - 1] = DN ? F::fma_(a1, b1, -q1) : q1;
    }
  };
  // the general path: scale2 with its special cases, one element at a time
  auto acc = [&](const T (&w)[NV]) {
    T v[NT];
    terms(scale2(w[0], nx), scale2(w[1], ny), CPLX ? scale2(w[2], nx) : (T)0, CPLX ? scale2(w[3], ny) : (T)0, v);
#pragma unroll
    for (int k = 0; k < NT; ++k)
      sum_step(o, v[k], s, t);
  };
  // the power-of-two scaling of a normal value to a normal result is an integer add on the
  // exponent field (scale2's fast path)
  auto normal_after = [&](T w, int n) {
    const int be = (int)((F::bits(w) & ~F::SIGN) >> F::MB);
    return (be > 0) && (be <= F::EMAXB) && (be + n > 0) && (be + n <= F::EMAXB);
  };
  auto fscale = [&](T w, int n) { return F::val(F::bits(w) + ((typename F::U)(long long)n << F::MB)); };
  if (live && l8 < m) {
    T cur[D][NV], nxt[D][NV];
#pragma unroll
    for (int d = 0; d < D; ++d)
      load(l8 + 8LL * d, cur[d]);
    for (long long i0 = l8; i0 < m; i0 += 8LL * D) {
#pragma unroll
      for (int d = 0; d < D; ++d)
        load(i0 + 8LL * (D + d), nxt[d]);
      // a full block of normal values: straight-line code, so that the products of later
      // elements fill the latency of the earlier elements' 2Sum recurrence
      bool fast = (i0 + 8LL * (D - 1) < m);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        fast = fast && normal_after(cur[d][0], nx) && normal_after(cur[d][1], ny);
        if (CPLX)
          fast = fast && normal_after(cur[d][2], nx) && normal_after(cur[d][3], ny);
      }
      if (fast) {
        T v[D][NT];
#pragma unroll
        for (int d = 0; d < D; ++d)
          terms(fscale(cur[d][0], nx), fscale(cur[d][1], ny), CPLX ? fscale(cur[d][2], nx) : (T)0,
                CPLX ? fscale(cur[d][3], ny) : (T)0, v[d]);
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
          for (int k = 0; k < NT; ++k)
            sum_step(o, v[d][k], s, t);
      }
      else {
#pragma unroll
        for (int d = 0; d < D; ++d)
          if (i0 + 8LL * d < m)
            acc(cur[d]);
      }
#pragma unroll
      for (int d = 0; d < D; ++d)
#pragma unroll
        for (int k = 0; k < NV; ++k)
          cur[d][k] = nxt[d][k];
    }
  }
  S = hsum<8>(s);
  Tt = hsum<8>(t);
}

}  // namespace vj
