// Mixed-precision one-sided Jacobi SVD: FP32 sweeps, FP64 refinement on the tensor cores.
//
// GB300 runs FP32 arithmetic at about 70 times its FP64 rate and exact products of 8-bit digits
// on the tensor cores at more than that, so most of the sweeps are done in FP32 and the FP64 work
// is matrix products. Starting from G_0 = A (FP64), V_0 = I, each preconditioning stage s = 1..S
//   1. rounds G_{s-1} (scaled by a power of two to max |g_ij| <= 1) to FP32;
//   2. runs FP32 one-sided Jacobi sweeps on it from W := I until no pair exceeds the FP32
//      tolerance: block sweeps with split-BF16x3 tensor-core products (blockjac.cu) where
//      there are enough block pairs, sweeps by small blocks of columns (colblk.cu) where a pair of
//      those fits in shared memory, else column-pair Hestenes sweeps (k_presweep_reg / k_presweep,
//      rotations from plain FP32 dot products);
//   3. widens W to FP64 and makes it unitary to FP64 accuracy by corrections from its Gram matrix,
//      its columns in ascending order of norm;
//   4. forms G_s = G_{s-1} W and V_s = V_{s-1} W.
// FP32 rounding is relative to each element, so from the second stage on the FP32 sweeps
// see the columns of G_{s-1} to their own relative accuracy and resolve the directions of
// small singular values that the first stage (on A itself) could not. Refinements G := G exp(K),
// V := V exp(K) with K from G's Gram matrix then bring the columns to FP64 orthogonality, two of
// them in general; FP64 sweeps with plain dot products (the same step kernel in FP64, on G and V
// themselves, with a scale factor per column and tracked norms) take over where they cannot.
// Every FP64 product of these phases is a sum of exact digit products on the tensor cores
// (fp64tc.cu), with as many digits as its own accuracy needs; V's are formed in two scalings where A's
// columns differ much in length (mult_cols). Finally dvjsvd_/zvjsvd_'s algorithm
// runs on G with V as the preset matrix (the reference's iwork[0] != 0 mode, src/dvjsvd.c:88-96,
// src/zvjsvd.c:100-110): G R = U Sigma and V R = V, so A = U Sigma V^H with the FP64
// algorithm's accuracy and convergence test; its first sweep is checked for every pair at
// once (by the last Gram matrix, whose error is bounded, or by jsvd.cu's k_certify and k_confirm)
// and skipped when it would transform nothing.
// Measured, before (FP64 products by a library, FP64 sweeps, column-pair FP32 sweeps) and now:
// 1024 x 1024 real 139 and 20.4 ms, 4096 x 2048 complex 1517 and 251 to 260 ms (by machine).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <chrono>
#include <cstring>
#include <algorithm>
#include <vector>

#include <cuda_runtime.h>

#include "fp64tc.cuh"
#include "gram_bound.cuh"
#include "presweep.cuh"
#include "svd_core.cuh"
#include "vj_fp.cuh"
#include "vj_host.h"

namespace vj {

// defined in blockjac.cu: block sweeps with split-BF16x3 tensor-core products
bool block_sweeps_apply(bool cplx, long long m, long long n, long long ld);
size_t block_sweep_scratch(bool cplx, long long m, long long n, int inner);
long long block_sweep(bool cplx, int m, int n, float *Gr, float *Gi, long long ldg, float *Wr, float *Wi,
                      long long ldw, unsigned char *scratch, unsigned *stats, float tol, int inner, int terms,
                      bool fast, cudaStream_t s, float *mu);

// defined in colblk.cu: sweeps by small blocks of columns, a CTA per pair of blocks
int col_blocks(bool cplx, long long m, long long n);
long long col_block_sweep(bool cplx, int m, int n, float *Gr, float *Gi, float *Wr, float *Wi, float tol, unsigned *cnt,
                          cudaStream_t s, float *mu);

// defined in jsvd.cu
template <typename T, bool CPLX>
vj_fint svd_dev_entry(vj_fnat m, vj_fnat n, T *G, vj_fnat ldG, T *Gi, vj_fnat ldGi, T *V, vj_fnat ldV, T *Vi,
                      vj_fnat ldVi, T *eS, T *fS, const unsigned *js, unsigned stp, unsigned swp, int preset,
                      bool certified, cudaStream_t s);

__global__ void k_to_f32(const double *A, long long ld, long long rows, long long cols, int e, float *B)
{
  for (long long j = blockIdx.y; j < cols; j += gridDim.y)
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += (long long)gridDim.x * blockDim.x)
      B[j * rows + i] = __double2float_rn(scale2(A[j * ld + i], e));
}

template <typename T> __global__ void k_eye_p(T *V, long long ld, long long n, int diag)
{
  for (long long j = blockIdx.y; j < n; j += gridDim.y)
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
      V[j * ld + i] = (diag && i == j) ? (T)1 : (T)0;
}

__global__ void k_absmax(const double *A, long long ld, long long rows, long long cols, unsigned long long *out)
{
  unsigned long long mx = 0ull;
  for (long long j = blockIdx.y; j < cols; j += gridDim.y)
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += (long long)gridDim.x * blockDim.x) {
      const unsigned long long b = (unsigned long long)__double_as_longlong(A[j * ld + i]) & 0x7fffffffffffffffull;
      mx = (b > mx) ? b : mx;
    }
  for (int o = 16; o >= 1; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = (w > mx) ? w : mx;
  }
  if ((threadIdx.x & 31) == 0 && mx)
    atomicMax(out, mx);
}

// Vector of 16 bytes: 4 floats or 2 doubles.
template <typename T> struct vec16;
template <> struct vec16<float> { using V = float4; static constexpr int E = 4; };
template <> struct vec16<double> { using V = double2; static constexpr int E = 2; };

// CTA-wide sums of a, b, cr, ci (up to 512 threads) into thread 0
template <typename T> __device__ void block_sum4(T &a, T &b, T &cr, T &ci, T (*red)[16])
{
  for (int o = 16; o >= 1; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    cr += __shfl_xor_sync(0xffffffffu, cr, o);
    ci += __shfl_xor_sync(0xffffffffu, ci, o);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[0][w] = a;
    red[1][w] = b;
    red[2][w] = cr;
    red[3][w] = ci;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = b = cr = ci = 0;
    for (int j = 0; j < (int)(blockDim.x >> 5); ++j) {
      a += red[0][j];
      b += red[1][j];
      cr += red[2][j];
      ci += red[3][j];
    }
  }
}

// rotate columns (x, y); with swap the rotated y goes to x's place and the rotated x to y's
template <typename T, bool CPLX, bool SHRT>
__device__ void rot_cols_(int rows, T *xr, T *xi, T *yr, T *yi, const Rot<T> &c)
{
  T *dxr = c.swap ? yr : xr, *dxi = c.swap ? yi : xi, *dyr = c.swap ? xr : yr, *dyi = c.swap ? xi : yi;
  Rot<T> k = c;
  k.shrt = SHRT;  // a compile-time form inside the loop
  unscaled_form(k);
  for (int i = threadIdx.x; i < rows; i += blockDim.x) {
    T pr = xr[i], qr = yr[i], pi = 0, qi = 0;
    if (CPLX) {
      pi = xi[i];
      qi = yi[i];
    }
    rot_elem<T, CPLX>(k, pr, pi, qr, qi);
    dxr[i] = pr;
    dyr[i] = qr;
    if (CPLX) {
      dxi[i] = pi;
      dyi[i] = qi;
    }
  }
}
template <typename T, bool CPLX>
__device__ void rot_cols(int rows, T *xr, T *xi, T *yr, T *yi, const Rot<T> &c)
{
  if (has_scales<T>() && c.shrt)
    rot_cols_<T, CPLX, true>(rows, xr, xi, yr, yi, c);
  else
    rot_cols_<T, CPLX, false>(rows, xr, xi, yr, yi, c);
}

// The same for the register kernels, U rows per thread loaded before any is stored: a
// store may alias a later load as far as the compiler knows, so the loop above waits for one
// memory round trip per row of the thread, which is most of a step at the small sizes the
// register kernels serve (U = 4 real / 2 complex: 1024 x 1024 real FP32 sweeps 92 -> 80 ms).
template <typename T, bool CPLX, bool SHRT, int U>
__device__ void rot_cols_batched_(int rows, T *xr, T *xi, T *yr, T *yi, const Rot<T> &c)
{
  T *dxr = c.swap ? yr : xr, *dxi = c.swap ? yi : xi, *dyr = c.swap ? xr : yr, *dyi = c.swap ? xi : yi;
  Rot<T> k = c;
  k.shrt = SHRT;
  unscaled_form(k);
  const int nt = (int)blockDim.x;
  for (int i0 = threadIdx.x; i0 < rows; i0 += U * nt) {
    T pr[U], qr[U], pi[U], qi[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * nt;
      pr[u] = qr[u] = pi[u] = qi[u] = (T)0;
      if (i < rows) {
        pr[u] = xr[i];
        qr[u] = yr[i];
        if (CPLX) {
          pi[u] = xi[i];
          qi[u] = yi[i];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * nt;
      if (i < rows) {
        rot_elem<T, CPLX>(k, pr[u], pi[u], qr[u], qi[u]);
        dxr[i] = pr[u];
        dyr[i] = qr[u];
        if (CPLX) {
          dxi[i] = pi[u];
          dyi[i] = qi[u];
        }
      }
    }
  }
}
template <typename T, bool CPLX, int U>
__device__ void rot_cols_batched(int rows, T *xr, T *xi, T *yr, T *yi, const Rot<T> &c)
{
  if (has_scales<T>() && c.shrt)
    rot_cols_batched_<T, CPLX, true, U>(rows, xr, xi, yr, yi, c);
  else
    rot_cols_batched_<T, CPLX, false, U>(rows, xr, xi, yr, yi, c);
}

// this thread's share of c = g_p^H g_q and, with NORMS, of |g_p|^2 and |g_q|^2
template <typename T, bool CPLX, bool NORMS>
__device__ __forceinline__ void pair_dots(int m, const T *gpr, const T *gqr, const T *gpi, const T *gqi, T &a, T &b,
                                          T &cr, T &ci)
{
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const T xr = gpr[i], yr = gqr[i];
    if (NORMS) {
      a = fma(xr, xr, a);
      b = fma(yr, yr, b);
    }
    cr = fma(xr, yr, cr);
    if (CPLX) {
      const T xi = gpi[i], yi = gqi[i];
      if (NORMS) {
        a = fma(xi, xi, a);
        b = fma(yi, yi, b);
      }
      cr = fma(xi, yi, cr);
      ci = fma(xr, yi, ci);
      ci = fma(-xi, yr, ci);
    }
  }
}
// One pivot step of one-sided Jacobi (Hestenes) with plain dot products, FP32 or FP64, on
// planar G (m x n) and W (n x n): CTA k takes pair (p, q) = row st of the pivot table,
// forms a = |g_p|^2, b = |g_q|^2, c = g_p^H g_q (per-thread partial sums and a block
// tree) and rotates columns p and q of G and W (hestenes, presweep.cuh). Any m; G is read
// twice. dsc, nrm: the column scales and tracked norms of the FP64 sweeps (Rot and
// tracked_norms, presweep.cuh), or nullptr.
template <typename T, bool CPLX>
__global__ void __launch_bounds__(256) k_presweep(int m, int n, T *Gr, long long ldr, T *Gi, long long ldi, T *Wr,
                                                  long long lwr, T *Wi, long long lwi, const unsigned *js, int st,
                                                  T tol, unsigned *cnt, T *dsc, T *nrm)
{
  __shared__ T red[4][16];
  __shared__ Rot<T> rs;
  pdl_enter();
  const int k = blockIdx.x;
  const unsigned p = js[(size_t)st * n + 2 * k], q = js[(size_t)st * n + 2 * k + 1];
  T *gpr = Gr + (size_t)p * ldr, *gqr = Gr + (size_t)q * ldr;
  T *gpi = CPLX ? Gi + (size_t)p * ldi : nullptr, *gqi = CPLX ? Gi + (size_t)q * ldi : nullptr;
  T nab[2];
  tracked_norms(nrm, p, q, nab);
  const bool norms = nab[0] < (T)0;
  T a = 0, b = 0, cr = 0, ci = 0;
  if (norms)
    pair_dots<T, CPLX, true>(m, gpr, gqr, gpi, gqi, a, b, cr, ci);
  else
    pair_dots<T, CPLX, false>(m, gpr, gqr, gpi, gqi, a, b, cr, ci);
  block_sum4(a, b, cr, ci, red);
  if (threadIdx.x == 0)
    pair_rotation(a, b, cr, ci, tol, cnt, dsc, p, q, &rs, nrm, nab);
  __syncthreads();
  const Rot<T> c = rs;
  if (!c.go)
    return;
  rot_cols<T, CPLX>(m, gpr, gpi, gqr, gqi, c);
  rot_cols<T, CPLX>(n, Wr + (size_t)p * lwr, CPLX ? Wi + (size_t)p * lwi : nullptr, Wr + (size_t)q * lwr,
                    CPLX ? Wi + (size_t)q * lwi : nullptr, c);
}

// the dot products of the register-resident column vectors of k_presweep_reg
template <typename T, bool CPLX, int R, bool NORMS, typename V>
__device__ __forceinline__ void reg_dots(const V (&xr)[R], const V (&yr)[R], const V (&xi)[R], const V (&yi)[R], T &a,
                                         T &b, T &cr, T &ci)
{
  constexpr int E = vec16<T>::E;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const T *X = reinterpret_cast<const T *>(&xr[r]), *Y = reinterpret_cast<const T *>(&yr[r]);
    const T *Xi = reinterpret_cast<const T *>(&xi[r]), *Yi = reinterpret_cast<const T *>(&yi[r]);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (NORMS) {
        a = fma(X[e], X[e], a);
        b = fma(Y[e], Y[e], b);
      }
      cr = fma(X[e], Y[e], cr);
      if (CPLX) {
        if (NORMS) {
          a = fma(Xi[e], Xi[e], a);
          b = fma(Yi[e], Yi[e], b);
        }
        cr = fma(Xi[e], Yi[e], cr);
        ci = fma(X[e], Yi[e], ci);
        ci = fma(-Xi[e], Y[e], ci);
      }
    }
  }
}

// the rotation of the register-resident column vectors of k_presweep_reg, written back
template <typename T, bool CPLX, int R, int NT, bool SHRT, typename V>
__device__ __forceinline__ void rot_regs(V (&xr)[R], V (&yr)[R], V (&xi)[R], V (&yi)[R], int mv, Rot<T> k, V *gpr,
                                         V *gqr, V *gpi, V *gqi)
{
  constexpr int E = vec16<T>::E;
  k.shrt = SHRT;
  unscaled_form(k);
  V *dpr = k.swap ? gqr : gpr, *dqr = k.swap ? gpr : gqr, *dpi = k.swap ? gqi : gpi, *dqi = k.swap ? gpi : gqi;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = threadIdx.x + r * NT;
    if (i < mv) {
      T *X = reinterpret_cast<T *>(&xr[r]), *Y = reinterpret_cast<T *>(&yr[r]);
      T *Xi = reinterpret_cast<T *>(&xi[r]), *Yi = reinterpret_cast<T *>(&yi[r]);
#pragma unroll
      for (int e = 0; e < E; ++e) {
        T d0 = 0, d1 = 0;
        rot_elem<T, CPLX>(k, X[e], CPLX ? Xi[e] : d0, Y[e], CPLX ? Yi[e] : d1);
      }
      dpr[i] = xr[r];
      dqr[i] = yr[r];
      if (CPLX) {
        dpi[i] = xi[r];
        dqi[i] = yi[r];
      }
    }
  }
}

// resident CTAs per SM the FP64 register kernels are compiled for: a pivot step of a
// 1024-column matrix is 512 CTAs, one wave on 152 SMs at 4 per SM and two at 3 (at
// 1024 x 1024 real the FP64 sweeps took 61 ms with 4 per SM, 80 ms with 3); 0 (the FP32
// kernels) leaves the compiler's own register choice, as a bound without a minimum does
template <typename T, bool CPLX, int R, int NT> __host__ __device__ constexpr int presweep_min_ctas()
{
  return (sizeof(T) == 8 && NT == 256) ? ((CPLX && R == 2) ? 3 : 4) : 0;
}

// The same step with the two columns of G held in registers between the dot products and
// the rotation (one read and one write of G): thread t of NT owns the 16-byte vectors
// t + NT r, r < R, of each column, so m <= NT R E (E = 4 floats or 2 doubles per vector);
// m % E == 0 and 16-byte aligned columns.
// PW: W's two columns are loaded as 16-byte vectors with G's at the start, and rotated from
// registers (real FP32 data with 16-byte aligned columns of W); otherwise they are read
// after the rotation is known.
template <typename T, bool CPLX, int R, int NT, bool PW = false>
__global__ void __launch_bounds__(NT, presweep_min_ctas<T, CPLX, R, NT>()) k_presweep_reg(int m, int n, T *Gr, long long ldr, T *Gi, long long ldi,
                                                      T *Wr, long long lwr, T *Wi, long long lwi, const unsigned *js,
                                                      int st, T tol, unsigned *cnt, T *dsc, T *nrm)
{
  static_assert(!PW || (!CPLX && sizeof(T) == 4), "W prefetch: real FP32 data");
  using V = typename vec16<T>::V;
  constexpr int E = vec16<T>::E;
  __shared__ T red[4][16];
  __shared__ Rot<T> rs;
  pdl_enter();
  const int k = blockIdx.x;
  const unsigned p = js[(size_t)st * n + 2 * k], q = js[(size_t)st * n + 2 * k + 1];
  V *gpr = reinterpret_cast<V *>(Gr + (size_t)p * ldr), *gqr = reinterpret_cast<V *>(Gr + (size_t)q * ldr);
  V *gpi = CPLX ? reinterpret_cast<V *>(Gi + (size_t)p * ldi) : nullptr;
  V *gqi = CPLX ? reinterpret_cast<V *>(Gi + (size_t)q * ldi) : nullptr;
  const int mv = m / E;
  V xr[R], yr[R], xi[R], yi[R];
  T a = 0, b = 0, cr = 0, ci = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = threadIdx.x + r * NT;
    V z;
    T *zz = reinterpret_cast<T *>(&z);
#pragma unroll
    for (int e = 0; e < E; ++e)
      zz[e] = 0;
    xr[r] = (i < mv) ? gpr[i] : z;
    yr[r] = (i < mv) ? gqr[i] : z;
    if (CPLX) {
      xi[r] = (i < mv) ? gpi[i] : z;
      yi[r] = (i < mv) ? gqi[i] : z;
    }
  }
  // W's columns (n <= m rows, so R vectors per thread cover them)
  const int nv = n / E;
  V *wpr = reinterpret_cast<V *>(Wr + (size_t)p * lwr), *wqr = reinterpret_cast<V *>(Wr + (size_t)q * lwr);
  V wp[PW ? R : 1], wq[PW ? R : 1];
  if constexpr (PW) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = threadIdx.x + r * NT;
      V z;
      T *zz = reinterpret_cast<T *>(&z);
#pragma unroll
      for (int e = 0; e < E; ++e)
        zz[e] = 0;
      wp[r] = (i < nv) ? wpr[i] : z;
      wq[r] = (i < nv) ? wqr[i] : z;
    }
  }
  // (the tracked norms are read after the column loads were issued: their latencies overlap)
  T nab[2];
  tracked_norms(nrm, p, q, nab);
  const bool norms = nab[0] < (T)0;
  if (norms)
    reg_dots<T, CPLX, R, true>(xr, yr, xi, yi, a, b, cr, ci);
  else
    reg_dots<T, CPLX, R, false>(xr, yr, xi, yi, a, b, cr, ci);
  block_sum4(a, b, cr, ci, red);
  if (threadIdx.x == 0)
    pair_rotation(a, b, cr, ci, tol, cnt, dsc, p, q, &rs, nrm, nab);
  __syncthreads();
  const Rot<T> c = rs;
  if (!c.go)
    return;
  if (has_scales<T>() && c.shrt)
    rot_regs<T, CPLX, R, NT, true>(xr, yr, xi, yi, mv, c, gpr, gqr, gpi, gqi);
  else
    rot_regs<T, CPLX, R, NT, false>(xr, yr, xi, yi, mv, c, gpr, gqr, gpi, gqi);
  if constexpr (PW)
    rot_regs<T, CPLX, R, NT, false>(wp, wq, wp, wq, nv, c, wpr, wqr, wpr, wqr);
  else
    rot_cols_batched<T, CPLX, CPLX ? 2 : 4>(n, Wr + (size_t)p * lwr, CPLX ? Wi + (size_t)p * lwi : nullptr,
                                            Wr + (size_t)q * lwr, CPLX ? Wi + (size_t)q * lwi : nullptr, c);
}

static dim3 grid2(long long rows, long long cols)
{
  long long gx = (rows + 255) / 256;
  if (gx > 32)
    gx = 32;
  long long gy = cols < 65535 ? cols : 65535;
  return dim3((unsigned)gx, (unsigned)(gy > 0 ? gy : 1));
}

template <typename T> __global__ void k_fill(T *x, int n, T v)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] = v;
}

// columns j of planar G (m x n) and W (n x n) times their scale dsc[j] (those != 1)
template <typename T, bool CPLX>
__global__ void k_apply_scales(int m, int n, T *Gr, long long ldr, T *Gi, long long ldi, T *Wr, long long lwr, T *Wi,
                               long long lwi, const T *dsc)
{
  for (int j = blockIdx.y; j < n; j += gridDim.y) {
    const T d = dsc[j];
    if (d == (T)1)
      continue;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (long long)m + n;
         i += (long long)gridDim.x * blockDim.x) {
      const bool g = i < m;
      const long long r = g ? i : i - m;
      T *pr = g ? Gr + (size_t)j * ldr + r : Wr + (size_t)j * lwr + r;
      *pr *= d;
      if (CPLX) {
        T *pi = g ? Gi + (size_t)j * ldi + r : Wi + (size_t)j * lwi + r;
        *pi *= d;
      }
    }
  }
}

// one sweep of presweep steps (stp launches); returns the number of rotations or < 0, and
// in *mu the largest |cos| of a rotated pair. With dsc (n entries of scratch) the columns
// carry scales during the sweep (Rot, presweep.cuh), multiplied into G and W at its end; with nrm
// (n entries) the squared column norms are tracked through the sweep (tracked_norms).
template <typename T, bool CPLX>
static long long presweep(int m, int n, T *Gr, long long ldr, T *Gi, long long ldi, T *Wr, long long lwr, T *Wi,
                          long long lwi, const unsigned *js, unsigned stp, T tol, unsigned *cnt, cudaStream_t s,
                          float *mu, T *dsc = nullptr, T *nrm = nullptr)
{
  constexpr int E = vec16<T>::E;
  const bool al = !(m % E) && !((ldr * (long long)sizeof(T)) % 16) && !((uintptr_t)Gr % 16) &&
                  (!CPLX || (!((ldi * (long long)sizeof(T)) % 16) && !((uintptr_t)Gi % 16)));
  if (cudaMemsetAsync(cnt, 0, 8, s) != cudaSuccess)
    return -1;
  if (dsc)
    k_fill<T><<<(n + 255) / 256, 256, 0, s>>>(dsc, n, (T)1);
  if (nrm)
    k_fill<T><<<(n + 255) / 256, 256, 0, s>>>(nrm, n, (T)-1);
  const unsigned nb = (unsigned)(n / 2);
  const long long cap = 256LL * E;  // rows per register vector slot
  void (*k)(int, int, T *, long long, T *, long long, T *, long long, T *, long long, const unsigned *, int, T,
            unsigned *, T *, T *) = k_presweep<T, CPLX>;
  int nt = 256;
  // register-resident columns: up to 2 vectors per thread and plane with 256 threads, then
  // (FP32) 2 vectors with 512 threads; beyond that the FP64 kernel's register use would
  // leave too few CTAs per SM to keep the FP64 pipe busy, and the two-pass kernel is
  // faster (measured at 4096x2048)
  if (al && m <= cap)
    k = k_presweep_reg<T, CPLX, 1, 256>;
  else if (al && m <= 2 * cap)
    k = k_presweep_reg<T, CPLX, 2, 256>;
  else if (al && sizeof(T) == 4 && m <= 4 * cap) {
    k = k_presweep_reg<T, CPLX, 2, 512>;
    nt = 512;
  }
  // real FP32 with 16-byte aligned columns of W: the variant that loads W with G
  if constexpr (!CPLX && sizeof(T) == 4) {
    const bool alw = !(n % E) && !((lwr * (long long)sizeof(T)) % 16) && !((uintptr_t)Wr % 16);
    if (alw && al && m <= cap)
      k = k_presweep_reg<T, CPLX, 1, 256, true>;
    else if (alw && al && m <= 2 * cap)
      k = k_presweep_reg<T, CPLX, 2, 256, true>;
    else if (alw && al && m <= 4 * cap)
      k = k_presweep_reg<T, CPLX, 2, 512, true>;
  }
  for (unsigned st = 0; st < stp; ++st)
    if (host::launch_pdl(k, dim3(nb), dim3(nt), 0, s, m, n, Gr, ldr, Gi, ldi, Wr, lwr, Wi, lwi, js, (int)st, tol,
                         cnt, dsc, nrm) != cudaSuccess)
      return -1;
  if (dsc)
    k_apply_scales<T, CPLX><<<grid2(m + n, n), 256, 0, s>>>(m, n, Gr, ldr, Gi, ldi, Wr, lwr, Wi, lwi, dsc);
  unsigned hc[2] = {0u, 0u};
  if (cudaGetLastError() != cudaSuccess || cudaMemcpyAsync(hc, cnt, 8, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return -1;
  memcpy(mu, &hc[1], 4);
  return (long long)hc[0];
}

// the plain Hestenes rotation of npairs disjoint pairs (2 npairs column indices at pairs)
template <bool CPLX>
static bool rotate_pairs(int m, int n, double *Gr, long long ldr, double *Gi, long long ldi, double *Vr, long long lvr,
                         double *Vi, long long lvi, const unsigned *pairs, int npairs, double tol, unsigned *cnt,
                         cudaStream_t s)
{
  double *none = nullptr;
  return cudaMemsetAsync(cnt, 0, 8, s) == cudaSuccess &&
         host::launch_pdl(k_presweep<double, CPLX>, dim3((unsigned)npairs), dim3(256), 0, s, m, n, Gr, ldr, Gi, ldi, Vr,
                          lvr, Vi, lvi, pairs, 0, tol, cnt, none, none) == cudaSuccess;
}

// squared 2-norms of the columns of planar G (one CTA per column)
template <bool CPLX>
__global__ void __launch_bounds__(256) k_colnorm2(int m, const double *Gr, long long ldr, const double *Gi,
                                                  long long ldi, double *out)
{
  __shared__ double red[8];
  const int j = blockIdx.x;
  double a = 0;
  for (int i = threadIdx.x; i < m; i += 256) {
    const double x = Gr[(size_t)j * ldr + i];
    a = fma(x, x, a);
    if (CPLX) {
      const double y = Gi[(size_t)j * ldi + i];
      a = fma(y, y, a);
    }
  }
  for (int o = 16; o >= 1; o >>= 1)
    a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0)
    red[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    a = 0;
    for (int w = 0; w < 8; ++w)
      a += red[w];
    out[j] = a;
  }
}

// B[:, j] = A[:, perm[j]] (rows x n, B with leading dimension rows)
__global__ void k_gather_cols(int rows, int n, const double *A, long long lda, const int *perm, double *B)
{
  for (int j = blockIdx.y; j < n; j += gridDim.y)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x)
      B[(size_t)j * rows + i] = A[(size_t)perm[j] * lda + i];
}

// squared 2-norms of the columns of planar FP32 G (one CTA per column): the order key of
// the orthonormalisation below
template <bool CPLX>
__global__ void __launch_bounds__(256) k_colnorm2_f32(int m, const float *Gr, const float *Gi, double *out)
{
  __shared__ double red[8];
  const int j = blockIdx.x;
  double a = 0;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const double x = Gr[(size_t)j * m + i];
    a = fma(x, x, a);
    if (CPLX) {
      const double y = Gi[(size_t)j * m + i];
      a = fma(y, y, a);
    }
  }
  for (int o = 16; o >= 1; o >>= 1)
    a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0)
    red[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    a = 0;
    for (int w = 0; w < 8; ++w)
      a += red[w];
    out[j] = a;
  }
}

// planar complex n x n matrix in FP64 (im null: real data), leading dimension n
struct Mat {
  double *re, *im;
};

// T[:, j] = W[:, perm[j]] widened to FP64
__global__ void k_widen_cols(int n, const float *W, const int *perm, double *T)
{
  for (int j = blockIdx.y; j < n; j += gridDim.y)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
      T[(size_t)j * n + i] = (double)W[(size_t)perm[j] * n + i];
}

// what an all-pairs kernel finds
struct PairStats {
  unsigned long long cosmax, cosbound;  // largest |cos| and largest upper bound of one (bits of doubles)
  double f2;                            // squared Frobenius norm of the rotation generator
  unsigned long long rowmax;            // its largest row sum (bits of a double)
  unsigned long long genmax, factmax;   // its largest entry in scaled form; that of the factor of G (bits)
  unsigned over, skipped;               // pairs above the tolerance; of those, not in the generator
  unsigned listed;                      // the latter again, as they are listed
};
// v into *p when larger (bits of non-negative doubles); the plain read spares most of the atomics
__device__ __forceinline__ void stat_max(unsigned long long *p, double v)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  if (b > *(volatile unsigned long long *)p)
    atomicMax(p, b);
}

// Kernels on the lower triangle of an n x n Hermitian matrix and its mirror, 32 x 32 tiles:
// thread (x, y) takes rows i = 32 blockIdx.x + x of columns j = 32 blockIdx.y + y + 8 k; f(i, j,
// diagonal) returns the mirror's value, which goes through shared memory and is stored by
// put(j, i, value) with its row j along the threads.
template <typename F, typename P> __device__ void lower_tiles(int n, F f, P put)
{
  __shared__ double2 t[32][33];
  const int bi = blockIdx.x, bj = blockIdx.y;
  if (bj > bi)
    return;
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int i = bi * 32 + threadIdx.x, j = bj * 32 + k;
    if (i < n && j < n && i >= j)
      t[k][threadIdx.x] = f(i, j);
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int j = bj * 32 + threadIdx.x, i = bi * 32 + k;
    if (i < n && j < n && i > j)
      put(j, i, t[threadIdx.x][k]);
  }
}

// M = -(strict upper triangle + half of the diagonal of E), E = H - I from H's lower triangle; the
// largest |E_ij| into st->cosmax
__global__ void __launch_bounds__(256) k_neg_upper(int n, Mat H, Mat M, PairStats *st)
{
  double mx = 0;
  lower_tiles(
      n,
      [&](int i, int j) {
        const size_t o = (size_t)j * n + i;
        const double re = H.re[o] - ((i == j) ? 1.0 : 0.0), im = (H.im && i != j) ? H.im[o] : 0.0;
        // (a NaN must not pass for a small value)
        const double a = fabs(re) + fabs(im);
        mx = (a <= 1e300) ? fmax(mx, a) : 1e300;
        M.re[o] = (i == j) ? -0.5 * re : 0.0;
        if (M.im)
          M.im[o] = 0.0;
        return make_double2(-re, im);
      },
      [&](int j, int i, double2 v) {
        M.re[(size_t)i * n + j] = v.x;
        if (M.im)
          M.im[(size_t)i * n + j] = v.y;
      });
  for (int o = 16; o >= 1; o >>= 1)
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (threadIdx.x == 0)
    stat_max(&st->cosmax, mx);
}

// The generator K of the rotation exp(K) that makes the columns of G orthogonal to first order,
// from the lower triangle of the Gram matrix H of the columns times 2^-e_j: K_ij = h_ij / (h_jj -
// h_ii) in the columns' true lengths, stored as K~_ij = 2^(e_i - e_j) K_ij (the factor of column i
// of length about 1 in column j of length about 1: a few times the cosine at most where the lengths
// differ, the cosine over the squared lengths' relative difference, up to 2^-6, where they nearly
// agree; st->genmax: the largest of them). Pairs with |cos| below `tol` / 4 are left alone; pairs with |K_ij| > 2^-6 (nearly
// equal lengths) too: they are counted, and the first `cap` of them go to list. rows: the row sums of
// |K_ij|. hb: bound of the error of each real sum in a Gram entry (1e300: none, no certificate).
__global__ void __launch_bounds__(256) k_generator(int n, Mat H, const int *e, Mat Kt, double tol, double hb,
                                                   PairStats *st, double *rows, uint2 *list, unsigned cap)
{
  double cm = 0, cb = 0, f2 = 0, km = 0;
  unsigned over = 0, skipped = 0;
  lower_tiles(
      n,
      [&](int i, int j) {
        const size_t o = (size_t)j * n + i;
        double2 kij = make_double2(0, 0), kji = kij;
        if (i != j) {
          const double hr = H.re[o], him = H.im ? H.im[o] : 0.0;
          const double hi = H.re[(size_t)i * n + i], hj = H.re[(size_t)j * n + j];
          if (hi > 0 && hj > 0) {
            const double a = H.im ? hypot(hr, him) : fabs(hr), ri = rsqrt(hi), rj = rsqrt(hj);
            const double c = a * (ri * rj);
            cm = (c <= 2.0) ? fmax(cm, c) : 2.0;  // (a NaN counts as large)
            cb = (c <= 2.0) ? fmax(cb, oz::cosine_bound(a, ri, rj, hb, H.im != nullptr)) : 2.0;
            over += (c > tol) ? 1u : 0u;
            if (c > 0.25 * tol) {
              // d = e_j - e_i: denominators h_jj 4^d - h_ii and h_jj - h_ii 4^-d
              const int d = max(-500, min(500, e[j] - e[i]));
              const double di = scalbn(hj, 2 * d) - hi, dj = hj - scalbn(hi, -2 * d);
              // |K_ij| = a 2^d / |di|
              const double k = scalbn(a, d);
              if (k <= 0.015625 * fabs(di)) {
                kij = make_double2(hr / di, him / di);
                kji = make_double2(-hr / dj, him / dj);
                km = fmax(km, a / fmin(fabs(di), fabs(dj)));
                const double q = k / fabs(di);
                f2 += 2.0 * q * q;
                if (q > 1e-7) {  // (n smaller ones add at most 1e-7 n to a row sum)
                  atomicAdd(rows + i, q);
                  atomicAdd(rows + j, q);
                }
              }
              else if (c > tol) {
                ++skipped;
                const unsigned at = atomicAdd(&st->listed, 1u);
                if (at < cap)
                  list[at] = make_uint2((unsigned)j, (unsigned)i);
              }
            }
          }
        }
        Kt.re[o] = kij.x;
        if (Kt.im)
          Kt.im[o] = kij.y;
        return kji;
      },
      [&](int j, int i, double2 v) {
        Kt.re[(size_t)i * n + j] = v.x;
        if (Kt.im)
          Kt.im[(size_t)i * n + j] = v.y;
      });
  for (int o = 16; o >= 1; o >>= 1) {
    cm = fmax(cm, __shfl_xor_sync(0xffffffffu, cm, o));
    cb = fmax(cb, __shfl_xor_sync(0xffffffffu, cb, o));
    km = fmax(km, __shfl_xor_sync(0xffffffffu, km, o));
    f2 += __shfl_xor_sync(0xffffffffu, f2, o);
    over += __shfl_xor_sync(0xffffffffu, over, o);
    skipped += __shfl_xor_sync(0xffffffffu, skipped, o);
  }
  if (threadIdx.x == 0 && blockIdx.y <= blockIdx.x) {
    stat_max(&st->cosmax, cm);
    stat_max(&st->cosbound, cb);
    stat_max(&st->genmax, km);
    if (f2 > 0)
      atomicAdd(&st->f2, f2);
    if (over)
      atomicAdd(&st->over, over);
    if (skipped)
      atomicAdd(&st->skipped, skipped);
  }
}

// the largest row sum of k_generator's rows
__global__ void __launch_bounds__(1024) k_rowmax(int n, const double *rows, PairStats *st)
{
  double m = 0;
  for (int i = threadIdx.x; i < n; i += 1024)
    m = fmax(m, rows[i]);
  for (int o = 16; o >= 1; o >>= 1)
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0)
    stat_max(&st->rowmax, m);
}

// y = a x + b y (y := a x when b is 0), n elements
__global__ void k_lincomb(long long n, double a, const double *x, double b, double *y)
{
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = (b == 0.0) ? a * x[i] : fma(a, x[i], b * y[i]);
}

// From the odd and even parts O~, E~ of exp(K) - I in scaled form (E may be empty): O~ := O~ + E~ (for
// the columns of G), and N = exp(K) - I in true form (for V), whose two entries of a pair both
// come from the scaled entry that is divided by the ratio of the lengths, by the parts' symmetry
// (O^H = -O, E^H = E): the other one would be multiplied by it, errors included. The largest |entry| of
// the new O~ into st->factmax.
__global__ void __launch_bounds__(256) k_exp_parts(int n, Mat O, Mat E, const int *e, Mat N, PairStats *st)
{
  __shared__ double2 so[32][33], se[32][33];
  double mx = 0;
  auto large = [&](const double2 &v) {
    const double a = fmax(fabs(v.x), fabs(v.y));
    mx = (v.x == v.x && v.y == v.y) ? fmax(mx, a) : 1e300;  // (a NaN must not pass for a small value)
  };
  const int bi = blockIdx.x, bj = blockIdx.y;
  if (bj > bi)
    return;
  auto get = [&](const Mat &M, size_t o) {
    return M.re ? make_double2(M.re[o], M.im ? M.im[o] : 0.0) : make_double2(0.0, 0.0);
  };
  // the tile's mirror: entries (j, i), rows j along the threads
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int j = bj * 32 + threadIdx.x, i = bi * 32 + k;
    if (i < n && j < n && i > j) {
      const size_t o = (size_t)i * n + j;
      so[threadIdx.x][k] = get(O, o);
      se[threadIdx.x][k] = get(E, o);
    }
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int i = bi * 32 + threadIdx.x, j = bj * 32 + k;
    if (i < n && j < n && i >= j) {
      const size_t o = (size_t)j * n + i;
      const double2 a = get(O, o), b = get(E, o);
      double2 x = make_double2(a.x + b.x, a.y + b.y), y = make_double2(0, 0);
      large(x);
      O.re[o] = x.x;
      if (O.im)
        O.im[o] = x.y;
      if (i != j) {
        const double2 c = so[k][threadIdx.x], f = se[k][threadIdx.x];
        so[k][threadIdx.x] = make_double2(c.x + f.x, c.y + f.y);
        large(so[k][threadIdx.x]);
        const int d = max(-2000, min(2000, e[j] - e[i]));
        if (d <= 0) {
          y = make_double2(scalbn(b.x - a.x, d), scalbn(a.y - b.y, d));  // (j, i) from (i, j)
          x = make_double2(scalbn(x.x, d), scalbn(x.y, d));
        }
        else {
          x = make_double2(scalbn(f.x - c.x, -d), scalbn(c.y - f.y, -d));
          y = make_double2(scalbn(c.x + f.x, -d), scalbn(c.y + f.y, -d));
        }
        se[k][threadIdx.x] = y;
      }
      N.re[o] = x.x;
      if (N.im)
        N.im[o] = x.y;
    }
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int j = bj * 32 + threadIdx.x, i = bi * 32 + k;
    if (i < n && j < n && i > j) {
      const size_t o = (size_t)i * n + j;
      O.re[o] = so[threadIdx.x][k].x;
      N.re[o] = se[threadIdx.x][k].x;
      if (O.im) {
        O.im[o] = so[threadIdx.x][k].y;
        N.im[o] = se[threadIdx.x][k].y;
      }
    }
  }
  for (int o = 16; o >= 1; o >>= 1)
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (threadIdx.x == 0)
    stat_max(&st->factmax, mx);
}

// the exponents' range
__global__ void __launch_bounds__(1024) k_spread(const int *e, int n, int *out)
{
  __shared__ int lo, hi;
  if (threadIdx.x == 0)
    lo = hi = e[0];
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += 1024) {
    atomicMin(&lo, e[i]);
    atomicMax(&hi, e[i]);
  }
  __syncthreads();
  if (threadIdx.x == 0)
    *out = hi - lo;
}

// Y (+)= the entries of two forms of one product, each from the one with the smaller sum of its operands'
// row exponents (er, ec: its error)
__global__ void k_choose(int n, const double *X0, const int *er0, const int *ec0, const double *X1, const int *er1,
                         const int *ec1, int add, double *Y, long long ld)
{
  for (int j = blockIdx.y; j < n; j += gridDim.y)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      const double v = (er1[i] + ec1[j] < er0[i] + ec0[j] ? X1 : X0)[(size_t)j * n + i];
      double *const y = Y + j * ld + i;
      *y = add ? *y + v : v;
    }
}

static bool copy2d(double *dst, long long ldd, const double *src, long long lds, long long rows, long long cols,
                   cudaStream_t s)
{
  return cudaMemcpy2DAsync(dst, (size_t)ldd * 8, src, (size_t)lds * 8, (size_t)rows * 8, (size_t)cols,
                           cudaMemcpyDeviceToDevice, s) == cudaSuccess;
}

template <bool CPLX>
static vj_fint mixed_dev(vj_fnat m_, vj_fnat n_, double *G, vj_fnat ldG, double *Gi, vj_fnat ldGi, double *V,
                         vj_fnat ldV, double *Vi, vj_fnat ldVi, double *eS, double *fS, const unsigned *js,
                         unsigned stp, unsigned swp, unsigned stages, cudaStream_t s, unsigned *presweeps)
{
  const host::NearestRounding rn;
  const long long m = (long long)m_, n = (long long)n_;
  if (presweeps)
    presweeps[0] = presweeps[1] = 0;
  if (!n)
    return 0;
  // the FP64 phase checks the reference's shape rules (src/dvjsvd.c:43-68) itself; they are
  // checked first here too, so that nothing runs on arguments that phase would reject
  if (m_ < n_ || (m % 8))
    return -1;
  if ((n & 1) || ((n >> 1) % 8))
    return -2;
  if (m > 0x3fffffffLL)
    return VJ_ERR_ARG;
  if (!stages)
    stages = 2;
  if (!host::gpu_ready())
    return VJ_ERR_NO_GPU;
  const int P = CPLX ? 2 : 1;
  const size_t mn = (size_t)m * n, nn = (size_t)n * n;
  // FP32 stages: block sweeps on the tensor cores where the shape has whole blocks and at least 16
  // block pairs per step; else sweeps by small blocks of columns in one or two CTAs (colblk.cu)
  // where a pair of blocks fits in shared memory; else column-pair sweeps. Measured, FP32 stages: 1024
  // x 1024 real 54 ms by column pairs, 16 by small blocks, 44 on the tensor cores; 2048 x 1024
  // complex 50 by small blocks, 41 on the tensor cores; 4096 x 2048 real 115 and 102. VJ_BLOCK=0 in
  // the environment selects the column-pair sweeps, VJ_BLOCK=1 the tensor-core block sweeps wherever
  // the shape allows; VJ_BLOCK_TERMS (6 or 3) the terms of the split products, VJ_BLOCK_INNER the
  // inner Jacobi sweeps per block pair.
  const char *eb = getenv("VJ_BLOCK");
  const bool blk = !(eb && *eb == '0') && block_sweeps_apply(CPLX, m, n, m) &&
                   ((eb && *eb == '1') || n >= (CPLX ? 1024 : 2048));
  const int ncol = (!(eb && *eb == '0') && !blk) ? col_blocks(CPLX, m, n) : 0;
  const char *et = getenv("VJ_BLOCK_TERMS");
  const int terms = (et && atoi(et) == 3) ? 3 : 6;
  const char *ei = getenv("VJ_BLOCK_INNER");
  const int inner = (ei && atoi(ei) >= 1 && atoi(ei) <= 8) ? atoi(ei) : 1;
  const size_t blkb = blk ? ((block_sweep_scratch(CPLX, m, n, inner) + 255) & ~(size_t)255) : 0;
  // scratch: the FP32 copy of G and W (P m n and P n n floats); five P n n matrices of doubles; two
  // digit operands of the FP64 products (fp64tc.cuh), the first as large as the columns or rows
  // of a panel of G's rows take, the second as an n x n matrix takes, with their exponents; counters;
  // the block sweeps' own. The columns' gather before the finishing sweeps goes through the digits'
  // room. Panels: the digits of all of G's columns take 16 (real) or 64 bytes per element, and
  // operands have at most oz::MAX_ROWS rows, so more digits than that gather takes and 2 GiB are cut
  // and multiplied a panel of rows at a time (whole up to 11,000 x 11,000 real, and 4,194,304 x 16 in
  // four).
  const int ni = (int)n, mi = (int)m;
  const oz::Source sc{G, Gi, (long long)ldG, (long long)(CPLX ? ldGi : ldG), ni, mi, nullptr, 0, oz::COLS};
  const long long row_digits = oz::pad(n, 128) * P * P * 2 * oz::DIGITS;  // bytes per row of G's columns
  long long pr = (long long)(std::max(mn * 8, (size_t)1 << 31) / (size_t)row_digits);
  pr = std::min(pr, oz::MAX_ROWS);
  const int panel = (int)((pr >= m) ? m : std::max(pr / 128 * 128, 128ll));
  auto panel_rows = [&](int r0) { return mi - r0 < panel ? mi - r0 : panel; };
  // the rows of G from r0 on, as columns (against which K runs along the rows) or rows of an operand
  auto g_cols = [&](int r0) {
    oz::Source p = sc;
    p.re = G + r0;
    p.im = CPLX ? Gi + r0 : nullptr;
    p.len = panel_rows(r0);
    return p;
  };
  auto g_rows = [&](int r0, const int *x) {
    return oz::Source{G + r0, CPLX ? Gi + r0 : nullptr, sc.ldr, sc.ldi, panel_rows(r0), ni, x, -1, oz::ROWS};
  };
  const oz::Operand oc = oz::shape(g_cols(0), CPLX), orw = oz::shape(g_rows(0, nullptr), CPLX);
  const oz::Operand on = oz::shape(oz::Source{G, Gi, 0, 0, ni, ni, nullptr, 0, oz::PROD}, CPLX);
  auto up = [](size_t x) { return (x + 1023) & ~(size_t)1023; };
  const size_t f32b = up(P * (mn + nn) * 4), f64b = up(5 * P * nn * 8);
  const size_t d1b = up(std::max({(size_t)oc.bytes(), (size_t)orw.bytes(), (size_t)on.bytes(), mn * 8}));
  const size_t d2b = up(std::max((size_t)on.bytes(), nn * 8));
  const size_t e1b = up((size_t)2 * std::max({oc.np, orw.np, on.np}) * 4), e2b = up((size_t)(2 * on.np) * 4);
  const size_t exb = up((size_t)3 * on.np * 4), ekb = up((size_t)n * 4), vecb = up((size_t)n * 16), partb = up(oz::part_bytes());
  host::Staging &stg = host::staging3();
  if (!stg.reserve(f32b + f64b + d1b + d2b + e1b + e2b + exb + ekb + vecb + partb + 1024 + blkb))
    return VJ_ERR_NOMEM;
  unsigned char *at = reinterpret_cast<unsigned char *>(stg.ptr);
  auto take = [&](size_t bytes) {
    unsigned char *r = at;
    at += bytes;
    return r;
  };
  float *G32 = reinterpret_cast<float *>(take(f32b));
  float *W32 = G32 + P * mn;
  double *f64 = reinterpret_cast<double *>(take(f64b));
  unsigned char *d1 = take(d1b), *d2 = take(d2b);
  int *e1 = reinterpret_cast<int *>(take(e1b)), *e2 = reinterpret_cast<int *>(take(e2b));
  int *const exr = reinterpret_cast<int *>(take(exb)), *const exc = exr + on.np;  // of the products' other form
  int *ek = reinterpret_cast<int *>(take(ekb));  // exponents of G's columns
  double *vec = reinterpret_cast<double *>(take(vecb));
  unsigned char *const part = take(partb);  // the sums of products whose K is split over CTAs
  unsigned char *cells = take(1024);
  unsigned char *bscr = at;
  unsigned long long *cell = reinterpret_cast<unsigned long long *>(cells);
  unsigned *cnt = reinterpret_cast<unsigned *>(cell + 1);
  unsigned *gerr = cnt + 4;
  PairStats *st = reinterpret_cast<PairStats *>(cells + 256);
  Mat M[5];
  for (int k = 0; k < 5; ++k)
    M[k] = Mat{f64 + (size_t)k * P * nn, CPLX ? f64 + (size_t)k * P * nn + nn : nullptr};
  double *const Y = M[4].re;
  const dim3 tiles((unsigned)((n + 31) / 32), (unsigned)((n + 31) / 32)), tblk(32, 8);
  if (cudaMemsetAsync(gerr, 0, 4, s) != cudaSuccess)
    return VJ_ERR_CUDA;
  // the columns (for X^H X) or rows (for X Y) of an n x n X, or X as the right factor, cut into digits
  auto cut = [&](const oz::Source &src, unsigned char *d, int *e, oz::Operand &o) {
    o = oz::shape(src, CPLX);
    o.d = d;
    o.e = e;
    return oz::split(src, o, s) == cudaSuccess;
  };
  auto cut_cols = [&](const double *re, const double *im, long long ldr, long long ldi, oz::Operand &o) {
    return cut(oz::Source{re, im, ldr, ldi, ni, ni, nullptr, 0, oz::COLS}, d1, e1, o);
  };
  auto cut_rows = [&](const double *re, const double *im, long long ldr, long long ldi, const int *x, oz::Operand &o) {
    return cut(oz::Source{re, im, ldr, ldi, ni, ni, x, -1, oz::ROWS}, d1, e1, o);
  };
  auto cut_prod = [&](const Mat &X, const int *x, oz::Operand &o) {
    return cut(oz::Source{X.re, X.im, n, n, ni, ni, x, 1, oz::PROD}, d2, e2, o);
  };
  // H's lower triangle = X^H X of columns cut into o
  auto gram = [&](const oz::Operand &o, const Mat &H, int nd) {
    oz::Operand a = o;
    a.halves = 1;
    return oz::gemm(a, o, oz::Result{H.re, H.im, n, n, ni, ni, nullptr, 1, 0, 1}, nd, gerr, part, s) == cudaSuccess;
  };
  // X (+)= A B for an n x n X
  auto mult = [&](const oz::Operand &A, const oz::Operand &B, const Mat &X, int add, int nd) {
    return oz::gemm(A, B, oz::Result{X.re, X.im, n, n, ni, ni, nullptr, 1, add, 0}, nd, gerr, part, s) == cudaSuccess;
  };
  // Y (+)= Y B for V or W, n x n, B as its digits or, where the columns of A differ in length by more than
  // six bits, by itself. Then an entry of a short column of Y in the row of a long column of A is small,
  // and A V = U Sigma needs it to its own accuracy; the digits of Y's rows and B's columns
  // resolve it to that of their largest entries only. So the product is formed once more with K scaled
  // by the columns' lengths (ek), as it is for G, and each entry taken from the form that resolves it better.
  // t0, t1: for the two forms. (The mixed SVD of a 1024 x 1024 real matrix with columns over 12 decades 19.0
  // -> 19.7 ms, the columns of A V - U Sigma 1.8e-6 -> 2.6e-15 of their sigma.)
  bool graded = false;
  struct Square {
    double *re, *im;
    long long ldr, ldi;
  };
  auto mult_cols = [&](const Square &y, const Mat &B, const oz::Operand &b, const Mat &t0, const Mat &t1, int add, int nd) {
    oz::Operand A, o = b;
    if (!graded)
      return cut_rows(y.re, y.im, y.ldr, y.ldi, nullptr, A) &&
             oz::gemm(A, o, oz::Result{y.re, y.im, y.ldr, y.ldi, ni, ni, nullptr, 1, add, 0}, nd, gerr, part, s) ==
                 cudaSuccess;
    if (!cut_rows(y.re, y.im, y.ldr, y.ldi, nullptr, A) || !mult(A, o, t0, 0, nd) ||
        !cut(oz::Source{y.re, y.im, y.ldr, y.ldi, ni, ni, ek, -1, oz::ROWS}, d1, exr, A) ||
        !cut(oz::Source{B.re, B.im, n, n, ni, ni, ek, 1, oz::PROD}, d2, exc, o) || !mult(A, o, t1, 0, nd))
      return false;
    k_choose<<<grid2(n, n), 256, 0, s>>>(ni, t0.re, e1, e2, t1.re, exr, exc, add, y.re, y.ldr);
    if (CPLX)
      k_choose<<<grid2(n, n), 256, 0, s>>>(ni, t0.im, e1, e2, t1.im, exr, exc, add, y.im, y.ldi);
    return cudaGetLastError() == cudaSuccess && cut_prod(B, nullptr, o);
  };
  const Square sv{V, Vi, (long long)ldV, (long long)(CPLX ? ldVi : ldV)};
  // G (+)= G B (G's columns times 2^ej).
  // G's rows enter with their columns' 2^-x
  auto mult_g = [&](const int *x, const oz::Operand &B, const int *ej, int add, int nd) {
    for (int r0 = 0; r0 < mi; r0 += panel) {
      oz::Operand A;
      if (!cut(g_rows(r0, x), d1, e1, A) ||
          oz::gemm(A, B, oz::Result{G + r0, CPLX ? Gi + r0 : nullptr, sc.ldr, sc.ldi, panel_rows(r0), ni, ej, 1, add, 0},
                   nd, gerr, part, s) != cudaSuccess)
        return false;
    }
    return true;
  };
  // H's lower triangle = G^H G, the columns divided by their powers of two (left in e1)
  auto gram_g = [&](const Mat &H, int nd) {
    oz::Operand o = oc;
    o.e = e1;
    if (oz::split_exponents(sc, o, s) != cudaSuccess)
      return false;
    for (int r0 = 0; r0 < mi; r0 += panel) {
      const oz::Source p = g_cols(r0);
      o = oz::shape(p, CPLX);
      o.d = d1;
      o.e = e1;
      oz::Operand a = o;
      a.halves = 1;
      if (oz::split_digits(p, o, s) != cudaSuccess ||
          oz::gemm(a, o, oz::Result{H.re, H.im, n, n, ni, ni, nullptr, 0, r0 ? 1 : 0, 1}, nd, gerr, part, s) != cudaSuccess)
        return false;
    }
    return true;
  };
  // digits that a correction of relative size x needs: what nd digits leave out, about 2^(5 - 8 nd)
  // of a product of rows of length 1, stays below 2^-57
  auto digits = [](double x) {
    const int nd = (int)std::ceil((62.0 + std::log2(std::max(x, 1e-20))) / 8.0);
    return nd < 3 ? 3 : nd > 8 ? 8 : nd;
  };
  PairStats hst;
  auto read_stats = [&]() {
    return cudaGetLastError() == cudaSuccess &&
           cudaMemcpyAsync(&hst, st, sizeof(hst), cudaMemcpyDeviceToHost, s) == cudaSuccess &&
           cudaStreamSynchronize(s) == cudaSuccess;
  };
  auto asdbl = [](unsigned long long b) {
    double v;
    memcpy(&v, &b, 8);
    return v;
  };
  // sqrt(m)/2 units of FP32 roundoff (the reference's FP32 tolerance), at least 8 units
  const float tol = fmaxf(0.5f * sqrtf((float)m), 8.f) * 5.9604645e-8f;
  const unsigned maxsw = swp < 60u ? swp : 60u;
  unsigned total32 = 0;
  bool dropped = false;  // a stage's W was not near unitary
  // the wall-clock time of each phase is kept for vj_last_mixed_phases (every phase ends
  // with a stream synchronisation, so host time is device time here); with VJ_TRACE=1 it
  // also goes to stderr
  const bool trace = host::trace_enabled();
  auto now = [] { return std::chrono::steady_clock::now(); };
  auto t0 = now();
  double ms32 = 0, msgemm = 0;
  for (unsigned stage = 0; stage < stages; ++stage) {
    // 1. scale to max |g| in [1/2, 1) and round to FP32
    if (cudaMemsetAsync(cell, 0, 8, s) != cudaSuccess)
      return VJ_ERR_CUDA;
    k_absmax<<<grid2(m, n), 256, 0, s>>>(G, (long long)ldG, m, n, cell);
    if (CPLX)
      k_absmax<<<grid2(m, n), 256, 0, s>>>(Gi, (long long)ldGi, m, n, cell);
    unsigned long long mb[9] = {};
    if (!stage) {
      if (oz::row_exponents(sc, ek, s) != cudaSuccess)
        return VJ_ERR_CUDA;
      k_spread<<<1, 1024, 0, s>>>(ek, ni, reinterpret_cast<int *>(cell + 8));
    }
    if (cudaMemcpyAsync(mb, cell, sizeof(mb), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return VJ_ERR_CUDA;
    double amax;
    memcpy(&amax, &mb[0], 8);
    if (!stage) {
      int spread;
      memcpy(&spread, &mb[8], 4);
      graded = spread > 6;
    }
    if (!(amax <= 1.7976931348623157e308))
      return CPLX ? -92 : -80;
    if (amax == 0.0)
      break;
    int e = 0;
    (void)std::frexp(amax, &e);
    k_to_f32<<<grid2(m, n), 256, 0, s>>>(G, (long long)ldG, m, n, -e, G32);
    if (CPLX)
      k_to_f32<<<grid2(m, n), 256, 0, s>>>(Gi, (long long)ldGi, m, n, -e, G32 + mn);
    k_eye_p<float><<<grid2(n, n), 256, 0, s>>>(W32, n, n, 1);
    if (CPLX)
      k_eye_p<float><<<grid2(n, n), 256, 0, s>>>(W32 + nn, n, n, 0);
    // 2. FP32 sweeps until a sweep rotates nothing
    // (a sweep whose rotated pairs were all within 4x the tolerance ends the stage without
    // a confirming sweep: the stage is a preconditioner, the next one finishes the work;
    // a stage that another one follows also ends once a sweep rotates fewer than 0.7 of
    // all possible pairs: the first stage works on A rounded to FP32, where the directions
    // of singular values below FP32 resolution are noise that the next stage resolves
    // properly. At 0.5 the 1024 x 1024 real matrix takes one sweep more; at 0.9 and above the
    // FP64 phase of matrices with sigma over 6 decades and more takes a refinement or, at 1,
    // sweeps more.)
    unsigned sw = 0;
    const float stop = 4.f * tol;
    const long long nbk = n / (CPLX ? 32 : 64), hw = CPLX ? 32 : 64;
    const long long cbn = ncol ? n / (ncol / 2) : 0;
    const double every = ncol ? (double)(cbn / 2) * (double)(ncol / 2) * ((double)ncol + (double)(cbn - 1) * (double)(ncol / 2))
                         : blk ? (double)(nbk / 2) * inner * (double)hw * (CPLX ? (double)nbk * (double)(2 * hw - 1) : (double)(2 * hw - 1) + (double)(nbk - 1) * (double)hw)
                             : (double)stp * (double)(n / 2);
    for (; sw < maxsw; ++sw) {
      float mu = 0.f;
      const long long hc =
          blk ? block_sweep(CPLX, mi, ni, G32, CPLX ? G32 + mn : nullptr, m, W32, CPLX ? W32 + nn : nullptr, n, bscr,
                            cnt, tol, inner, terms, true, s, &mu)
          : ncol ? col_block_sweep(CPLX, mi, ni, G32, CPLX ? G32 + mn : nullptr, W32, CPLX ? W32 + nn : nullptr, tol, cnt,
                                   s, &mu)
              : presweep<float, CPLX>(mi, ni, G32, m, CPLX ? G32 + mn : nullptr, m, W32, n, CPLX ? W32 + nn : nullptr,
                                      n, js, stp, tol, cnt, s, &mu);
      if (hc < 0)
        return VJ_ERR_CUDA;
      if (trace)
        std::fprintf(stderr, "mixed SVD stage %u sweep %u: %lld rotations, max scaled |h_pq| %.3e\n", stage, sw, hc,
                     (double)mu);
      if (!hc)
        break;
      if (mu < stop || (stage + 1 < stages && (double)hc < 0.7 * every)) {
        ++sw;
        break;
      }
    }
    if (trace)
      std::fprintf(stderr, "mixed SVD stage %u: %u FP32 sweeps\n", stage, sw);
    total32 += sw;
    {
      const auto t1 = now();
      ms32 += std::chrono::duration<double, std::milli>(t1 - t0).count();
      t0 = t1;
    }
    if (!sw)
      break;  // already orthogonal to the FP32 level: later stages would change nothing
    // 3. W (FP64) made unitary, with its columns in ascending order of the norms of the FP32 G's
    //    columns: W^H W = I + E with E of the order of FP32 rounding, and the factor R of its
    //    Cholesky factorisation R^H R is I + U to first order, U the strict upper triangle of E
    //    and half its diagonal; W := W (I - U), repeated while the second-order terms left
    //    (about E^2) exceed FP64 rounding. Two rounds of a Gram product and a correction, all
    //    on the tensor cores, in place of a factorisation and a triangular solve on the FP64
    //    unit. The correction is upper triangular, so it mixes into each column of G Q only
    //    columns of smaller norm. (The first refinement below still meets scaled inner products
    //    of up to ~5e-3 at 4096 x 2048 complex with sigma down to 1e-8: the FP32 rounding of W's
    //    own entries couples large columns of G into small ones, which no orthonormalisation of
    //    W undoes; the descending order measured worse.)
    const Mat &T = M[0];
    std::vector<int> hp((size_t)n), he;  // (read by copies that the first round's read_stats waits for)
    {
      double *nrm = vec;
      int *perm = reinterpret_cast<int *>(vec + n);
      k_colnorm2_f32<CPLX><<<(unsigned)n, 256, 0, s>>>(mi, G32, CPLX ? G32 + mn : nullptr, nrm);
      std::vector<double> hn((size_t)n);
      if (cudaMemcpyAsync(hn.data(), nrm, (size_t)n * 8, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
          cudaStreamSynchronize(s) != cudaSuccess)
        return VJ_ERR_CUDA;
      for (int j = 0; j < ni; ++j)
        hp[(size_t)j] = j;
      std::stable_sort(hp.begin(), hp.end(), [&](int x, int y) { return hn[(size_t)x] < hn[(size_t)y]; });
      if (cudaMemcpyAsync(perm, hp.data(), (size_t)n * 4, cudaMemcpyHostToDevice, s) != cudaSuccess)
        return VJ_ERR_CUDA;
      k_widen_cols<<<grid2(n, n), 256, 0, s>>>(ni, W32, perm, T.re);
      if (CPLX)
        k_widen_cols<<<grid2(n, n), 256, 0, s>>>(ni, W32 + nn, perm, T.im);
      if (graded) {
        // the lengths of the columns that W makes (FP32 has no shorter ones than 2^-149)
        he.resize((size_t)n);
        for (int j = 0; j < ni; ++j) {
          const double x = hn[(size_t)hp[(size_t)j]];
          he[(size_t)j] = (x > 0) ? std::max(std::ilogb(x) / 2, -149) : -149;
        }
        if (cudaMemcpyAsync(ek, he.data(), (size_t)n * 4, cudaMemcpyHostToDevice, s) != cudaSuccess)
          return VJ_ERR_CUDA;
      }
    }
    oz::Operand oa, ob;
    // (the Gram matrices before the last need no more digits than their own second-order terms
    // justify: 4 give E to 1e-9, 6 to 1e-13; up to n = 256, where the digits cost less than the launches
    // and the wait of the round that they save, all 8: 16 x 16 real 1.54 -> 1.36 ms)
    int nd = (n <= 256) ? 8 : 4;
    for (int round = 0;; ++round) {
      if (!cut_cols(T.re, T.im, n, n, oa) || !gram(oa, M[1], nd) ||
          cudaMemsetAsync(st, 0, sizeof(PairStats), s) != cudaSuccess)
        return VJ_ERR_CUDA;
      k_neg_upper<<<tiles, tblk, 0, s>>>(ni, M[1], M[2], st);
      if (!read_stats())
        return VJ_ERR_CUDA;
      const double emax = asdbl(hst.cosmax), rn_ = std::sqrt((double)n);
      if (trace)
        std::fprintf(stderr, "mixed SVD stage %u: largest entry of W^H W - I %.2e\n", stage, emax);
      // (G and V are as the stages before left them: the FP64 phase takes it from there)
      dropped = !(emax < 0.03) || round == 8;
      if (dropped)
        break;
      if (!cut_prod(M[2], nullptr, ob) || !mult_cols(Square{T.re, T.im, n, n}, M[2], ob, M[3], M[4], 1, digits(emax)))
        return VJ_ERR_CUDA;
      const double next = std::max(emax * emax * rn_, nd == 4 ? 1e-9 : nd == 6 ? 1e-13 : 0.0);
      if (nd == 8 && next < 2e-17)
        break;
      nd = (next * next * rn_ < 2e-17) ? 8 : 6;
    }
    if (dropped) {
      total32 -= sw;
      break;
    }
    // 4. V <- V W (V_0 = I, so the first stage that rotates sets V = W), G <- G W; G's columns
    //    enter the product with their lengths' powers of two moved to the rows of W, so that the
    //    digits resolve every column of the result to its own length
    if (oz::row_exponents(sc, ek, s) != cudaSuccess)
      return VJ_ERR_CUDA;
    if (total32 == sw) {
      if (!copy2d(V, ldV, T.re, n, n, n, s) || (CPLX && !copy2d(Vi, ldVi, T.im, n, n, n, s)))
        return VJ_ERR_CUDA;
    }
    else if (!cut_prod(T, nullptr, ob) || !mult_cols(sv, T, ob, M[3], M[4], 0, 8))
      return VJ_ERR_CUDA;
    if (!cut_prod(T, ek, ob) || !mult_g(ek, ob, nullptr, 0, 8))
      return VJ_ERR_CUDA;
    {
      if (cudaStreamSynchronize(s) != cudaSuccess)
        return VJ_ERR_CUDA;
      const auto t1 = now();
      msgemm += std::chrono::duration<double, std::milli>(t1 - t0).count();
      t0 = t1;
    }
  }
  if (presweeps)
    presweeps[0] = total32;
  if (!total32) {
    // nothing was rotated (zero matrix, columns already orthogonal, or a first stage dropped): V := I
    k_eye_p<double><<<grid2(n, n), 256, 0, s>>>(V, (long long)ldV, n, 1);
    if (CPLX)
      k_eye_p<double><<<grid2(n, n), 256, 0, s>>>(Vi, (long long)ldVi, n, 0);
  }
  // 5. G's columns from FP32 to FP64 orthogonality, to half the reference's tolerance sqrt(m) eps / 2
  //    (pairs the reference would still rotate are rotated here), by refinements on the tensor
  //    cores: the Gram matrix of the columns to FP64 accuracy, the generator K of the rotation
  //    that makes them orthogonal to first order, N = exp(K) - I by its series, and G := G + G N,
  //    V := V + V N. What is left is of second order, so two refinements and the Gram matrix that
  //    confirms them replace the plain-dot FP64 sweeps (4096 x 2048 complex: 689 ms of sweeps).
  //    Pairs of nearly equal norms, whose rotation is not small, are rotated one by one before;
  //    whatever that and a refinement cannot improve goes to the sweeps, which run until no pair
  //    is left.
  bool certified = false;  // every cosine is below the finishing check's limit (k_generator's bound)
  if (total32 || dropped) {
    const double u = 1.1102230246251565e-16;
    const double tol64 = 0.5 * std::sqrt((double)m) * u;
    // the finishing check's limit (jsvd.cu, k_certify)
    const double lim = 0.9 * std::sqrt((double)m) * u - 16.0 * u;
    // swp caps the phase: what changes G and V, refinements, rotations of single pairs and sweeps, each
    // pass over the pairs counted (20 sweeps at most)
    unsigned sw64 = 0, passes = 0;
    bool sweeps = true;
    double before = 1e300;
    // (the entries of a Gram matrix of several panels are rounded sums of the panels')
    const double pan = (panel < mi) ? 4.0 * u * (double)((mi + panel - 1) / panel) : 0.0;
    constexpr unsigned MAXIT = 20;  // Gram matrices at most
    constexpr unsigned CAP = 8192;  // pairs of nearly equal norms that are rotated one by one
    uint2 *const list = reinterpret_cast<uint2 *>(d2);  // (free between the products)
    double *const rows = vec;
    const Mat &H = M[0], &K = M[1], &S = M[2], &Q = M[3], &E = M[4];
    // the Gram matrix with nd digits, the generator and what it finds; columns' exponents in ek
    auto survey = [&](int nd) {
      // what the 8 digits leave out of a real sum over the P m elements of K
      const double hb = (nd == 8) ? (double)((long long)P * m) * oz::OMITTED8 : 1e300;
      if (!gram_g(H, nd) || cudaMemcpyAsync(ek, e1, (size_t)n * 4, cudaMemcpyDeviceToDevice, s) != cudaSuccess ||
          cudaMemsetAsync(st, 0, sizeof(PairStats), s) != cudaSuccess ||
          cudaMemsetAsync(rows, 0, (size_t)n * 8, s) != cudaSuccess)
        return false;
      k_generator<<<tiles, tblk, 0, s>>>(ni, H, ek, K, tol64, hb, st, rows, list, CAP);
      k_rowmax<<<1, 1024, 0, s>>>(ni, rows, st);
      return read_stats();
    };
    for (unsigned it = 0; it < MAXIT && swp; ++it) {
      oz::Operand oa, ob;
      // (5 digits give the first cosines, of the order of FP32 rounding, to about 1e-11)
      const int nd = it ? 8 : 5;
      if (!survey(nd))
        return VJ_ERR_CUDA;
      const double cmax = asdbl(hst.cosmax), norm = std::min(std::sqrt(hst.f2), asdbl(hst.rowmax) + 1e-7 * (double)n);
      if (trace)
        std::fprintf(stderr, "mixed SVD refinement %u: %u pairs above the tolerance, max |cos| %.3e, |K| <= %.2e, %u left "
                     "out, %.1f ms since the phase began\n", it, hst.over, cmax, norm, hst.skipped,
                     std::chrono::duration<double, std::milli>(now() - t0).count());
      if (nd == 8 && !hst.over && cmax <= tol64) {
        sweeps = false;
        certified = (asdbl(hst.cosbound) + pan <= lim);
        break;
      }
      if (passes >= swp)
        break;
      if (hst.skipped) {
        // pairs of nearly equal norms: rotate disjoint ones of them by their angles and look again
        // (many of them are clusters, where the sweeps do better)
        std::vector<uint2> hl(hst.skipped < CAP ? hst.skipped : CAP);
        std::vector<unsigned> hp;
        std::vector<char> used((size_t)n, 0);
        if (hst.skipped > (unsigned)(n / 2) || hst.skipped > CAP || it + 1u == MAXIT ||
            cudaMemcpyAsync(hl.data(), list, hl.size() * sizeof(uint2), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
          break;
        std::sort(hl.begin(), hl.end(), [](const uint2 &x, const uint2 &y) { return x.x != y.x ? x.x < y.x : x.y < y.y; });
        for (const uint2 &q : hl)
          if (!used[q.x] && !used[q.y]) {
            used[q.x] = used[q.y] = 1;
            hp.push_back(q.x);
            hp.push_back(q.y);
          }
        unsigned *const dp = reinterpret_cast<unsigned *>(list);
        if (cudaMemcpyAsync(dp, hp.data(), hp.size() * 4, cudaMemcpyHostToDevice, s) != cudaSuccess ||
            !rotate_pairs<CPLX>(mi, ni, G, sc.ldr, Gi, sc.ldi, V, (long long)ldV, Vi, (long long)(CPLX ? ldVi : ldV), dp,
                                (int)(hp.size() / 2), tol64, cnt, s) ||
            cudaStreamSynchronize(s) != cudaSuccess)
          return VJ_ERR_CUDA;
        ++passes;
        continue;
      }
      if (!(norm <= 0.48) || !(cmax <= 0.25 * before))
        break;
      before = cmax;
      // The series below is to eighth order (|K|^9 / 9! stays below rounding up to 0.06); the
      // rotation by a larger K is that by K / 2^r, 2^r times. (4096 x 2048 complex with sigma down to
      // 1e-8, whose FP32 stages leave |K| = 0.2: 194 ms instead of 1016 with the sweeps)
      int reps = 1;
      while (norm > 0.06 * reps)
        reps *= 2;
      const double f = norm / reps;
      if (reps > 1)
        k_lincomb<<<(unsigned)std::min<size_t>((P * nn + 255) / 256, 4096), 256, 0, s>>>((long long)(P * nn), 1.0 / reps,
                                                                                      K.re, 0.0, K.re);
      // orders of the series: |K|^(order + 1) / (order + 1)! below 5e-17
      const int order = (f < 1e-8) ? 1 : (f < 6e-6) ? 2 : (f < 1.8e-4) ? 3 : (f < 1.4e-3) ? 4 : (f < 5.7e-3) ? 5 : (f < 0.015) ? 6 : (f < 0.03) ? 7 : 8;
      const long long np = (long long)(P * nn);
      const unsigned gl = (unsigned)((np + 255) / 256 < 4096 ? (np + 255) / 256 : 4096);
      // digits for the powers of K and for V N; for G N by the largest entry of its factor, which may be
      // any number of times the largest cosine (pairs of nearly equal lengths), below
      const double x = std::max(f, asdbl(hst.genmax) / reps);
      const int nk = digits(x * x), nv = digits(f);
      // exp(K) - I = E + O with E = K^2 (1/2! + K^2 (1/4! + ...)), O = K + K (K^2 (1/3! + K^2 (1/5! + ...)))
      static const double inv[9] = {1.0, 1.0, 1.0 / 2, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720, 1.0 / 5040, 1.0 / 40320};
      Mat Ev{nullptr, nullptr};
      if (order >= 2) {
        const Mat &P2 = H;  // K^2 takes the Gram matrix's place
        if (!cut_rows(K.re, K.im, n, n, nullptr, oa) || !cut_prod(K, nullptr, ob) || !mult(oa, ob, P2, 0, nk))
          return VJ_ERR_CUDA;
        Ev = E;
        const int te = order & ~1, to = (order - 1) | 1;  // the last even and odd orders
        const bool powers = te >= 4 || to >= 5;
        if (powers && !cut_rows(P2.re, P2.im, n, n, nullptr, oa))
          return VJ_ERR_CUDA;
        // X := c_last K^2, then X := c K^2 + K^2 X down to the order of `first`
        auto horner = [&](const Mat &X, int last, int first) {
          k_lincomb<<<gl, 256, 0, s>>>(np, inv[last], P2.re, 0.0, X.re);
          for (int k = last - 2; k >= first; k -= 2) {
            if (!cut_prod(X, nullptr, ob) || !mult(oa, ob, Q, 0, nk))
              return false;
            k_lincomb<<<gl, 256, 0, s>>>(np, inv[k], P2.re, 0.0, X.re);
            k_lincomb<<<gl, 256, 0, s>>>(np, 1.0, Q.re, 1.0, X.re);
          }
          return true;
        };
        if (!horner(E, te, 2) || (to >= 3 && !horner(S, to, 3)))
          return VJ_ERR_CUDA;
        if (to >= 3 && (!cut_rows(K.re, K.im, n, n, nullptr, oa) || !cut_prod(S, nullptr, ob) ||
                        !mult(oa, ob, K, 1, nk)))
          return VJ_ERR_CUDA;
      }
      k_exp_parts<<<tiles, tblk, 0, s>>>(ni, K, Ev, ek, Q, st);
      // (entries up to x in K~ make entries up to x (1 + n x) in exp(K~) - I while n x is below 1: where that
      // is the largest entry of K~ but for a tenth, the factor's own need not be waited for)
      double fact = asdbl(hst.genmax) / reps;
      if ((double)n * fact <= 0.1)
        fact *= 1.1;
      else {
        if (!read_stats())
          return VJ_ERR_CUDA;
        fact = asdbl(hst.factmax);
      }
      const int ng = digits(std::max(8.0 * cmax, fact));
      if (!cut_prod(K, nullptr, ob))
        return VJ_ERR_CUDA;
      for (int r = 0; r < reps; ++r)
        if (!mult_g(ek, ob, ek, 1, ng))
          return VJ_ERR_CUDA;
      if (!cut_prod(Q, nullptr, ob))
        return VJ_ERR_CUDA;
      for (int r = 0; r < reps; ++r)
        if (!mult_cols(sv, Q, ob, S, E, 1, graded ? std::max(nv, ng) : nv))
          return VJ_ERR_CUDA;
      ++sw64;
      ++passes;
    }
    const unsigned maxsw64 = std::min(swp - std::min(passes, swp), 20u);
    // A sweep whose rotated pairs all had |cos| <= 1e-11 leaves off-diagonal terms of the
    // order of their squares (times n / relative gap), far below the tolerance: its
    // confirming sweep is skipped, the reference's sweep below confirms.
    for (unsigned sw = 0; sweeps && sw < maxsw64; ++sw) {
      float mu = 0.f;
      const long long hc = presweep<double, CPLX>(mi, ni, G, (long long)ldG, Gi, (long long)(CPLX ? ldGi : ldG), V,
                                                  (long long)ldV, Vi, (long long)(CPLX ? ldVi : ldV), js, stp, tol64,
                                                  cnt, s, &mu, vec, vec + n);
      if (hc < 0)
        return VJ_ERR_CUDA;
      if (trace)
        std::fprintf(stderr, "mixed SVD FP64 sweep %u: %lld rotations, max |cos| %.3e, %.1f ms since the phase began\n",
                     sw, hc, (double)mu, std::chrono::duration<double, std::milli>(now() - t0).count());
      if (!hc)
        break;
      ++sw64;
      if (mu <= 1e-11f)
        break;
    }
    // (the sweeps' result is certified by its Gram matrix, too)
    if (sweeps && sw64) {
      if (!survey(8))
        return VJ_ERR_CUDA;
      certified = (!hst.over && asdbl(hst.cosbound) + pan <= lim);
    }
    unsigned herr = 0;
    if (cudaMemcpyAsync(&herr, gerr, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess || herr)
      return VJ_ERR_CUDA;
    if (presweeps)
      presweeps[1] = sw64;
    // columns in descending order of their norms, the order the reference's sweeps keep
    // (src/dvjsvd.c:367-370): its sweeps then have no pair to reorder
    double *nrm = vec;
    int *perm = reinterpret_cast<int *>(vec + n);
    double *Gp = reinterpret_cast<double *>(d1);
    k_colnorm2<CPLX><<<(unsigned)n, 256, 0, s>>>(mi, G, (long long)ldG, Gi, (long long)(CPLX ? ldGi : ldG), nrm);
    std::vector<double> hn((size_t)n);
    std::vector<int> hp((size_t)n);
    if (cudaMemcpyAsync(hn.data(), nrm, (size_t)n * 8, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return VJ_ERR_CUDA;
    for (int j = 0; j < ni; ++j)
      hp[(size_t)j] = j;
    std::stable_sort(hp.begin(), hp.end(), [&](int x, int y) { return hn[(size_t)x] > hn[(size_t)y]; });
    bool moved = false;
    for (int j = 0; j < ni && !moved; ++j)
      moved = (hp[(size_t)j] != j);
    if (moved) {
      if (cudaMemcpyAsync(perm, hp.data(), (size_t)n * 4, cudaMemcpyHostToDevice, s) != cudaSuccess)
        return VJ_ERR_CUDA;
      for (int pl = 0; pl < P; ++pl) {
        double *Gd = pl ? Gi : G, *Vd = pl ? Vi : V;
        const long long lg = pl ? (long long)ldGi : (long long)ldG, lv = pl ? (long long)ldVi : (long long)ldV;
        k_gather_cols<<<grid2(m, n), 256, 0, s>>>(mi, ni, Gd, lg, perm, Gp);
        k_gather_cols<<<grid2(n, n), 256, 0, s>>>(ni, ni, Vd, lv, perm, Y);
        if (!copy2d(Gd, lg, Gp, m, m, n, s) || !copy2d(Vd, lv, Y, n, n, n, s))
          return VJ_ERR_CUDA;
      }
      // the host vectors are read by the copy above: wait before they go out of scope
      if (cudaStreamSynchronize(s) != cudaSuccess)
        return VJ_ERR_CUDA;
    }
  }
  double ms64 = 0;
  {
    const auto t1 = now();
    ms64 = std::chrono::duration<double, std::milli>(t1 - t0).count();
    t0 = t1;
  }
  // 6. FP64 finishing sweeps (the reference's algorithm) with V preset
  const vj_fint r = svd_dev_entry<double, CPLX>(m_, n_, G, ldG, Gi, ldGi, V, ldV, Vi, ldVi, eS, fS, js, stp, swp, 2, certified, s);
  const double msfin = std::chrono::duration<double, std::milli>(now() - t0).count();
  // FP32 launches: 5 per step of a block sweep on the tensor cores (Gram, its reduction, the pair
  // eigenproblems, R, the rotation), 1 per step of a sweep by small blocks (n / b steps each), else 1
  // per pivot step
  const double steps32 = blk    ? (double)total32 * (double)(n / (CPLX ? 32 : 64)) * 5.0
                         : ncol ? (double)total32 * (double)(n / (ncol / 2))
                                : (double)total32 * stp;
  host::mixed_phases_set(ms32, msgemm, ms64, msfin, steps32, blk ? 1.0 : 0.0);
  if (trace)
    std::fprintf(stderr, "mixed SVD phases (ms): FP32 sweeps %.1f, orthonormalisation + products %.1f, FP64 refinement + sort %.1f, "
                 "finishing %.1f, certified %d\n", ms32, msgemm, ms64, msfin, certified ? 1 : 0);
  return r;
}

}  // namespace vj

extern "C" {

vj_fint vj_dvjsvd_mixed_dev(vj_fnat m, vj_fnat n, double *G, vj_fnat ldG, double *V, vj_fnat ldV, double *eS,
                            double *fS, const unsigned *js, unsigned stp, unsigned swp, unsigned stages,
                            unsigned *presweeps, void *stream)
{
  return vj::mixed_dev<false>(m, n, G, ldG, nullptr, ldG, V, ldV, nullptr, ldV, eS, fS, js, stp, swp, stages,
                              (cudaStream_t)stream, presweeps);
}

vj_fint vj_zvjsvd_mixed_dev(vj_fnat m, vj_fnat n, double *Gr, vj_fnat ldGr, double *Gi, vj_fnat ldGi, double *Vr,
                            vj_fnat ldVr, double *Vi, vj_fnat ldVi, double *eS, double *fS, const unsigned *js,
                            unsigned stp, unsigned swp, unsigned stages, unsigned *presweeps, void *stream)
{
  return vj::mixed_dev<true>(m, n, Gr, ldGr, Gi, ldGi, Vr, ldVr, Vi, ldVi, eS, fS, js, stp, swp, stages,
                             (cudaStream_t)stream, presweeps);
}

}  // extern "C"
