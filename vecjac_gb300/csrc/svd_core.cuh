// Device building blocks of the one-sided Jacobi SVD shared by the one-launch-per-step
// driver (jsvd.cu) and the batched persistent kernel (batch.cu): the AVX-512-exact column
// norm, the compensated scaled dot products in the reference's lane order, the pair
// classification (convergence test, shear test, prescale, 2x2) and the transformation of a
// column pair. Reference: src/dvjsvd.c:195-602, src/zvjsvd.c:214-652 and the L1 kernels
// they call (src/ddpscl.c, src/zdpscl.c, src/djrot.c, src/djrotf.c, src/zjrot.c,
// src/zjrotf.c, src/dgsscl.c, src/zgsscl.c).
#pragma once
#include <cfloat>
#include <cmath>

#include <cuda_runtime.h>

#include "jac2.cuh"
#include "svd_dot.cuh"
#include "svd_norm.cuh"
#include "vj_host.h"

namespace vj {

// control block of one pivot step (triple-buffered across launches)
struct Ctl {
  double MGbase, MVbase;  // max |G|, max |V| after this step's own rescaling (in T's range)
  unsigned long long nMG, nMV;  // atomicMax of max |.| of the transformed columns (T bits)
  int sT, sV;                   // accumulated power-of-two scalings of G and V
  int ovf;                      // a norm computed at the end of the previous step overflowed
  int pad;
};

struct SvdGlobal {
  long long err;                // 0 or the (negative) error code, atomicMin
  unsigned long long swt;       // transformed pairs in the current sweep
  Ctl ctl[3];
  // per-phase SM cycles of CTA 0 (the JTRACE split of src/dvjsvd.c:635), when tracing:
  // 0 control + rescaling, 1 staging, 2 dot products, 3 2x2 + classification, 4 rotations, 5 norms
  unsigned long long phase[8];
};

template <typename T> struct SvdArgs {
  int trace;                    // record per-phase cycles (VJ_TRACE=1)
  int trackv;                   // V is a preset matrix: its largest entry is tracked
  long long m, n, ldG, ldGi, ldV, ldVi;
  T *G, *Gi, *V, *Vi, *eS, *fS;
  const unsigned *js;
  SvdGlobal *g;
  T tol, gst;
  int nrm_exp, rot;
  long long e_dot, e_doti, e_appg, e_appv;
};

// ---- TMA (cp.async.bulk) staging of a column pair into shared memory ----
__device__ __forceinline__ unsigned smem_u32(const void *p)
{
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void tma_load_1d(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned phase)
{
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0u;
}
// bounded wait on phase 0 of the barrier; false after the iteration limit
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long *bar)
{
  for (unsigned it = 0; it < (1u << 22); ++it)
    if (mbar_try_wait(bar, 0u))
      return true;
  return false;
}

// (e, f) of a norm d: d = f 2^e, f in [1,2) (src/dznrm2.h:4-23)
template <typename T> __device__ __forceinline__ void ef_split(T d, T &e, T &f)
{
  using F = fp<T>;
  if (visfinite(d)) {
    if (d == (T)0) {
      e = vneg(F::inf());
      f = vor((T)1, vsgn(d));
    }
    else {
      const int k = ilogb_(d);
      e = (T)k;
      f = scale2(d, -k);
    }
  }
  else {
    e = F::inf();
    f = vor((visnan(d) ? (T)0 : (T)1), vsgn(d));
  }
}


// VDHYPOT (src/vecdef.h:80-92) on scalars
template <typename T> __device__ __forceinline__ T vhypot(T x, T y)
{
  const T x_ = vabs(x), y_ = vabs(y);
  const T m_ = vmin(x_, y_), M_ = vmax(x_, y_);
  T z = fp<T>::div(m_, M_);
  z = vmax(z, (T)0);
  z = fp<T>::fma_(z, z, (T)1);
  z = fp<T>::sqrt_(z);
  return z * M_;
}

// norm of column c (real, or complex with planes) by one warp; writes eS/fS; returns d
template <typename T, bool CPLX> __device__ T col_norm(const SvdArgs<T> &a, long long c)
{
  T d = warp_nrm2(a.G + c * a.ldG, a.m);
  if (CPLX) {
    const T di = warp_nrm2(a.Gi + c * a.ldGi, a.m);
    d = vhypot(d, di);
  }
  if ((threadIdx.x & 31) == 0) {
    T e, f;
    ef_split(d, e, f);
    a.eS[c] = e;
    a.fS[c] = f;
  }
  return d;
}

// Programmatic dependent launch: wait until the previous grid of the stream has completed
// and its writes are visible (a no-op for a launch without the attribute), then allow the
// next grid to be scheduled while this one runs, which hides the launch gap between the
// many short step kernels of a sweep.
__device__ __forceinline__ void pdl_enter()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// efcmp (src/defops.h:46)
template <typename T> __device__ __forceinline__ int efcmp(T e0, T f0, T e1, T f1)
{
  if (e0 > e1) return 1;
  if (e0 < e1) return -1;
  if (f0 > f1) return 1;
  if (f0 < f1) return -1;
  return 0;
}
template <typename T> __device__ __forceinline__ bool eflt(T e0, T e1, T f0, T f1)
{
  return (e0 < e1) || ((e0 == e1) && (f0 < f1));
}
template <typename T> __device__ __forceinline__ bool efle(T e0, T e1, T f0, T f1)
{
  return (e0 < e1) || ((e0 == e1) && (f0 <= f1));
}

template <typename T> struct PairState {
  T ep, fp, eq, fq;      // norms (e, f) of columns p, q
  T a21r, a21i;          // scaled dot (cosine of the angle)
  T c, cat, sat;         // rotation: cosine, Re/Im of e^{i alpha} tangent
  int code;              // 3/-3 shear (+/- permute), 2/-2 rotate, -1 swap, 1 nothing
  int skip;              // an error stops this pair
};

// step-start decisions of src/dvjsvd.c:199-233 and the overflow branch :276-295
template <typename T> struct Decision {
  int gres, vres, ovf;   // rescale G (sR < 0), rescale V, retry after a norm overflow
  int sNg, sNv;          // exponents used
  T MG, MV;              // values after the step's rescaling
  int sT, sV;
};

template <typename T> __device__ __forceinline__ int ef_exp(T x)
{
  // dbl2ef exponent of a nonnegative finite MG / MV (> 0)
  return ilogb_(x);
}

template <typename T> __device__ Decision<T> decide(const SvdArgs<T> &a, const Ctl &cur)
{
  Decision<T> d;
  T MG = (T)cur.MGbase, MV = (T)cur.MVbase;
  const T nMG = bitst<T>(cur.nMG), nMV = bitst<T>(cur.nMV);
  MG = fmax(MG, nMG);
  MV = fmax(MV, nMV);
  int eM = ef_exp(MG);
  int sR = a.rot - eM;
  const int sN = a.nrm_exp - eM - 1;
  d.sT = cur.sT;
  d.gres = (sR < 0);
  d.sNg = sN;
  if (d.gres) {
    MG = scale2(MG, sN);
    d.sT += sN;
  }
  eM = ef_exp(MV);
  sR = a.rot - eM;
  d.sNv = sR;
  d.vres = (sR < 0);
  d.sV = cur.sV;
  if (d.vres) {
    MV = scale2(MV, sR);
    d.sV += sR;
  }
  d.ovf = (!d.gres && cur.ovf);
  if (d.ovf) {
    // the reference rescales G by its current sN, which the V block has just set (src/dvjsvd.c:227,281)
    MG = scale2(MG, d.sNv);
    d.sT += d.sNv;
  }
  d.MG = MG;
  d.MV = MV;
  return d;
}

template <typename T> __device__ void scale_cols(T *A, long long ld, long long rows, long long c0, long long c1,
                                                 int e)
{
  for (long long i = threadIdx.x; i < rows; i += blockDim.x) {
    A[c0 * ld + i] = scale2(A[c0 * ld + i], e);
    A[c1 * ld + i] = scale2(A[c1 * ld + i], e);
  }
}

template <typename T> __device__ __forceinline__ void amax(typename fp<T>::U &m, T v)
{
  const typename fp<T>::U b = fp<T>::bits(v) & ~fp<T>::SIGN;
  m = (b > m) ? b : m;
}

// What the classification of a pair takes from the columns' norms alone: the order of the
// norms, the shear test and the Gram prescale (src/dvjsvd.c:349-405).
template <typename T> struct PairPre {
  T w11, w22, dd;  // scaled squared-norm ratios and the prescale exponent (<= 0)
  int ngs, cgs;    // p shorter than q; a shear instead of a rotation
};

template <typename T> __device__ __forceinline__ PairPre<T> pair_pre(T ep, T fp_, T eq, T fq, T gst)
{
  using F = fp<T>;
  PairPre<T> r;
  const T e1 = ep, e2 = eq, f1 = fp_, f2 = fq;
  const bool ngs = eflt(e1, e2, f1, f2);
  T maf = ngs ? f1 : f2, mae = ngs ? e1 : e2;
  const T Maf = ngs ? f2 : f1, Mae = ngs ? e2 : e1;
  maf = gst * maf;
  mae = mae + getexp(maf);
  maf = getmant(maf);
  r.ngs = ngs ? 1 : 0;
  r.cgs = eflt(mae, Mae, maf, Maf) ? 1 : 0;
  T f12 = F::div(f1, f2), e12 = e1 - e2, f21 = F::div(f2, f1), e21 = e2 - e1;
  e12 = e12 + getexp(f12);
  f12 = getmant(f12);
  e21 = e21 + getexp(f21);
  f21 = getmant(f21);
  const bool c12 = efle(e12, e21, f12, f21);
  const T E = c12 ? e21 : e12;
  const T dd = vmin(svdc<T>::MAX_FIN_EXP - E, (T)0);
  e12 = e12 + dd;
  e21 = e21 + dd;
  r.w11 = scalef(f12, e12);
  r.w22 = scalef(f21, e21);
  r.dd = dd;
  return r;
}

// the code of a transformed pair: 3/-3 shear, 2/-2 rotation (src/dvjsvd.c:422-459)
template <typename T> __device__ __forceinline__ int pair_code(const PairPre<T> &r, unsigned perm)
{
  if (r.cgs)
    return r.ngs ? -3 : 3;
  return perm ? -2 : 2;
}

// Convergence test, shear test, Gram prescale, 2x2 EVD and classification of one pair
// (src/dvjsvd.c:349-459): fills s.code (3/-3 shear, 2/-2 rotation, -1 swap, 1 nothing) and
// the rotation (c, cat, sat); returns whether the pair counts as transformed (|a21| >= tol).
// A swap (-1) must be completed by the caller by exchanging the pair's (eS, fS).
template <typename T, bool CPLX>
__device__ bool pair_classify(T ep, T fp_, T eq, T fq, T zr, T zi, T tol, T gst, PairState<T> &s)
{
  const T ab = CPLX ? vhypot(zr, zi) : vabs(zr);
  const bool trans = (tol <= ab);
  if (trans) {
    const PairPre<T> r = pair_pre(ep, fp_, eq, fq, gst);
    const T w21r = scalef(zr, r.dd);
    unsigned perm;
    T cc, at, sat = 0, l1, l2;
    if (CPLX)
      perm = cjac2<T, 0>(r.w11, r.w22, w21r, scalef(zi, r.dd), cc, at, sat, l1, l2);
    else
      perm = rjac2<T, 0>(r.w11, r.w22, w21r, cc, at, l1, l2);
    s.c = cc;
    s.cat = at;
    s.sat = sat;
    s.code = pair_code(r, perm);
  }
  else if (efcmp(ep, fp_, eq, fq) < 0)
    s.code = -1;
  else
    s.code = 1;
  return trans;
}

// exchange two columns
template <typename T> __device__ __forceinline__ void swap_cols(T *x, T *y, long long rows, int ltid, int TPP)
{
#pragma unroll 4
  for (long long i = ltid; i < rows; i += TPP) {
    const T t = x[i];
    x[i] = y[i];
    y[i] = t;
  }
}

// Rows of a column pair rotated, UR of a thread's rows at a time with the next UR loaded before
// these are stored: a store may alias a later load as far as the compiler knows, so a
// row-by-row loop would wait for one memory round trip per row. Reads (rx, ry), writes (x, y) and, when STG, the staged copy
// as well; mx and my collect max |.| of what x and y receive when track is set. The products by the
// cosine are three-register FMAs (vj_fp.cuh, FpOps).
template <typename T, bool STG, int UR>
__device__ __forceinline__ void rot_real(int rows, const T *rx, const T *ry, T *x, T *y, T *sx, T *sy, T at, T c,
                                         bool perm, int ltid, int TPP, bool track, typename fp<T>::U &mx,
                                         typename fp<T>::U &my)
{
  using F = fp<T>;
  const FpOps<T> o = FpOps<T>::make();
  const bool cone = (c == (T)1);
  // the permuted form writes (y - t x) c to x and (x + t y) c to y: the same two products
  // with the destinations exchanged
  T *const dx = perm ? y : x, *const dy = perm ? x : y, *const dsx = perm ? sy : sx, *const dsy = perm ? sx : sy;
  typename F::U mu = 0, mw = 0;
  T nu[UR], nw[UR];
  auto load = [&](int i0) {
#pragma unroll
    for (int k = 0; k < UR; ++k) {
      const int i = i0 + k * TPP;
      if (i < rows) {
        nu[k] = rx[i];
        nw[k] = ry[i];
      }
    }
  };
  load(ltid);
  for (int i0 = ltid; i0 < rows; i0 += UR * TPP) {
    T u[UR], w[UR];
#pragma unroll
    for (int k = 0; k < UR; ++k) {
      u[k] = nu[k];
      w[k] = nw[k];
    }
    load(i0 + UR * TPP);
    auto rotate = [&](int k) {
      const T x = u[k];
      u[k] = F::fma_(w[k], at, x);
      w[k] = F::fma_(-x, at, w[k]);
      if (!cone) {
        u[k] = o.mul(u[k], c);
        w[k] = o.mul(w[k], c);
      }
    };
    auto store = [&](int k) {
      const int i = i0 + k * TPP;
      dx[i] = u[k];
      dy[i] = w[k];
      if (STG) {
        dsx[i] = u[k];
        dsy[i] = w[k];
      }
      if (track) {
        amax(mu, u[k]);
        amax(mw, w[k]);
      }
    };
    // (all of a batch's FMAs before the first use of their results)
    if (i0 + (UR - 1) * TPP < rows) {
#pragma unroll
      for (int k = 0; k < UR; ++k)
        rotate(k);
#pragma unroll
      for (int k = 0; k < UR; ++k)
        store(k);
    }
    else {
#pragma unroll
      for (int k = 0; k < UR - 1; ++k)
        if (i0 + k * TPP < rows)
          rotate(k);
#pragma unroll
      for (int k = 0; k < UR - 1; ++k)
        if (i0 + k * TPP < rows)
          store(k);
    }
  }
  if (track) {
    mx = perm ? mw : mu;
    my = perm ? mu : mw;
  }
}

template <typename T, bool STG, int UR>
__device__ __forceinline__ void rot_cplx(int rows, const T *rxr, const T *rxi, const T *ryr, const T *ryi, T *xr,
                                         T *xi, T *yr, T *yi, T *sxr, T *sxi, T *syr, T *syi, T cta, T sta, T c,
                                         bool perm, int ltid, int TPP, bool track, typename fp<T>::U *m4)
{
  using F = fp<T>;
  const FpOps<T> o = FpOps<T>::make();
  const bool cone = (c == (T)1);
  const T cna = -cta;
  T *const dar = perm ? yr : xr, *const dai = perm ? yi : xi, *const dbr = perm ? xr : yr, *const dbi = perm ? xi : yi;
  T *const sar = perm ? syr : sxr, *const sai = perm ? syi : sxi, *const sbr = perm ? sxr : syr,
           *const sbi = perm ? sxi : syi;
  typename F::U mar = 0, mai = 0, mbr = 0, mbi = 0;
  T nxr[UR], nxi[UR], nyr[UR], nyi[UR];
  auto load = [&](int i0) {
#pragma unroll
    for (int k = 0; k < UR; ++k) {
      const int i = i0 + k * TPP;
      if (i < rows) {
        nxr[k] = rxr[i];
        nxi[k] = rxi[i];
        nyr[k] = ryr[i];
        nyi[k] = ryi[i];
      }
    }
  };
  load(ltid);
  for (int i0 = ltid; i0 < rows; i0 += UR * TPP) {
    T xr_[UR], xi_[UR], yr_[UR], yi_[UR];
#pragma unroll
    for (int k = 0; k < UR; ++k) {
      xr_[k] = nxr[k];
      xi_[k] = nxi[k];
      yr_[k] = nyr[k];
      yi_[k] = nyi[k];
    }
    load(i0 + UR * TPP);
    auto rotate = [&](int k) {
      const T x_r = xr_[k], x_i = xi_[k], y_r = yr_[k], y_i = yi_[k];
      xr_[k] = F::fma_(y_r, cta, F::fma_(-y_i, sta, x_r));
      xi_[k] = F::fma_(y_r, sta, F::fma_(y_i, cta, x_i));
      yr_[k] = F::fma_(x_r, cna, F::fma_(-x_i, sta, y_r));
      yi_[k] = F::fma_(x_r, sta, F::fma_(x_i, cna, y_i));
      if (!cone) {
        xr_[k] = o.mul(xr_[k], c);
        xi_[k] = o.mul(xi_[k], c);
        yr_[k] = o.mul(yr_[k], c);
        yi_[k] = o.mul(yi_[k], c);
      }
    };
    auto store = [&](int k) {
      const int i = i0 + k * TPP;
      dar[i] = xr_[k];
      dai[i] = xi_[k];
      dbr[i] = yr_[k];
      dbi[i] = yi_[k];
      if (STG) {
        sar[i] = xr_[k];
        sai[i] = xi_[k];
        sbr[i] = yr_[k];
        sbi[i] = yi_[k];
      }
      if (track) {
        amax(mar, xr_[k]);
        amax(mai, xi_[k]);
        amax(mbr, yr_[k]);
        amax(mbi, yi_[k]);
      }
    };
    if (i0 + (UR - 1) * TPP < rows) {
#pragma unroll
      for (int k = 0; k < UR; ++k)
        rotate(k);
#pragma unroll
      for (int k = 0; k < UR; ++k)
        store(k);
    }
    else {
#pragma unroll
      for (int k = 0; k < UR - 1; ++k)
        if (i0 + k * TPP < rows)
          rotate(k);
#pragma unroll
      for (int k = 0; k < UR - 1; ++k)
        if (i0 + k * TPP < rows)
          store(k);
    }
  }
  if (track) {
    m4[0] = perm ? mbr : mar;
    m4[1] = perm ? mar : mbr;
    m4[2] = perm ? mbi : mai;
    m4[3] = perm ? mai : mbi;
  }
}

// The transformation of one classified pair applied by a group of TPP threads (ltid =
// this thread's index in the group): rotation (src/djrot.c, src/djrotf.c, src/zjrot.c,
// src/zjrotf.c), shear (src/dgsscl.c, src/zgsscl.c) or swap, to the columns of G (read from
// rp/rq[/rpi/rqi], which is a staged copy when STG, written to both; the columns themselves
// otherwise) and of V. mx collects this thread's max |.| of the rows that the transformed
// columns p and q of G receive (their imaginary planes in mx[2], mx[3]) and mV, with trackv,
// that of V. Returns whether mx holds the maxima of the changed columns: false for an FP64
// rotation, and for a rotation by nothing or by a plain exchange, whose columns count as changed
// without being tracked. UR: rows per thread in flight (rot_real; half of it for complex columns).
template <typename T, bool CPLX, bool STG, int UR>
__device__ bool pair_apply(const PairState<T> &s, long long m, long long nv, T *Gp, T *Gq, T *Gip, T *Giq, T *Vp,
                           T *Vq, T *Vip, T *Viq, T *rp, T *rq, T *rpi, T *rqi, T *eSp, T *eSq, T *fSp, T *fSq,
                           int ltid, int TPP, bool trackv, typename fp<T>::U (&mx)[CPLX ? 4 : 2],
                           typename fp<T>::U &mV)
{
  using F = fp<T>;
  using U = typename F::U;
  const int code = s.code;
  if (code == 1) {
    // the pair is in order and orthogonal: nothing to apply
  }
  else if (code == -1) {
    // (the staged copy is not read again: a swapped pair's norms are exchanged, not recomputed)
    #pragma unroll 4
    for (long long i = ltid; i < m; i += TPP) {
      const T x = rp[i], y = rq[i];
      Gp[i] = y; Gq[i] = x;
      if (CPLX) { const T xi = rpi[i], yi = rqi[i]; Gip[i] = yi; Giq[i] = xi; }
    }
    swap_cols(Vp, Vq, nv, ltid, TPP);
    if (CPLX)
      swap_cols(Vip, Viq, nv, ltid, TPP);
  }
  else if (code == 3 || code == -3) {
    // Gram-Schmidt-like shear (src/dgsscl.c:5-85, src/zgsscl.c)
    const T ex = s.ep, ey = s.eq, fx = s.fp, fy = s.fq;
    const int nx = -(int)ex, ny = -(int)ey;
    const int px = (int)ex, py = (int)ey;
    if (code == 3) {
      const T ff = F::div(fy, fx);
      const T tfr = -s.a21r * ff;
      const T tfi = CPLX ? (s.a21i * ff) : (T)0;
      #pragma unroll 4
      for (long long i = ltid; i < m; i += TPP) {
        if (CPLX) {
          const T xri_ = scale2(rp[i], nx), xii_ = scale2(rpi[i], nx);
          const T yri_ = scale2(rq[i], ny), yii_ = scale2(rqi[i], ny);
          const T xr = F::fma_(tfr, xri_, F::fma_(-tfi, xii_, yri_));
          const T xi = F::fma_(tfr, xii_, F::fma_(tfi, xri_, yii_));
          const T ur = scale2(xr, py), ui = scale2(xi, py);
          Gq[i] = ur; Giq[i] = ui;
          if (STG) { rq[i] = ur; rqi[i] = ui; }
          amax(mx[1], ur); amax(mx[CPLX ? 3 : 1], ui);
        }
        else {
          const T xi = scale2(rp[i], nx);
          const T yi = scale2(rq[i], ny);
          const T u = scale2(F::fma_(tfr, xi, yi), py);
          Gq[i] = u;
          if (STG) rq[i] = u;
          amax(mx[1], u);
        }
      }
    }
    else {
      const T ff = F::div(fx, fy);
      const T tfr = -s.a21r * ff;
      const T tfi = CPLX ? (-s.a21i * ff) : (T)0;
      #pragma unroll 4
      for (long long i = ltid; i < m; i += TPP) {
        if (CPLX) {
          const T yri = rq[i], yii = rqi[i], xri = rp[i], xii = rpi[i];
          Gp[i] = yri; Gip[i] = yii;
          if (STG) { rp[i] = yri; rpi[i] = yii; }
          const T yri_ = scale2(yri, ny), yii_ = scale2(yii, ny);
          const T xri_ = scale2(xri, nx), xii_ = scale2(xii, nx);
          const T vr = F::fma_(tfr, yri_, F::fma_(-tfi, yii_, xri_));
          const T vi = F::fma_(tfr, yii_, F::fma_(tfi, yri_, xii_));
          const T ur = scale2(vr, px), ui = scale2(vi, px);
          Gq[i] = ur; Giq[i] = ui;
          if (STG) { rq[i] = ur; rqi[i] = ui; }
          amax(mx[1], ur); amax(mx[CPLX ? 3 : 1], ui);
        }
        else {
          const T xi = rp[i], yi = rq[i];
          Gp[i] = yi;
          if (STG) rp[i] = yi;
          const T u = scale2(F::fma_(tfr, scale2(yi, ny), scale2(xi, nx)), px);
          Gq[i] = u;
          if (STG) rq[i] = u;
          amax(mx[1], u);
        }
      }
      swap_cols(Vp, Vq, nv, ltid, TPP);
      if (CPLX)
        swap_cols(Vip, Viq, nv, ltid, TPP);
      if (ltid == 0) {
        *eSp = s.eq; *eSq = s.ep;
        *fSp = s.fq; *fSq = s.fp;
      }
    }
  }
  else {
    // rotation (src/djrot.c, src/djrotf.c, src/zjrot.c, src/zjrotf.c); code -2 permutes
    const bool perm = (code == -2);
    const T c = s.c, at = s.cat, sat = s.sat;
    // the reference marks both columns as changed after any rotation (src/dvjsvd.c:573)
    const bool real_rot = (!CPLX) || (sat == (T)0);
    if (real_rot && at == (T)0) {
      // c == 1: identity (or a swap when permuting); c != 1 "never happens" (-4 / -10)
      if (c == (T)1 && perm) {
        #pragma unroll 4
        for (long long i = ltid; i < m; i += TPP) {
          const T x = rp[i], y = rq[i];
          Gp[i] = y; Gq[i] = x;
          if (STG) { rp[i] = y; rq[i] = x; }
          if (CPLX) {
            const T xi = rpi[i], yi = rqi[i];
            Gip[i] = yi; Giq[i] = xi;
            if (STG) { rpi[i] = yi; rqi[i] = xi; }
          }
        }
        swap_cols(Vp, Vq, nv, ltid, TPP);
        if (CPLX)
          swap_cols(Vip, Viq, nv, ltid, TPP);
      }
      return false;
    }
    // FP64 rotations do not collect the largest |.|: a result of the FP64 unit that goes on to the
    // integer pipe costs more (1024 x 1024: 17.1k clocks for G's columns instead of 11.1k) than
    // another pass over the columns (0.8k).
    constexpr bool TRK = sizeof(T) == 4;
    U v0 = 0, v1 = 0;
    if (real_rot) {
      rot_real<T, STG, UR>((int)m, rp, rq, Gp, Gq, rp, rq, at, c, perm, ltid, TPP, TRK, mx[0], mx[1]);
      rot_real<T, false, UR>((int)nv, Vp, Vq, Vp, Vq, nullptr, nullptr, at, c, perm, ltid, TPP, trackv, v0, v1);
      if (trackv)
        mV = (v0 > v1) ? v0 : v1;
      if (CPLX) {
        rot_real<T, STG, UR>((int)m, rpi, rqi, Gip, Giq, rpi, rqi, at, c, perm, ltid, TPP, TRK, mx[CPLX ? 2 : 0],
                                  mx[CPLX ? 3 : 1]);
        rot_real<T, false, UR>((int)nv, Vip, Viq, Vip, Viq, nullptr, nullptr, at, c, perm, ltid, TPP, trackv, v0, v1);
        if (trackv) {
          v0 = (v0 > v1) ? v0 : v1;
          mV = (v0 > mV) ? v0 : mV;
        }
      }
    }
    else if constexpr (CPLX) {
      U v4[4] = {0, 0, 0, 0};
      rot_cplx<T, STG, UR / 2>((int)m, rp, rpi, rq, rqi, Gp, Gip, Gq, Giq, rp, rpi, rq, rqi, at, sat, c, perm, ltid,
                                TPP, TRK, mx);
      rot_cplx<T, false, UR / 2>((int)nv, Vp, Vip, Vq, Viq, Vp, Vip, Vq, Viq, nullptr, nullptr, nullptr, nullptr,
                                    at, sat, c, perm, ltid, TPP, trackv, v4);
      if (trackv) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mV = (v4[k] > mV) ? v4[k] : mV;
      }
    }
    return TRK;
  }
  return true;
}

// What pair_apply does to V's columns, apart from it: rows rows from Vp, Vq (imaginary parts Vip,
// Viq) on, by ltid of TPP threads
template <typename T, bool CPLX, int UR>
__device__ __forceinline__ void v_apply(const PairState<T> &s, int rows, T *Vp, T *Vq, T *Vip, T *Viq, int ltid, int TPP)
{
  const int code = s.code;
  if (s.skip || code == 1 || code == 3)
    return;
  const bool rot = (code == 2 || code == -2), perm = (code == -2);
  const bool real_rot = !CPLX || s.sat == (T)0;
  if (rot && !(real_rot && s.cat == (T)0)) {
    typename fp<T>::U m[4] = {0, 0, 0, 0};
    if (real_rot) {
      rot_real<T, false, UR>(rows, Vp, Vq, Vp, Vq, nullptr, nullptr, s.cat, s.c, perm, ltid, TPP, false, m[0], m[1]);
      if (CPLX)
        rot_real<T, false, UR>(rows, Vip, Viq, Vip, Viq, nullptr, nullptr, s.cat, s.c, perm, ltid, TPP, false, m[2],
                               m[3]);
    }
    else if constexpr (CPLX)
      rot_cplx<T, false, UR / 2>(rows, Vp, Vip, Vq, Viq, Vp, Vip, Vq, Viq, nullptr, nullptr, nullptr, nullptr, s.cat,
                                 s.sat, s.c, perm, ltid, TPP, false, m);
  }
  else if (!rot || (s.c == (T)1 && perm)) {
    swap_cols(Vp, Vq, rows, ltid, TPP);
    if (CPLX)
      swap_cols(Vip, Viq, rows, ltid, TPP);
  }
}

}  // namespace vj
