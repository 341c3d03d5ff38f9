// FP32 one-sided Jacobi sweeps by small blocks of columns, one CTA per pair of blocks: the FP32
// stages of the mixed-precision SVD (mixed.cu) for matrices whose pair of blocks fits in a
// CTA's shared memory.
//
// A sweep of column pairs is n pivot steps of 2-4 us that are launch, load and reduction
// latency (3.5 us per step at 1024 x 1024 real, 512 CTAs of one pair each). Here the n columns are
// cut into blocks of b (8 real, 4 complex; half of that for longer columns) and a CTA takes a pair
// of blocks: it copies their 2b columns of G and of the rotation accumulator W into shared memory
// (bulk copies; W's arrive during the eigenproblem), forms the 2b x 2b Gram matrix of G's (all
// warps, rows over threads, a lane's partial sums of all entries in registers), runs one cyclic
// two-sided Jacobi sweep on it, accumulating the rotation R, and writes G R and W R. A sweep is
// n / b such steps (modulus ordering of the blocks and inside them, with the longer column first:
// it needs half as many sweeps as the round-robin ordering), so the per-step latencies are paid
// n / b instead of n times. FP32 Gram entries are as accurate relative to the column
// norms as the dot products of a column pair; the sweeps precondition the FP64 phases, which
// decide the result.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "pjs.cuh"
#include "svd_core.cuh"
#include "vj_host.h"

namespace vj {
namespace cb {

constexpr int NT = 256;
constexpr size_t SMEM_MAX = 208 * 1024;

struct Args {
  float *Gr, *Gi, *Wr, *Wi;  // leading dimensions m and n
  int m, n, nb, step;
  float tol;
  unsigned *cnt;  // rotations; largest |cos| (bits)
};

// sum of v over the warp's lanes for `COUNT` values: lane l ends with the sums of the values whose
// index is l mod 32 (recursive halving: COUNT instead of 5 COUNT shuffles)
template <int COUNT> __device__ __forceinline__ void warp_sums(float (&v)[COUNT], float *out)
{
  const int lane = threadIdx.x & 31;
  constexpr int PADDED = (COUNT + 31) / 32 * 32;
#pragma unroll
  for (int g = 0; g < PADDED; g += 32) {
    float w[32];
#pragma unroll
    for (int i = 0; i < 32; ++i)
      w[i] = (g + i < COUNT) ? v[(g + i < COUNT) ? g + i : 0] : 0.0f;
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
      const bool up = (lane & h) != 0;
#pragma unroll
      for (int i = 0; i < h; ++i) {
        const float send = up ? w[i] : w[i + h], keep = up ? w[i + h] : w[i];
        w[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
      }
    }
    if (g + lane < COUNT)
      out[g + lane] = w[0];
  }
}

// NC: columns of a block pair (2 b)
template <bool CPLX, int NC> __global__ void __launch_bounds__(NT, 1) k_col_blocks(Args a)
{
  constexpr int B = NC / 2, P = CPLX ? 2 : 1;
  constexpr int NH = NC * (NC + 1) / 2;                      // entries of the upper triangle
  constexpr int NA = CPLX ? NC + 2 * (NH - NC) : NH;         // real sums: diagonal, then pairs (re, im)
  extern __shared__ __align__(128) float X[];                // plane, column, m rows of G and n of W
  __shared__ float part[NT / 32][NA];
  __shared__ float Hr[2][NC][NC + 1], Hi[2][CPLX ? NC : 1][NC + 1];  // (this step's and the next's)
  __shared__ __align__(16) float Rr[NC][NC], Ri[CPLX ? NC : 1][NC];
  __shared__ unsigned long long bar[2];
  __shared__ unsigned s_rot, s_mu;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned I, J;
  pair_mod((unsigned)a.nb, (unsigned)a.step, blockIdx.x, I, J);
  const int m = a.m, n = a.n, rows = m + n;
  auto col = [&](int c) { return (c < B) ? (int)I * B + c : (int)J * B + (c - B); };
  auto xcol = [&](int pl, int c) { return X + (size_t)(pl * NC + c) * rows; };
  if (tid == 0) {
    mbar_init(&bar[0], 1u);
    mbar_init(&bar[1], 1u);
    s_rot = s_mu = 0u;
  }
  __syncthreads();
  pdl_enter();
  if (tid == 0) {
    mbar_expect_tx(&bar[0], (unsigned)(NC * P * m * 4));
    for (int c = 0; c < NC; ++c) {
      tma_load_1d(xcol(0, c), a.Gr + (size_t)col(c) * m, (unsigned)(m * 4), &bar[0]);
      if (CPLX)
        tma_load_1d(xcol(1, c), a.Gi + (size_t)col(c) * m, (unsigned)(m * 4), &bar[0]);
    }
    mbar_expect_tx(&bar[1], (unsigned)(NC * P * n * 4));
    for (int c = 0; c < NC; ++c) {
      tma_load_1d(xcol(0, c) + m, a.Wr + (size_t)col(c) * n, (unsigned)(n * 4), &bar[1]);
      if (CPLX)
        tma_load_1d(xcol(1, c) + m, a.Wi + (size_t)col(c) * n, (unsigned)(n * 4), &bar[1]);
    }
  }
  bool ok = mbar_wait_bounded(&bar[0]);
  // ---- Gram matrix: rows over threads, four at a time ----
  if (ok) {
    float acc[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i)
      acc[i] = 0.0f;
    for (int g = tid; g < (m >> 2); g += NT) {
      float4 xr[NC], xi[CPLX ? NC : 1];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        xr[c] = reinterpret_cast<const float4 *>(xcol(0, c))[g];
        if (CPLX)
          xi[c] = reinterpret_cast<const float4 *>(xcol(1, c))[g];
      }
      auto dot = [](const float4 &u, const float4 &v, float s) {
        s = __fmaf_rn(u.x, v.x, s);
        s = __fmaf_rn(u.y, v.y, s);
        s = __fmaf_rn(u.z, v.z, s);
        return __fmaf_rn(u.w, v.w, s);
      };
      auto ndot = [](const float4 &u, const float4 &v, float s) {
        s = __fmaf_rn(-u.x, v.x, s);
        s = __fmaf_rn(-u.y, v.y, s);
        s = __fmaf_rn(-u.z, v.z, s);
        return __fmaf_rn(-u.w, v.w, s);
      };
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        acc[i] = dot(xr[i], xr[i], acc[i]);
        if (CPLX)
          acc[i] = dot(xi[CPLX ? i : 0], xi[CPLX ? i : 0], acc[i]);
      }
      int e = NC;
#pragma unroll
      for (int i = 0; i < NC; ++i)
#pragma unroll
        for (int j = i + 1; j < NC; ++j) {
          acc[e] = dot(xr[i], xr[j], acc[e]);
          if (CPLX) {
            // g_i^H g_j
            acc[e] = dot(xi[CPLX ? i : 0], xi[CPLX ? j : 0], acc[e]);
            acc[e + 1] = dot(xr[i], xi[CPLX ? j : 0], acc[e + 1]);
            acc[e + 1] = ndot(xi[CPLX ? i : 0], xr[j], acc[e + 1]);
            e += 2;
          }
          else
            ++e;
        }
    }
    warp_sums<NA>(acc, part[warp]);
  }
  __syncthreads();
  for (int q = tid; q < NC * NC; q += NT) {
    const int i = q / NC, j = q % NC;
    if (i <= j) {
      const int u = i * NC - i * (i + 1) / 2 + (j - i - 1);  // pair (i, j) among the pairs
      const int e = (i == j) ? i : NC + (CPLX ? 2 : 1) * u;
      float s = 0.0f, t = 0.0f;
      for (int w = 0; w < NT / 32; ++w) {
        s += part[w][e];
        if (CPLX && i != j)
          t += part[w][e + 1];
      }
      Hr[0][i][j] = Hr[0][j][i] = s;
      if (CPLX) {
        Hi[0][CPLX ? i : 0][j] = t;
        Hi[0][CPLX ? j : 0][i] = -t;
      }
    }
    Rr[i][j] = (i == j) ? 1.0f : 0.0f;
    if (CPLX)
      Ri[CPLX ? i : 0][j] = 0.0f;
  }
  __syncthreads();
  // ---- one cyclic Jacobi sweep of H, rotations accumulated in R ----
  // A step takes B disjoint pairs. Thread u B + v transforms the 2 x 2 block of row pair u and
  // column pair v, the threads after those a row of R each for one pair; all of them compute the
  // one or two rotations they need from H as the last step left it, and write H for the next one,
  // so a step has one barrier.
  struct Rotation {
    float cs, sr, si;  // cosine, sine times e^{i phi}
    bool go, sw;       // rotated; the second new column is the longer one and goes first
  };
  float mu = 0.0f;
  unsigned nrot = 0u;
  for (int st = 0; st < NC; ++st) {
    const int cur = st & 1;
    // the rotation of pair (p, q): t^2 + 2 zeta t - 1 = 0, zeta = (b - a) / (2 |c|)
    auto rotation = [&](int p, int q, float *cosine) {
      const float ha = Hr[cur][p][p], hb = Hr[cur][q][q], cr = Hr[cur][p][q], ci = CPLX ? Hi[cur][CPLX ? p : 0][q] : 0.0f;
      Rotation r{1.0f, 0.0f, 0.0f, false, false};
      // (in terms of the cosine, so that short columns' squares do not underflow)
      const float ra = rsqrtf(ha), rb = rsqrtf(hb), xr = cr * ra * rb, xi = CPLX ? ci * ra * rb : 0.0f;
      const float c2 = CPLX ? __fmaf_rn(xr, xr, xi * xi) : xr * xr;
      if (ha > 0.0f && hb > 0.0f && c2 >= a.tol * a.tol) {
        const float ic = rsqrtf(c2), zeta = 0.5f * (hb - ha) * ra * rb * ic, az = fabsf(zeta);
        const float t = (az > 1e15f) ? __fdividef(0.5f, zeta)
                                     : copysignf(__fdividef(1.0f, az + sqrtf(__fmaf_rn(az, az, 1.0f))), zeta);
        const float d = __fmaf_rn(t, t, 1.0f), ac = c2 * ic * (ha * ra) * (hb * rb);
        float cs = rsqrtf(d);
        cs = __fmaf_rn(cs * 0.5f, __fmaf_rn(-d * cs, cs, 1.0f), cs);
        const float sn = t * cs * ic;
        r = Rotation{cs, sn * xr, CPLX ? sn * xi : 0.0f, true, hb + t * ac > ha - t * ac};
        if (cosine)
          *cosine = c2 * ic;
      }
      return r;
    };
    // (x, y) <- (cs x - conj(s) y, cs y + s x), exchanged when the second is the longer
    auto turn = [](const Rotation &r, float2 &x, float2 &y) {
      float2 u, v;
      if (CPLX) {
        u = make_float2(__fmaf_rn(r.cs, x.x, -__fmaf_rn(r.sr, y.x, r.si * y.y)),
                        __fmaf_rn(r.cs, x.y, -__fmaf_rn(r.sr, y.y, -(r.si * y.x))));
        v = make_float2(__fmaf_rn(r.cs, y.x, __fmaf_rn(r.sr, x.x, -(r.si * x.y))),
                        __fmaf_rn(r.cs, y.y, __fmaf_rn(r.sr, x.y, r.si * x.x)));
      }
      else {
        u = make_float2(__fmaf_rn(r.cs, x.x, -(r.sr * y.x)), 0.0f);
        v = make_float2(__fmaf_rn(r.cs, y.x, r.sr * x.x), 0.0f);
      }
      x = r.sw ? v : u;
      y = r.sw ? u : v;
    };
    if (tid < B * B) {
      const int u = tid / B, v = tid % B;
      unsigned pu, qu, pv, qv;
      pair_mod(NC, (unsigned)st, (unsigned)u, pu, qu);
      pair_mod(NC, (unsigned)st, (unsigned)v, pv, qv);
      float cosine = 0.0f;
      const Rotation rv = rotation((int)pv, (int)qv, (u == v) ? &cosine : nullptr);
      Rotation ru = rotation((int)pu, (int)qu, nullptr);
      if (u == v) {
        nrot += rv.go ? 1u : 0u;
        mu = fmaxf(mu, cosine);
      }
      auto h = [&](unsigned i, unsigned j) {
        return make_float2(Hr[cur][i][j], CPLX ? Hi[cur][CPLX ? i : 0][j] : 0.0f);
      };
      float2 b00 = h(pu, pv), b01 = h(pu, qv), b10 = h(qu, pv), b11 = h(qu, qv);
      turn(rv, b00, b01);
      turn(rv, b10, b11);
      ru.si = -ru.si;  // rows: the conjugate
      turn(ru, b00, b10);
      turn(ru, b01, b11);
      auto put = [&](unsigned i, unsigned j, const float2 &x) {
        Hr[cur ^ 1][i][j] = x.x;
        if (CPLX)
          Hi[cur ^ 1][CPLX ? i : 0][j] = x.y;
      };
      put(pu, pv, b00);
      put(pu, qv, b01);
      put(qu, pv, b10);
      put(qu, qv, b11);
    }
    else if (tid < B * B + NC * B) {
      const int w = tid - B * B, u = w % B, i = w / B;
      unsigned p, q;
      pair_mod(NC, (unsigned)st, (unsigned)u, p, q);
      const Rotation r = rotation((int)p, (int)q, nullptr);
      if (r.go) {
        float2 x = make_float2(Rr[i][p], CPLX ? Ri[CPLX ? i : 0][p] : 0.0f),
               y = make_float2(Rr[i][q], CPLX ? Ri[CPLX ? i : 0][q] : 0.0f);
        turn(r, x, y);
        Rr[i][p] = x.x;
        Rr[i][q] = y.x;
        if (CPLX) {
          Ri[CPLX ? i : 0][p] = x.y;
          Ri[CPLX ? i : 0][q] = y.y;
        }
      }
    }
    __syncthreads();
  }
  if (nrot) {
    atomicAdd(&s_rot, nrot);
    atomicMax(&s_mu, __float_as_uint(mu));
  }
  ok = mbar_wait_bounded(&bar[1]) && ok;
  if (!__syncthreads_and(ok)) {
    // a copy did not land within the limit: flag it, wait for both once more, touch nothing
    if (tid == 0)
      atomicOr(a.cnt + 2, 1u);
    (void)mbar_wait_bounded(&bar[0]);
    (void)mbar_wait_bounded(&bar[1]);
    return;
  }
  if (!s_rot)
    return;
  if (tid == 0) {
    atomicAdd(a.cnt, s_rot);
    atomicMax(a.cnt + 1, s_mu);
  }
  // ---- G R and W R: four rows per thread ----
  for (int g = tid; g < (rows >> 2); g += NT) {
    const bool isg = g < (m >> 2);
    F32x2 o[CPLX ? 2 : 1][NC][2];
#pragma unroll
    for (int pl = 0; pl < P; ++pl)
#pragma unroll
      for (int j = 0; j < NC; ++j)
        o[pl][j][0] = o[pl][j][1] = f2_make(0.0f, 0.0f);
#pragma unroll 4
    for (int i = 0; i < NC; ++i) {
      const float4 x = reinterpret_cast<const float4 *>(xcol(0, i))[g];
      const F32x2 x0 = f2_make(x.x, x.y), x1 = f2_make(x.z, x.w);
      F32x2 y0 = x0, y1 = x1;
      if (CPLX) {
        const float4 y = reinterpret_cast<const float4 *>(xcol(1, i))[g];
        y0 = f2_make(y.x, y.y);
        y1 = f2_make(y.z, y.w);
      }
#pragma unroll
      for (int j = 0; j < NC; j += 4) {
        const float4 rr = *reinterpret_cast<const float4 *>(&Rr[i][j]);
        const float rv[4] = {rr.x, rr.y, rr.z, rr.w};
        float iv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (CPLX) {
          const float4 ri = *reinterpret_cast<const float4 *>(&Ri[CPLX ? i : 0][j]);
          iv[0] = ri.x;
          iv[1] = ri.y;
          iv[2] = ri.z;
          iv[3] = ri.w;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const F32x2 c = f2_make(rv[k], rv[k]);
          o[0][j + k][0] = f2_fma(x0, c, o[0][j + k][0]);
          o[0][j + k][1] = f2_fma(x1, c, o[0][j + k][1]);
          if (CPLX) {
            const F32x2 s = f2_make(iv[k], iv[k]), ns = f2_make(-iv[k], -iv[k]);
            o[0][j + k][0] = f2_fma(y0, ns, o[0][j + k][0]);
            o[0][j + k][1] = f2_fma(y1, ns, o[0][j + k][1]);
            o[CPLX ? 1 : 0][j + k][0] = f2_fma(x0, s, f2_fma(y0, c, o[CPLX ? 1 : 0][j + k][0]));
            o[CPLX ? 1 : 0][j + k][1] = f2_fma(x1, s, f2_fma(y1, c, o[CPLX ? 1 : 0][j + k][1]));
          }
        }
      }
    }
    const size_t ld = isg ? (size_t)m : (size_t)n;
    const int r4 = isg ? g : g - (m >> 2);
#pragma unroll
    for (int pl = 0; pl < P; ++pl) {
      float *const base = isg ? (pl ? a.Gi : a.Gr) : (pl ? a.Wi : a.Wr);
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        float4 v;
        f2_get(o[pl][j][0], v.x, v.y);
        f2_get(o[pl][j][1], v.z, v.w);
        reinterpret_cast<float4 *>(base + (size_t)col(j) * ld)[r4] = v;
      }
    }
  }
}

static size_t smem(bool cplx, int nc, long long m, long long n) { return (size_t)nc * (cplx ? 2u : 1u) * (size_t)(m + n) * 4u; }

}  // namespace cb

// columns per block pair of the small-block sweeps for this shape, or 0 when they do not apply:
// whole blocks, at least two of them, and a pair's columns within a CTA's shared memory
int col_blocks(bool cplx, long long m, long long n)
{
  if ((m & 3) || (n & 3))
    return 0;
  for (int nc = cplx ? 8 : 16; nc >= (cplx ? 4 : 8); nc >>= 1)
    if (n % nc == 0 && cb::smem(cplx, nc, m, n) <= cb::SMEM_MAX)
      return nc;
  return 0;
}

// one block sweep; the number of rotations (< 0: an error) and the largest |cos| of a rotated pair
long long col_block_sweep(bool cplx, int m, int n, float *Gr, float *Gi, float *Wr, float *Wi, float tol, unsigned *cnt,
                          cudaStream_t s, float *mu)
{
  const int nc = col_blocks(cplx, m, n);
  void (*const k)(cb::Args) = cplx ? (nc == 8 ? cb::k_col_blocks<true, 8> : cb::k_col_blocks<true, 4>)
                                   : (nc == 16 ? cb::k_col_blocks<false, 16> : cb::k_col_blocks<false, 8>);
  const size_t sm = cb::smem(cplx, nc, m, n);
  if (!nc || cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess ||
      cudaMemsetAsync(cnt, 0, 12, s) != cudaSuccess)
    return -1;
  cb::Args a{Gr, Gi, Wr, Wi, m, n, n / (nc / 2), 0, tol, cnt};
  for (a.step = 0; a.step < a.nb; ++a.step)
    if (host::launch_pdl(k, dim3((unsigned)(a.nb / 2)), dim3(cb::NT), sm, s, a) != cudaSuccess)
      return -1;
  unsigned hc[3] = {0u, 0u, 1u};
  if (cudaGetLastError() != cudaSuccess || cudaMemcpyAsync(hc, cnt, 12, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess || hc[2])
    return -1;
  memcpy(mu, &hc[1], 4);
  return (long long)hc[0];
}

}  // namespace vj
