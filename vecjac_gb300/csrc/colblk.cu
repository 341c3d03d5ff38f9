// FP32 one-sided Jacobi sweeps by small blocks of columns, a CTA or a small cluster per pair of
// blocks: the FP32 stages of the mixed-precision SVD (mixed.cu) for matrices whose pair of blocks
// fits in shared memory.
//
// A sweep of column pairs is n pivot steps of 2-4 us that are launch, load and reduction
// latency (3.5 us per step at 1024 x 1024 real, 512 CTAs of one pair each). Here the n columns are
// cut into blocks of b (8 real, 4 complex; half of that for longer columns) and a CTA takes a pair
// of blocks: it copies their 2b columns of G and of the rotation accumulator W into shared memory
// (bulk copies; W's arrive during the eigenproblem), forms the 2b x 2b Gram matrix of G's (all
// warps, rows over threads, a lane's partial sums of all entries in registers), runs one cyclic
// two-sided Jacobi sweep (over the pairs between the blocks only, but for the first step) on it,
// accumulating the rotation R, and writes G R and W R. A sweep is
// n / b such steps (modulus ordering of the blocks and inside them, with the longer column first:
// it needs half as many sweeps as the round-robin ordering), so the per-step latencies are paid
// n / b instead of n times. Where the pairs leave SMs idle, or their columns need more shared
// memory, the CTAs of a cluster split the rows: each adds up the partial Gram sums of all of them
// in the same order, solves the same eigenproblem and rotates its own rows. FP32 Gram entries are as accurate relative to the column
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
constexpr size_t SMEM_MAX = 204 * 1024;

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
  __shared__ float part[NT / 32][NA], total[NA], gram[NA];
  __shared__ float Hr[2][NC][NC + 1], Hi[2][CPLX ? NC : 1][NC + 1];  // (this step's and the next's)
  __shared__ __align__(16) float Rr[NC][NC], Ri[CPLX ? NC : 1][NC];
  __shared__ unsigned short ptab[NC][B];  // p | q << 8 of pair u of a step
  __shared__ unsigned long long bar[2];
  __shared__ unsigned s_rot, s_mu;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int m = a.m, n = a.n;
  unsigned rank, cs;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(cs));
  const int pairno = (int)(blockIdx.x / cs);
  // this CTA's rows of G and of W, in groups of four
  const int g0 = (int)((long long)(m >> 2) * rank / cs), g1 = (int)((long long)(m >> 2) * (rank + 1) / cs);
  const int w0 = (int)((long long)(n >> 2) * rank / cs), w1 = (int)((long long)(n >> 2) * (rank + 1) / cs);
  const int gq = g1 - g0, wq = w1 - w0, rows = 4 * (gq + wq);
  unsigned I, J;
  pair_mod((unsigned)a.nb, (unsigned)a.step, (unsigned)pairno, I, J);
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
    mbar_expect_tx(&bar[0], (unsigned)(NC * P * gq * 16));
    for (int c = 0; c < NC && gq; ++c) {
      tma_load_1d(xcol(0, c), a.Gr + (size_t)col(c) * m + 4 * g0, (unsigned)(gq * 16), &bar[0]);
      if (CPLX)
        tma_load_1d(xcol(1, c), a.Gi + (size_t)col(c) * m + 4 * g0, (unsigned)(gq * 16), &bar[0]);
    }
    mbar_expect_tx(&bar[1], (unsigned)(NC * P * wq * 16));
    for (int c = 0; c < NC && wq; ++c) {
      tma_load_1d(xcol(0, c) + 4 * gq, a.Wr + (size_t)col(c) * n + 4 * w0, (unsigned)(wq * 16), &bar[1]);
      if (CPLX)
        tma_load_1d(xcol(1, c) + 4 * gq, a.Wi + (size_t)col(c) * n + 4 * w0, (unsigned)(wq * 16), &bar[1]);
    }
  }
  // every pair of the columns in the first step of a sweep (which takes every block once), the pairs
  // between the two blocks in the others: half of the Jacobi steps, and no more sweeps
  const int nst = a.step ? B : NC;
  if (tid < NC * B) {
    unsigned p, q;
    pair_mod(NC, (unsigned)(tid / B), (unsigned)(tid % B), p, q);
    if (nst == B) {
      p = tid % B;
      q = B + (tid % B + tid / B) % B;
    }
    ptab[tid / B][tid % B] = (unsigned short)(p | (q << 8));
  }
  // (one answer per warp: its lanes go into the shuffles of the sums together, or none does)
  bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bar[0]));
  // ---- Gram matrix: rows over threads, four at a time ----
  if (ok) {
    float acc[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i)
      acc[i] = 0.0f;
    for (int g = tid; g < gq; g += NT) {
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
  if (cs > 1) {
    // every CTA's sums to every CTA; the same sums in the same order everywhere
    __syncthreads();
    for (int e = tid; e < NA; e += NT) {
      float t = 0.0f;
      for (int w = 0; w < NT / 32; ++w)
        t += part[w][e];
      total[e] = t;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int e = tid; e < NA; e += NT) {
      float t = 0.0f;
      for (unsigned r = 0; r < cs; ++r) {
        unsigned addr;
        float v;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(&total[e])), "r"(r));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
        t += v;
      }
      gram[e] = t;
    }
    // (no CTA leaves, or writes its sums again, before all have read them: waited for at the end)
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  else {
    __syncthreads();
    for (int e = tid; e < NA; e += NT) {
      float t = 0.0f;
      for (int w = 0; w < NT / 32; ++w)
        t += part[w][e];
      gram[e] = t;
    }
  }
  auto leave = [&]() {
    if (cs > 1)
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  };
  __syncthreads();
  for (int q = tid; q < NC * NC; q += NT) {
    const int i = q / NC, j = q % NC;
    if (i <= j) {
      const int u = i * NC - i * (i + 1) / 2 + (j - i - 1);  // pair (i, j) among the pairs
      const int e = (i == j) ? i : NC + (CPLX ? 2 : 1) * u;
      Hr[0][i][j] = Hr[0][j][i] = gram[e];
      if (CPLX) {
        const float t = (i != j) ? gram[e + 1] : 0.0f;
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
  const float tol2 = a.tol * a.tol;
  float mu2 = 0.0f;
  unsigned nrot = 0u;
  for (int st = 0; st < nst; ++st) {
    const int cur = st & 1;
    // the rotation of pair (p, q): with d = b - a and w = sqrt(d^2 + 4 |c|^2), cs^2 = (1 + |d| / w) / 2
    // and the sine times e^{i phi} sign(d) c / (w cs); two reciprocal roots, refined by a Newton
    // step each, as the dependent operations of a step are all that counts here
    auto rotation = [&](int p, int q, float *cos2) {
      const float ha = Hr[cur][p][p], hb = Hr[cur][q][q], cr = Hr[cur][p][q], ci = CPLX ? Hi[cur][CPLX ? p : 0][q] : 0.0f;
      // (c and d over sqrt(a b): squares of short columns' entries would leave the range)
      const float ir = rsqrtf(ha) * rsqrtf(hb), xr = cr * ir, xi = ci * ir, d = (hb - ha) * ir;
      const float c2 = CPLX ? __fmaf_rn(xr, xr, xi * xi) : xr * xr;
      // (no branch: what a pair that is not rotated computes is dropped at the end)
      const bool go = ha > 0.0f && hb > 0.0f && c2 >= tol2 && fabsf(d) < 1e18f;
      const float w2 = __fmaf_rn(d, d, 4.0f * c2);
      float iw = rsqrtf(w2);
      iw = __fmaf_rn(0.5f * iw, __fmaf_rn(-w2 * iw, iw, 1.0f), iw);
      const float u = __fmaf_rn(0.5f * fabsf(d), iw, 0.5f);
      float iu = rsqrtf(u);
      iu = __fmaf_rn(0.5f * iu, __fmaf_rn(-u * iu, iu, 1.0f), iu);
      const float k = go ? copysignf(iw * iu, d) : 0.0f;
      // (the new norms are a - t |c| and b + t |c| with t of d's sign: the longer stays the longer)
      const Rotation r{go ? u * iu : 1.0f, go ? k * xr : 0.0f, (CPLX && go) ? k * xi : 0.0f, go, go && d >= 0.0f};
      if (cos2)
        *cos2 = go ? c2 : 0.0f;
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
      const unsigned tu = ptab[st][u], tv = ptab[st][v], pu = tu & 255u, qu = tu >> 8, pv = tv & 255u, qv = tv >> 8;
      auto h = [&](unsigned i, unsigned j) {
        return make_float2(Hr[cur][i][j], CPLX ? Hi[cur][CPLX ? i : 0][j] : 0.0f);
      };
      float2 b00 = h(pu, pv), b01 = h(pu, qv), b10 = h(qu, pv), b11 = h(qu, qv);
      float cosine = 0.0f;
      const Rotation rv = rotation((int)pv, (int)qv, &cosine);
      Rotation ru = rotation((int)pu, (int)qu, nullptr);
      if (u == v) {
        nrot += rv.go ? 1u : 0u;
        mu2 = fmaxf(mu2, cosine);
      }
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
      const unsigned t = ptab[st][u], p = t & 255u, q = t >> 8;
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
    atomicMax(&s_mu, __float_as_uint(sqrtf(mu2)));
  }
  ok = mbar_wait_bounded(&bar[1]) && ok;
  if (!__syncthreads_and(ok)) {
    // a copy did not land within the limit: flag it, wait for both once more, touch nothing
    if (tid == 0)
      atomicOr(a.cnt + 2, 1u);
    (void)mbar_wait_bounded(&bar[0]);
    (void)mbar_wait_bounded(&bar[1]);
    leave();
    return;
  }
  if (!s_rot) {
    leave();
    return;
  }
  if (tid == 0 && rank == 0) {
    atomicAdd(a.cnt, s_rot);
    atomicMax(a.cnt + 1, s_mu);
  }
  // ---- G R and W R: four rows per thread ----
  for (int g = tid; g < gq + wq; g += NT) {
    const bool isg = g < gq;
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
    const int r4 = isg ? g0 + g : w0 + g - gq;
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
  leave();
}

// a CTA's share of the columns of a pair of blocks
static size_t smem(bool cplx, int nc, int cs, long long m, long long n)
{
  return (size_t)nc * (cplx ? 2u : 1u) * 16u * (size_t)((m / 4 + cs - 1) / cs + (n / 4 + cs - 1) / cs);
}

struct Shape {
  int nc, cs;  // columns per pair of blocks (0: not for this shape), CTAs per pair
};
// As wide blocks as shared memory allows a cluster; two CTAs per pair where that keeps all of a step's
// on the GPU at once, or as many as shared memory asks for.
static Shape shape(bool cplx, long long m, long long n)
{
  if ((m & 3) || (n & 3))
    return Shape{0, 0};
  const int sms = host::sm_count();
  for (int nc = cplx ? 8 : 16; nc >= (cplx ? 4 : 8); nc >>= 1) {
    if (n % nc)
      continue;
    // (more than two CTAs per pair only for room: the exchange of the sums costs what they save)
    int cs = ((n / nc) * 2 <= sms) ? 2 : 1;
    while (cs < 8 && smem(cplx, nc, cs, m, n) > SMEM_MAX)
      cs *= 2;
    if (smem(cplx, nc, cs, m, n) <= SMEM_MAX)
      return Shape{nc, cs};
  }
  return Shape{0, 0};
}

}  // namespace cb

// columns per block pair of the small-block sweeps for this shape, or 0 when they do not apply
int col_blocks(bool cplx, long long m, long long n) { return cb::shape(cplx, m, n).nc; }

// one block sweep; the number of rotations (< 0: an error) and the largest |cos| of a rotated pair
long long col_block_sweep(bool cplx, int m, int n, float *Gr, float *Gi, float *Wr, float *Wi, float tol, unsigned *cnt,
                          cudaStream_t s, float *mu)
{
  const cb::Shape sh = cb::shape(cplx, m, n);
  const int nc = sh.nc;
  void (*const k)(cb::Args) = cplx ? (nc == 8 ? cb::k_col_blocks<true, 8> : cb::k_col_blocks<true, 4>)
                                   : (nc == 16 ? cb::k_col_blocks<false, 16> : cb::k_col_blocks<false, 8>);
  const size_t sm = cb::smem(cplx, nc ? nc : 4, sh.cs ? sh.cs : 1, m, n);
  if (!nc || cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess ||
      cudaMemsetAsync(cnt, 0, 12, s) != cudaSuccess)
    return -1;
  cb::Args a{Gr, Gi, Wr, Wi, m, n, n / (nc / 2), 0, tol, cnt};
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)sh.cs;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  cfg.gridDim = dim3((unsigned)(a.nb / 2 * sh.cs));
  cfg.blockDim = dim3(cb::NT);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = s;
  for (a.step = 0; a.step < a.nb; ++a.step)
    if (cudaLaunchKernelEx(&cfg, k, a) != cudaSuccess)
      return -1;
  unsigned hc[3] = {0u, 0u, 1u};
  if (cudaGetLastError() != cudaSuccess || cudaMemcpyAsync(hc, cnt, 12, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess || hc[2])
    return -1;
  memcpy(mu, &hc[1], 4);
  return (long long)hc[0];
}

}  // namespace vj
