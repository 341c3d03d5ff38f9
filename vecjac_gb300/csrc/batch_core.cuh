// The batched SVD's per-matrix driver (svd_one): a team of CTAs (one, or the CTAs of a
// cluster) runs the reference's algorithm on one matrix (src/dvjsvd.c:78-638); and the
// batch's argument and shared-memory layouts. Kept apart from the kernel and its launcher
// (batch.cu) so that a host harness can run it with an emulated CTA.
//
// A step goes through the team's pairs in four phases: the dot products (LANES lanes per
// pair), the classification (a thread per pair: the 2x2 with its divisions costs a warp the
// same for one lane as for 32, so it is done by as few warps as hold the pairs), the rotation
// of a pair and the sums of squares of its new columns (a warp per pair), and the tails of
// the norms (a thread per pair). What the reference decides between the steps (rescaling, the
// retry after a norm overflow, errors) is decided by every thread from the same few words at
// the start of the next step, as in the one-launch-per-step kernel (jsvd.cu); a step has three
// barriers of a CTA and one of the team.
#pragma once
#include "pjs.cuh"
#include "svd_core.cuh"

namespace vj {

constexpr int BATCH_MAXN = 512;

// what the launches of one call share about the batch (batch.cu, k_plan)
struct BatchPlan {
  // work-queue heads: matrices for whole clusters, wide ones and the others for single CTAs
  unsigned next_large, next_wide, next;
  unsigned end_large, end_wide;  // one past the last large, wide matrix in the caller's order
  double limit, wide;            // a matrix of a larger cost (batch_cost) is large, wide
  unsigned on_sm[2][256];        // CTAs of each SM that have come to take single matrices, by launch
};

template <typename T> struct BatchArgs {
  long long count;
  const long long *m, *n, *offG, *offV, *offS;
  const int *order;
  T *G, *V, *eS, *fS;
  long long *info;
  BatchPlan *plan;
  int strategy;
  unsigned swp;
  int sms;   // SMs of the device
  int part;  // 0 all matrices, 1 large and wide ones, 2 the others
  int fill;  // the launch of the CTAs that the clusters leave room for
};

// what a step leaves for the next (three slots in turn: read, written, being cleared)
// (32-bit words: another CTA's shared memory takes 32-bit atomics)
struct BatchCtl {
  unsigned nmg;   // largest |.| of the transformed columns: the high word of its bits
  int ovf, edot;  // a norm overflowed; a dot product was not finite
};

template <typename T> struct BatchShared {
  BatchCtl ctl[3];
  unsigned swt[3];        // transformed pairs per sweep (slots in turn)
  unsigned long long mx;  // max |g_ij| over this CTA's columns (T bits)
  // this CTA's pairs of the step: scaled dot product (then the rotation's tangent), cosine,
  // class; the new columns' sums of squares and largest magnitudes
  T z[BATCH_MAXN / 2], c[BATCH_MAXN / 2], acc[BATCH_MAXN / 2][2];
  typename fp<T>::U cmx[BATCH_MAXN / 2][2];
  int code[BATCH_MAXN / 2];
};

// The CTAs that work on one matrix: this CTA's rank among them; their shared words are rank
// 0's (s0 of svd_one).
struct Team {
  int rank, size;
};

__device__ __forceinline__ void warp_sync()
{
#ifdef __CUDA_ARCH__
  __syncwarp();
#else
  __syncthreads();  // (a host harness's CTA is one warp)
#endif
}

// barrier of the team's threads; orders their memory accesses
__device__ __forceinline__ void team_sync(const Team &tm)
{
#ifdef __CUDA_ARCH__
  if (tm.size > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    return;
  }
#else
  (void)tm;
#endif
  __syncthreads();
}

// the address of this CTA's shared word p in the team's CTA r
template <typename P> __device__ __forceinline__ P *team_peer(const Team &tm, P *p, int r)
{
#ifdef __CUDA_ARCH__
  if (tm.size > 1) {
    unsigned long long d;
    asm("mapa.u64 %0, %1, %2;" : "=l"(d) : "l"((unsigned long long)p), "r"(r));
    return reinterpret_cast<P *>(d);
  }
#endif
  (void)tm;
  (void)r;
  return p;
}

// max and sum into a shared word of this CTA or of another of the cluster (as explicit
// operations on the cluster's shared memory: a generic atomic of an address that may be
// shared was seen to miss the other CTA's word)
__device__ __forceinline__ void team_max(unsigned *p, unsigned v)
{
#ifdef __CUDA_ARCH__
  asm volatile("red.relaxed.cluster.shared::cluster.max.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
#else
  *p = (v > *p) ? v : *p;  // (a host harness's lanes take turns)
#endif
}
__device__ __forceinline__ void team_add(unsigned *p, unsigned v)
{
#ifdef __CUDA_ARCH__
  asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
#else
  *p += v;
#endif
}

// the high word of a magnitude's bits, all that MG is needed for (its exponent, and whether
// it is finite), and a value with that high word
template <typename T> __device__ __forceinline__ unsigned hi_word(typename fp<T>::U b)
{
  return (sizeof(T) == 8) ? (unsigned)((unsigned long long)b >> 32) : (unsigned)b;
}
template <typename T> __device__ __forceinline__ T from_hi(unsigned h)
{
  return (sizeof(T) == 8) ? bitst<T>((unsigned long long)h << 32) : bitst<T>((unsigned long long)h);
}

__device__ __forceinline__ void step_pair(int strategy, unsigned n, unsigned st, unsigned k, unsigned &p,
                                          unsigned &q)
{
  if (strategy == 2)
    pair_rr(n, st, k, p, q);
  else
    pair_mod(n, st, k, p, q);
}

// A by 2^e, a column per warp
template <typename T>
__device__ void team_scale(T *A, long long rows, long long cols, int e, int gw, int GW)
{
  if (!e)
    return;
  for (long long j = gw; j < cols; j += GW)
    for (long long i = threadIdx.x & 31; i < rows; i += 32)
      A[j * rows + i] = scale2(A[j * rows + i], e);
}

#ifdef __CUDA_ARCH__
// pair_sumsq for columns whose scale factors are not normal
__device__ __noinline__ void pair_sumsq_rare(int m, const float *x, const float *y, unsigned mx, unsigned my, float &ax,
                                             float &ay)
{
  pair_sumsq<float>(m, x, y, mx, my, ax, ay);
}
// the largest of m, |x| and |y|, a NaN if one is one
__device__ __forceinline__ float max_nan(float m, float x, float y)
{
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(x), "f"(y));
  return r;
}
// the larger of m and |x|, a NaN if either is one
__device__ __forceinline__ float max_nan(float m, float x)
{
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(m), "f"(fabsf(x)));
  return r;
}
// A pair of FP32 columns of up to 32 K rows in registers: rotated (rot_real of svd_core.cuh),
// written back, and the new columns' largest magnitudes and sums of squares (pair_sumsq, the same
// values in the same order) from the registers, so that a rotation waits for memory once: for the
// loads of G's and V's columns together. Rows of a lane are 32 apart, as the sums take them, and
// two of them share a packed operation.
template <int K> struct ColsF32 {
  float u[K], w[K];
  __device__ __forceinline__ void load(int rows, const float *x, const float *y)
  {
    const int lane = (int)(threadIdx.x & 31u);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const bool in = lane + 32 * k < rows;
      u[k] = in ? x[lane + 32 * k] : 0.0f;
      w[k] = in ? y[lane + 32 * k] : 0.0f;
    }
  }
  __device__ __forceinline__ void rotate(float at, float c)
  {
    const F32x2 t = f2_make(at, at), tn = f2_make(-at, -at), cc = f2_make(c, c);
    const bool cone = (c == 1.0f);
#pragma unroll
    for (int k = 0; k < K; k += 2) {
      const F32x2 x = f2_make(u[k], u[k + 1]), y = f2_make(w[k], w[k + 1]);
      F32x2 a = f2_fma(y, t, x), b = f2_fma(x, tn, y);
      if (!cone) {
        a = f2_mul(a, cc);
        b = f2_mul(b, cc);
      }
      f2_get(a, u[k], u[k + 1]);
      f2_get(b, w[k], w[k + 1]);
    }
  }
  __device__ __forceinline__ void store(int rows, float *x, float *y) const
  {
    const int lane = (int)(threadIdx.x & 31u);
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (lane + 32 * k < rows) {
        x[lane + 32 * k] = u[k];
        y[lane + 32 * k] = w[k];
      }
  }
};
template <int K>
__device__ __forceinline__ void rot_sum_f32(int m, int n, float *x, float *y, float *vx, float *vy, float at, float c,
                                            bool perm, unsigned (&mx)[2], float &ax, float &ay)
{
  ColsF32<K> g, v;
  g.load(m, x, y);
  v.load(n, vx, vy);
  g.rotate(at, c);
  g.store(m, perm ? y : x, perm ? x : y);
  v.rotate(at, c);
  v.store(n, perm ? vy : vx, perm ? vx : vy);
  float mu = 0.0f, mw = 0.0f;
#pragma unroll
  for (int k = 0; k < K; k += 2) {
    mu = max_nan(mu, g.u[k], g.u[k + 1]);
    mw = max_nan(mw, g.w[k], g.w[k + 1]);
  }
  const unsigned bu = warp_max_bits(fp<float>::bits(mu)), bw = warp_max_bits(fp<float>::bits(mw));
  mu = fp<float>::val(bu);
  mw = fp<float>::val(bw);
  const int ku = (bu && visfinite(mu)) ? -ilogb_(mu) : 0, kw = (bw && visfinite(mw)) ? -ilogb_(mw) : 0;
  constexpr int B = fp<float>::BIAS;
  mx[0] = perm ? bw : bu;
  mx[1] = perm ? bu : bw;
  if (ku >= 1 - B && ku <= B && kw >= 1 - B && kw <= B) {
    const F32x2 pu = f2_make(pow2<float>(ku), pow2<float>(ku)), pw = f2_make(pow2<float>(kw), pow2<float>(kw));
    float su = 0.0f, sw = 0.0f;
#pragma unroll
    for (int k = 0; k < K; k += 2) {
      float a0, a1, b0, b1;
      f2_get(f2_mul(f2_make(g.u[k], g.u[k + 1]), pu), a0, a1);
      f2_get(f2_mul(f2_make(g.w[k], g.w[k + 1]), pw), b0, b1);
      su = __fmaf_rn(a1, a1, __fmaf_rn(a0, a0, su));
      sw = __fmaf_rn(b1, b1, __fmaf_rn(b0, b0, sw));
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      su = su + __shfl_down_sync(0xffffffffu, su, o);
      sw = sw + __shfl_down_sync(0xffffffffu, sw, o);
    }
    ax = perm ? sw : su;
    ay = perm ? su : sw;
  }
  else {
    __syncwarp();
    pair_sumsq_rare(m, x, y, mx[0], mx[1], ax, ay);
  }
}
// rot_real (svd_core.cuh) for longer FP32 columns at 8-byte boundaries and one warp: two rows per
// load and packed FMAs; m is a multiple of 16. UR loads of two rows in flight.
struct RotF32 {
  F32x2 t, tn, c;
  const unsigned long long *rx, *ry;
  unsigned long long *dx, *dy;
  float mu, mw;
};
template <bool TRACK, int UR> __device__ __forceinline__ void rot_f32_rows(RotF32 &r, int i, bool cone)
{
  F32x2 u[UR], w[UR];
#pragma unroll
  for (int k = 0; k < UR; ++k) {
    u[k].v = r.rx[i + 32 * k];
    w[k].v = r.ry[i + 32 * k];
  }
#pragma unroll
  for (int k = 0; k < UR; ++k) {
    F32x2 a = f2_fma(w[k], r.t, u[k]), b = f2_fma(u[k], r.tn, w[k]);
    if (!cone) {
      a = f2_mul(a, r.c);
      b = f2_mul(b, r.c);
    }
    r.dx[i + 32 * k] = a.v;
    r.dy[i + 32 * k] = b.v;
    if (TRACK) {
      float a0, a1, b0, b1;
      f2_get(a, a0, a1);
      f2_get(b, b0, b1);
      r.mu = max_nan(max_nan(r.mu, a0), a1);
      r.mw = max_nan(max_nan(r.mw, b0), b1);
    }
  }
}
template <bool TRACK>
__device__ __forceinline__ void rot_f32(int m, float *x, float *y, float at, float c, bool perm, unsigned &mx,
                                        unsigned &my)
{
  const bool cone = (c == 1.0f);
  RotF32 r;
  r.t = f2_make(at, at);
  r.tn = f2_make(-at, -at);
  r.c = f2_make(c, c);
  r.rx = reinterpret_cast<const unsigned long long *>(x);
  r.ry = reinterpret_cast<const unsigned long long *>(y);
  r.dx = reinterpret_cast<unsigned long long *>(perm ? y : x);
  r.dy = reinterpret_cast<unsigned long long *>(perm ? x : y);
  r.mu = r.mw = 0.0f;
  const int h = m >> 1;
  int i = (int)(threadIdx.x & 31u);
  for (; i + 96 < h; i += 128)
    rot_f32_rows<TRACK, 4>(r, i, cone);
  if (i + 32 < h) {
    rot_f32_rows<TRACK, 2>(r, i, cone);
    i += 64;
  }
  if (i < h)
    rot_f32_rows<TRACK, 1>(r, i, cone);
  if (TRACK) {
    mx = fp<float>::bits(perm ? r.mw : r.mu);
    my = fp<float>::bits(perm ? r.mu : r.mw);
  }
}
#endif

// the norm from its scaled sum of squares; the same as warp_nrm2's
template <typename T> __device__ __forceinline__ T finish_nrm(T acc, typename fp<T>::U mx)
{
  const T a = fp<T>::val(mx);
  if (!visfinite(a))
    return visnan(a) ? fp<T>::qnan() : a;
  if (mx == 0)
    return (T)0;
  return scale2(sqrt_ge1(acc), ilogb_(a));  // (the largest magnitude scales to [1, 2): acc >= 1)
}

// What a step needs seldom or once per round is kept out of line: inlined, its registers would
// be taken from the loops over the rows (FP32 at 64 registers: 1256 bytes of spills).
// a pair's class and rotation
template <typename T> struct PairClass {
  T c, cat;
  int code, trans;
};
template <typename T> __device__ __noinline__ PairClass<T> classify_pair(T ep, T fp_, T eq, T fq, T zr, T tol, T gst)
{
  PairState<T> s;
  s.c = (T)1;
  s.cat = (T)0;
  const bool t = pair_classify<T, false>(ep, fp_, eq, fq, zr, (T)0, tol, gst, s);
  return PairClass<T>{s.c, s.cat, s.code, t ? 1 : 0};
}
// everything but a rotation: shears, swaps and rotations by nothing (pair_apply); mx: the
// changed columns' largest |.|, or false
template <typename T>
__device__ __noinline__ bool apply_other(const PairState<T> &b, int m, int n, T *Gp, T *Gq, T *Vp, T *Vq, T *eSp, T *eSq,
                                         T *fSp, T *fSq, typename fp<T>::U (&mx)[2])
{
  typename fp<T>::U mV = 0;
  return pair_apply<T, false, false, 4>(b, m, n, Gp, Gq, nullptr, nullptr, Vp, Vq, nullptr, nullptr, Gp, Gq, nullptr,
                                        nullptr, eSp, eSq, fSp, fSq, (int)(threadIdx.x & 31u), 32, false, mx, mV);
}
// the columns' largest |.| (of this lane's rows)
template <typename T> __device__ __noinline__ void cols_max(int m, const T *x, const T *y, typename fp<T>::U (&mx)[2])
{
#pragma unroll 4
  for (int i = (int)(threadIdx.x & 31u); i < m; i += 32) {
    amax(mx[0], x[i]);
    amax(mx[1], y[i]);
  }
}
// norm of column c into eS, fS; *ovf set when it overflows
template <typename T> __device__ __noinline__ void one_norm(int m, const T *x, T *eS, T *fS, int *ovf)
{
  const T d = warp_nrm2(x, m);
  if ((threadIdx.x & 31u) == 0) {
    T e, f;
    ef_split(d, e, f);
    *eS = e;
    *fS = f;
    if (!(d <= svdc<T>::RMAX))
      *(volatile int *)ovf = 1;
  }
}
// a norm from its sum of squares into eS, fS; whether it overflows
template <typename T> __device__ __noinline__ bool put_norm(T acc, typename fp<T>::U mx, T *eS, T *fS)
{
  const T d = finish_nrm<T>(acc, mx);
  T e, f;
  ef_split(d, e, f);
  *eS = e;
  *fS = f;
  return !(d <= svdc<T>::RMAX);
}

// an FP64 dot product (its registers apart: 1500 matrices of up to 128 rows 109.5 -> 105.1 ms; FP32
// ones are faster with theirs shared)
__device__ __noinline__ double far_nu(int m, const double *x, const double *y, double ex, double ey, bool live)
{
  double zr, zi;
  pair_nu<double, false>(m, x, nullptr, y, nullptr, ex, ey, live, zr, zi);
  return zr;
}

// the whole SVD of one matrix by this team; returns the sweep count or an error code
template <typename T>
__device__ long long svd_one(const BatchArgs<T> &a, BatchShared<T> &sh, long long m_, long long n_, T *G, T *V, T *eS,
                             T *fS, Team tm = Team{0, 1}, BatchShared<T> *s0 = nullptr)
{
  using F = fp<T>;
  using U = typename F::U;
  constexpr int L = svdc<T>::LANES;
  constexpr int PW = 32 / L;  // pairs whose dot products a warp forms at once
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int gw = tm.rank * nw + warp, GW = tm.size * nw;  // this warp among the team's
  if (!s0)
    s0 = &sh;
  if (!n_)
    return 0;
  if (m_ < n_ || (m_ % L) || m_ > 0x7fffffffLL)
    return -1;
  if ((n_ & 1) || ((n_ >> 1) % L) || n_ > BATCH_MAXN)
    return -2;
  const int m = (int)m_, n = (int)n_, n_2 = n >> 1;
  // column c of G (a column's rows are an int, the matrix's elements need not be)
  auto col = [&](int c) { return G + (size_t)c * (size_t)m; };
  const long long E_MG = -80, E_DOT = -320, E_APPG = -580;
  if (tid == 0) {
    for (int k = 0; k < 3; ++k) {
      sh.ctl[k] = BatchCtl{};
      sh.swt[k] = 0u;
    }
    sh.mx = 0ull;
  }
  __syncthreads();
  {
    // max |g_ij| (a NaN counts as inf, as VMINPD(|x|, inf) maps it); V := I, eS = -inf, fS = 1
    const U inf = F::bits(F::inf());
    U mx = 0;
    for (int j = gw; j < n; j += GW) {
      const T *x = col(j);
      for (int i = lane; i < m; i += 32) {
        U b = F::bits(x[i]) & ~F::SIGN;
        b = (b > inf) ? inf : b;
        mx = (b > mx) ? b : mx;
      }
      for (int i = lane; i < n; i += 32)
        V[j * n + i] = (i == j) ? (T)1 : (T)0;
      if (lane == 0) {
        eS[j] = vneg(F::inf());
        fS[j] = (T)1;
      }
    }
    mx = warp_max_bits(mx);
    if (lane == 0 && mx)
      atomicMax(&sh.mx, (unsigned long long)mx);
  }
  team_sync(tm);
  T MG = (T)0;
  {
    unsigned long long mx = 0ull;
    for (int r = 0; r < tm.size; ++r) {
      const unsigned long long v = *(volatile unsigned long long *)team_peer(tm, &sh.mx, r);
      mx = (v > mx) ? v : mx;
    }
    MG = bitst<T>(mx);
  }
  if (tm.size > 1)
    team_sync(tm);  // (a CTA may leave and reuse its words only when all have read them)
  if (!(MG <= svdc<T>::RMAX))
    return E_MG;
  if (MG == (T)0)
    return 0;
  // global prescale (src/dvjsvd.c:120-137)
  const int ROT = svdc<T>::ROT_R;
  const T M_m = F::div(svdc<T>::RMAX, (T)((unsigned long long)m << 1u));
  const int NRM = ilogb_(M_m);
  int sN = NRM - ilogb_(MG) - 1;
  if (sN) {
    team_scale(G, m, n, sN, gw, GW);
    MG = scale2(MG, sN);
  }
  int sT = sN;
  const T tol = F::sqrt_((T)m) * scale2(svdc<T>::EPS, -1);
  const T gst = scale2(tol, (int)svdc<T>::MAX_FIN_EXP);
  // norms of all columns, a column per warp (the columns that this warp has just scaled)
  auto all_norms = [&](int *ovf) {
    for (int c = gw; c < n; c += GW)
      one_norm<T>(m, col(c), eS + c, fS + c, ovf);
  };
  const unsigned stp = (a.strategy == 2) ? (unsigned)(n - 1) : (unsigned)n;
  const unsigned swp = a.swp;
  if (swp) {
    warp_sync();
    all_norms(&s0->ctl[0].ovf);
  }
  team_sync(tm);
  // (FP32 columns are rotated two rows per load where they start at 8-byte boundaries)
  const bool al8 = !(((uintptr_t)G | (uintptr_t)V) & 7u);
  (void)al8;
  // this CTA's groups of PW pairs (dealt out to the team's CTAs in turn) and its pairs
  const int litems = (n_2 / PW - tm.rank + tm.size - 1) / tm.size, lpairs = litems * PW;
  unsigned sw = 0, g = 0;
  while (sw < swp) {
    unsigned cnt = 0;  // this lane's transformed pairs of the sweep
    for (unsigned st = 0; st < stp; ++st, ++g) {
      // ---- between the steps (src/dvjsvd.c:199-233, :276-295), decided by every thread alike ----
      const BatchCtl *cur = &s0->ctl[g % 3u];
      BatchCtl *nxt = &s0->ctl[(g + 1u) % 3u];
      const T nMG = from_hi<T>(*(volatile const unsigned *)&cur->nmg);
      const int ovf = *(volatile const int *)&cur->ovf, edot = *(volatile const int *)&cur->edot;
      if (tm.rank == 0 && tid == 0) {
        BatchCtl *clr = &s0->ctl[(g + 2u) % 3u];
        clr->nmg = 0u;
        clr->ovf = 0;
        clr->edot = 0;
      }
      if (edot || !visfinite(nMG)) {
        if (tm.size > 1)
          team_sync(tm);
        return edot ? E_DOT : E_APPG;
      }
      MG = fmax(MG, nMG);
      const int eM = ilogb_(MG);
      const bool gres = (ROT - eM < 0);
      if (gres || ovf) {
        // G's own rescaling, or (the reference's retry) by the exponent that the V block has
        // set, ROT - 0; then every norm anew
        const int e = gres ? (NRM - eM - 1) : ROT;
        team_sync(tm);  // every thread has read the slot
        if (tm.rank == 0 && tid == 0)
          s0->ctl[g % 3u].ovf = 0;
        team_sync(tm);
        team_scale(G, m, n, e, gw, GW);
        MG = scale2(MG, e);
        sT += e;
        warp_sync();
        all_norms(&s0->ctl[g % 3u].ovf);
        team_sync(tm);
        const int again = *(volatile const int *)&s0->ctl[g % 3u].ovf;
        if (tm.size > 1)
          team_sync(tm);
        if (again)
          return (long long)VJ_ERR_ARG;
      }
      const bool last = (sw + 1u == swp) && (st + 1u == stp);
      // the global pair and the columns of this CTA's pair lp (items of PW pairs are dealt out
      // to the team's CTAs in turn)
      auto pair_of = [&](int lp, unsigned &p, unsigned &q) {
        step_pair(a.strategy, (unsigned)n, st, (unsigned)(((lp / PW) * tm.size + tm.rank) * PW + lp % PW), p, q);
      };
      // ---- scaled dot products (src/dvjsvd.c:297-348), PW pairs per warp ----
      for (int li = warp; li < litems; li += nw) {
        const int lp = li * PW + lane / L;
        unsigned p, q;
        pair_of(lp, p, q);
        const T ep = eS[p], eq = eS[q];
        const bool live = (eq >= -svdc<T>::RMAX) && (ep >= -svdc<T>::RMAX);
        T zr, zi;
        if constexpr (sizeof(T) == 8)
          zr = far_nu(m, col(q), col(p), live ? eq : (T)0, live ? ep : (T)0, live);
        else
          pair_nu<T, false>(m, col(q), nullptr, col(p), nullptr, live ? eq : (T)0, live ? ep : (T)0, live, zr, zi);
        if (lane % L == 0)
          sh.z[lp] = live ? zr : (T)0;
      }
      __syncthreads();
      // ---- convergence test, 2x2, classification, a pair per thread (src/dvjsvd.c:349-459) ----
      for (int lp = tid; lp < lpairs; lp += (int)blockDim.x) {
        unsigned p, q;
        pair_of(lp, p, q);
        const T ep = eS[p], fp_ = fS[p], eq = eS[q], fq = fS[q];
        const T z = qdiv(sh.z[lp], fq * fp_);
        PairClass<T> s{(T)1, (T)0, 1, 0};
        if (!visfinite(z))
          *(volatile int *)&nxt->edot = 1;
        else {
          s = classify_pair<T>(ep, fp_, eq, fq, z, tol, gst);
          cnt += (unsigned)s.trans;
        }
        if (s.code == -1) {
          eS[p] = eq; eS[q] = ep;
          fS[p] = fq; fS[q] = fp_;
        }
        // (a shear needs the dot product itself and the old norms)
        const bool shear = (s.code == 3 || s.code == -3);
        sh.z[lp] = shear ? z : s.cat;
        sh.c[lp] = s.c;
        sh.code[lp] = s.code;
      }
      __syncthreads();
      // ---- transformations (src/dvjsvd.c:460-574) and the new columns' sums of squares
      // (:236-275), a pair per warp ----
      U mG = 0;
      for (int lp = warp; lp < lpairs; lp += nw) {
        const int code = sh.code[lp];
        if (code == 1)
          continue;
        unsigned p, q;
        pair_of(lp, p, q);
        T *Gp = col(p), *Gq = col(q), *Vp = V + p * n, *Vq = V + q * n;
        const T at = sh.z[lp], cc = sh.c[lp];
        U mx[2] = {0, 0};
        bool trk = true, have = false;  // have: the sums of squares, too
        T ax = (T)0, ay = (T)0;
        if ((code == 2 || code == -2) && at != (T)0) {
          U d0, d1;
          bool done = false;
#ifdef __CUDA_ARCH__
          if constexpr (sizeof(T) == 4)
            if (m <= 256) {
              if (m <= 128)
                rot_sum_f32<4>(m, n, Gp, Gq, Vp, Vq, at, cc, code == -2, mx, ax, ay);
              else
                rot_sum_f32<8>(m, n, Gp, Gq, Vp, Vq, at, cc, code == -2, mx, ax, ay);
              have = done = true;
            }
            else if (al8) {
              rot_f32<true>(m, Gp, Gq, at, cc, code == -2, mx[0], mx[1]);
              rot_f32<false>(n, Vp, Vq, at, cc, code == -2, d0, d1);
              done = true;
            }
#endif
          if (!done) {
            trk = (sizeof(T) == 4);  // (FP64: the columns' largest entries by a pass of their own, svd_core.cuh)
            rot_real<T, false, 4>(m, Gp, Gq, Gp, Gq, nullptr, nullptr, at, cc, code == -2, lane, 32, trk, mx[0], mx[1]);
            rot_real<T, false, 4>(n, Vp, Vq, Vp, Vq, nullptr, nullptr, at, cc, code == -2, lane, 32, false, d0, d1);
          }
        }
        else {
          PairState<T> b;
          b.code = code;
          b.skip = 0;
          b.c = cc;
          b.cat = b.a21r = at;
          b.sat = b.a21i = (T)0;
          b.ep = eS[p];
          b.eq = eS[q];
          b.fp = fS[p];
          b.fq = fS[q];
          warp_sync();  // (a permuting shear exchanges the norms)
          trk = apply_other<T>(b, m, n, Gp, Gq, Vp, Vq, eS + p, eS + q, fS + p, fS + q, mx);
        }
        if (code == -1)
          continue;
        if (!have) {
          warp_sync();  // the columns as written by the other lanes
          if (!trk)
            cols_max<T>(m, Gp, Gq, mx);
          mx[0] = warp_max_bits(mx[0]);
          mx[1] = warp_max_bits(mx[1]);
        }
        mG = (mx[0] > mG) ? mx[0] : mG;
        mG = (mx[1] > mG) ? mx[1] : mG;
        if (last)
          continue;
        if (!have)
          pair_sumsq<T>(m, Gp, Gq, mx[0], mx[1], ax, ay);
        if (lane == 0) {
          sh.acc[lp][0] = ax;
          sh.acc[lp][1] = ay;
          sh.cmx[lp][0] = mx[0];
          sh.cmx[lp][1] = mx[1];
        }
      }
      if (lane == 0 && mG)
        team_max(&nxt->nmg, hi_word<T>(mG));
      __syncthreads();
      // ---- the norms' tails, a pair per thread ----
      if (!last)
        for (int lp = tid; lp < lpairs; lp += (int)blockDim.x) {
          const int code = sh.code[lp];
          if (code == 1 || code == -1)
            continue;
          unsigned p, q;
          pair_of(lp, p, q);
          bool o = false;
          if (code == 2 || code == -2)
            o = put_norm<T>(sh.acc[lp][0], sh.cmx[lp][0], eS + p, fS + p);
          if (put_norm<T>(sh.acc[lp][1], sh.cmx[lp][1], eS + q, fS + q) || o)
            *(volatile int *)&nxt->ovf = 1;
        }
      if (st + 1u == stp && cnt)
        team_add(&s0->swt[sw % 3u], cnt);
      team_sync(tm);
    }
    const unsigned swt = *(volatile unsigned *)&s0->swt[sw % 3u];
    if (tm.rank == 0 && tid == 0)
      s0->swt[(sw + 1u) % 3u] = 0u;
    // the last step's errors
    const BatchCtl *cur = &s0->ctl[g % 3u];
    const T nMG = from_hi<T>(*(volatile const unsigned *)&cur->nmg);
    const int edot = *(volatile const int *)&cur->edot;
    if (edot || !visfinite(nMG)) {
      if (tm.size > 1)
        team_sync(tm);
      return edot ? E_DOT : E_APPG;
    }
    if (!swt)
      break;
    ++sw;
  }
  if (sw < swp) {
    // U = G diag(1/f) 2^-e and eS -= sT (src/dvjsvd.c:604-631); V was never rescaled
    for (int j = gw; j < n; j += GW) {
      const T f = fS[j], e = eS[j], sc = vneg(e);
      T *x = col(j);
      for (int i = lane; i < m; i += 32)
        x[i] = scalef(qdiv(x[i], f), sc);
      warp_sync();
      if (lane == 0)
        eS[j] = e - (T)sT;
    }
  }
  team_sync(tm);
  return (long long)sw;
}

}  // namespace vj
