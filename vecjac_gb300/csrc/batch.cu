// Batched one-sided Jacobi SVD: thousands of independent matrices of uneven size in one call
// of persistent launches (real FP64 and FP32; every matrix with dvjsvd_'s / svjsvd_'s
// result).
//
// A matrix is worked on by one CTA, or, when it is so large that its CTA would finish after
// the rest of the batch and clusters do them sooner (k_plan), by a cluster of BATCH_CS CTAs (svd_one's
// team, batch_core.cuh). Each team runs the reference driver on its matrix (src/dvjsvd.c:78-638). Matrices
// are handed out by atomic work queues in the order the caller gives (largest first balances the tail); a matrix stops at its own convergence (its own sweep
// count, its own info entry), so uneven convergence does not hold the batch back. Pivot pairs
// are computed on the fly from the strategy's closed form (pjs.cuh), so no tables are stored.
// Matrix sizes: m >= n, n <= 512, and the reference's divisibility rules (the host wrapper
// pads with zero rows/columns).
#include <cuda_runtime.h>

#include "batch_core.cuh"

namespace vj {

// CTAs per cluster: 300 FP32 matrices of up to 512 rows take 717 ms by single CTAs and 171 ms in clusters
// of 4 (119 ms in clusters of 8), 1500 FP64 ones of up to 128 rows 129, 117 and 145 ms: a cluster
// larger than its matrix leaves CTAs idle.
constexpr int BATCH_CS = 4;

// What a matrix gains from a cluster over a CTA, by the groups of pairs per warp of a CTA: measured
// alone on the GPU, FP64 1.5, 2.0, 3.0 and 3.6 times at 1, 2, 4 and 8 groups per warp (128 x 64 to 512 x
// 256 by 256 and 128 threads), FP32 1.2, 1.5, 1.9, 2.4 and 3.0 at 1 to 16 (more where single CTAs'
// matrices would not fit in L2 together: 152 of 512 x 256 106 ms by clusters, 155 by CTAs).
template <typename T> __device__ __forceinline__ double team_gain(long long n, int warps)
{
  const float r = fmaxf((float)n / (float)(2 * (32 / svdc<T>::LANES) * warps), 0.25f);
  const float g = (sizeof(T) == 8) ? 1.5f * sqrtf(r) : 1.25f * exp2f(0.42f * log2f(r));
  return (double)fminf(fmaxf(g, 1.05f), (sizeof(T) == 8) ? 3.7f : 3.2f);
}

// Unless the caller sets the number of CTAs per SM, the batch is done in two parts: the large
// matrices and the wide ones, whose cost is more than BATCH_WIDE of a CTA's share of the batch, by
// two CTAs of 128 registers per SM, and the others by four CTAs of 64 registers, which start as the
// first launch's end. A matrix is done sooner by one of two CTAs than of four, which counts at the
// end of the batch; many small ones are done sooner by four, whose waits for memory and for the few
// threads of a 2x2 overlap. (The first part has a second launch, of the CTAs that its clusters leave room
// for, batch_dev.) 4000 FP32 matrices of up to 256 rows: 141 ms (two CTAs 141, four 154),
// 1500 FP64 ones of up to 128 rows: 105 ms (105, 115), 4000 FP64 16 x 16: 16.8 ms (22.3, 17.2),
// 4000 FP32 64 x 32: 10.1 ms (11.8, 10.6). With a smaller BATCH_WIDE, 2000 FP64 64 x 64 take 154
// instead of 141 ms, with a larger one the uneven batches 151 and 119 ms (at 0.6).
constexpr double BATCH_WIDE = 0.15;

// a matrix's work, up to its number of sweeps
__device__ __forceinline__ double batch_cost(long long m, long long n)
{
  return (n > 0 && m > 0) ? (double)n * (double)n * (double)(m + n) : 0.0;
}

// The queues' heads and the sizes from which a matrix is large (done by a cluster) and wide, for `teams`
// clusters, `slots` CTAs of `warps` warps in all. Large is what costs more than a CTA slot would have of
// the batch and has enough groups of pairs for more than the warps of one CTA, or nothing, where
// single CTAs would be done sooner: the times of both are estimated in units of a matrix's cost on an SM
// of its own, from the clusters' matrices in rounds (the last, partly filled one at 0.8), all work at
// the rates of clusters and of single CTAs (two on an SM take 1.45 times as long as one: an SM's rate
// grows with the root of their number; half of the longest matrix where they queue), and the longest single matrix
// after the clusters that it waits for. Equal matrices, one per SM, went through the clusters in three
// rounds before: 152 FP64 128 x 64 42 ms, 22 by single CTAs, 152 FP32 304 x 32 3.9 and 1.5; uneven ones
// keep their clusters (300 FP64 of up to 128 rows 45 ms, 135 without). One CTA of 1024 threads.
template <typename T>
__global__ void __launch_bounds__(1024) k_plan(BatchArgs<T> a, int teams, int slots, int warps)
{
  // sums: cost of all, number and time of the large ones, cost of the others; maxima: cost of all, time of
  // the large ones, cost of the others; minimum: time of the large ones
  enum { ALL, NUM, TIME, OTHERS, MOST, TMOST, OMOST, TLEAST, NV };
  __shared__ double sh[NV][32];
  __shared__ unsigned end, endw;
  const int tid = threadIdx.x;
  double v[NV] = {0, 0, 0, 0, 0, 0, 0, 1e300};
  // the values of `mask` over all threads, to every one of them
  auto reduce = [&](unsigned mask) {
    auto warp = [&](int k) {
      for (int o = 16; o >= 1; o >>= 1) {
        const double w = __shfl_xor_sync(0xffffffffu, v[k], o);
        v[k] = (k < MOST) ? v[k] + w : (k < TLEAST) ? fmax(v[k], w) : fmin(v[k], w);
      }
    };
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (mask >> k & 1u) {
        warp(k);
        if ((tid & 31) == 0)
          sh[k][tid >> 5] = v[k];
      }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (mask >> k & 1u) {
        v[k] = sh[k][tid & 31];
        warp(k);
      }
  };
  for (long long i = tid; i < a.count; i += blockDim.x) {
    const double w = batch_cost(a.m[i], a.n[i]);
    v[ALL] += w;
    v[MOST] = fmax(v[MOST], w);
  }
  if (tid == 0)
    end = endw = 0u;
  reduce(1u << ALL | 1u << MOST);
  const double c = v[ALL];
  const double nmin = 2.0 * (32 / svdc<T>::LANES) * warps;  // columns that one CTA's warps take at once
  double limit = fmax(c / slots, 2.0 * nmin * nmin * nmin);
  if (v[MOST] > limit) {
    for (long long i = tid; i < a.count; i += blockDim.x) {
      const double w = batch_cost(a.m[i], a.n[i]);
      if (w > limit) {
        const double t = w / team_gain<T>(a.n[i], warps);
        v[NUM] += 1;
        v[TIME] += t;
        v[TMOST] = fmax(v[TMOST], t);
        v[TLEAST] = fmin(v[TLEAST], t);
      }
      else {
        v[OTHERS] += w;
        v[OMOST] = fmax(v[OMOST], w);
      }
    }
    reduce(1u << NUM | 1u << TIME | 1u << OTHERS | 1u << TMOST | 1u << OMOST | 1u << TLEAST);
    const double rate = sqrt((double)a.sms * (double)slots), t = v[TIME] / teams;
    const double rounds = fmax(v[TMOST], t + ((v[NUM] > teams) ? 0.8 * v[TLEAST] : 0.0));
    const double with = fmax(fmax(rounds, t + v[OTHERS] / rate + (((double)a.count - v[NUM] > slots) ? 0.5 * v[OMOST] : 0.0)),
                             ((v[NUM] >= teams) ? t : 0.0) + v[OMOST]);
    const double without = fmax(v[MOST], c / rate + ((a.count > slots) ? 0.5 * v[MOST] : 0.0));
    if (without <= with)
      limit = 1e300;
  }
  for (long long i = tid; i < a.count; i += blockDim.x) {
    const int b = a.order ? a.order[i] : (int)i;
    if (batch_cost(a.m[b], a.n[b]) > limit)
      atomicMax(&end, (unsigned)(i + 1));
    if (batch_cost(a.m[b], a.n[b]) > BATCH_WIDE * c / slots)
      atomicMax(&endw, (unsigned)(i + 1));
  }
  if (tid < 512)
    a.plan->on_sm[tid >> 8][tid & 255] = 0u;
  __syncthreads();
  if (tid == 0) {
    a.plan->next_large = 0u;
    a.plan->next_wide = 0u;
    a.plan->next = 0u;
    a.plan->end_large = end;
    a.plan->end_wide = endw;
    a.plan->limit = limit;
    a.plan->wide = BATCH_WIDE * c / slots;
  }
}

// (one copy of the driver for the two places that call it)
template <typename T>
__device__ __noinline__ void svd_matrix(const BatchArgs<T> &a, BatchShared<T> &sh, int b, Team tm, BatchShared<T> *s0)
{
  const long long r = svd_one<T>(a, sh, a.m[b], a.n[b], a.G + a.offG[b], a.V + a.offV[b], a.eS + a.offS[b],
                                 a.fS + a.offS[b], tm, s0);
  if (threadIdx.x == 0 && tm.rank == 0)
    a.info[b] = r;
}

// MINB: the register bound for MINB resident CTAs of 256 threads per SM (more, smaller
// CTAs when the caller launches fewer threads per CTA). The best bound depends on the
// batch (the autotuner of vecjac_gb300/batch.py searches it with the CTA size); a.part says which
// of the batch's matrices the launch does.
template <typename T, int MINB>
__global__ void __launch_bounds__(256, MINB) k_batch(BatchArgs<T> a)
{
  __shared__ BatchShared<T> sh;
  __shared__ long long s_b[2];
  unsigned rank, size;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
  BatchPlan *const plan = a.plan;
  const double limit = plan->limit, widec = plan->wide;
  const unsigned end = plan->end_large;
  auto large = [&](int b) { return batch_cost(a.m[b], a.n[b]) > limit; };
  if (a.part != 2)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // the large matrices, by whole clusters
  if (end && size > 1u) {
    const Team tm{(int)rank, (int)size};
    // rank 0's shared words as seen from this CTA
    BatchShared<T> *const s0 = team_peer(tm, &sh, 0);
    volatile long long *const b0 = team_peer(tm, s_b, 0);
    for (int it = 0;; it ^= 1) {
      if (rank == 0 && threadIdx.x == 0) {
        long long got = -1;
        for (;;) {
          const unsigned i = atomicAdd(&plan->next_large, 1u);
          if (i >= end)
            break;
          const int b = a.order ? a.order[i] : (int)i;
          if (large(b)) {
            got = b;
            break;
          }
        }
        s_b[it] = got;
      }
      team_sync(tm);
      const long long b = b0[it];
      if (b < 0)
        break;
      svd_matrix<T>(a, sh, (int)b, tm, s0);
    }
    team_sync(tm);  // no CTA's shared words are read by another from here on
  }
  // the others, by single CTAs: the r-th CTA of an SM takes part when there are more than r
  // matrices per SM, so that few matrices spread over the SMs (108 FP64 matrices of up to 35
  // rows: 9.2 ms when the two CTAs of an SM may both take one, 7.1 ms apart)
  const bool split = end && (size > 1u || a.part == 2 || a.fill);
  if (threadIdx.x == 0) {
    unsigned sm;
    asm("mov.u32 %0, %%smid;" : "=r"(sm));
    s_b[1] = (long long)atomicAdd(&plan->on_sm[a.part == 2][sm & 255u], 1u);
  }
  __syncthreads();
  unsigned *const head = (a.part == 1) ? &plan->next_wide : &plan->next;
  const long long stop = (s_b[1] * (long long)a.sms >= a.count) ? 0
                         : (a.part == 1)                        ? (long long)plan->end_wide
                                                                : a.count;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      long long got = -1;
      for (;;) {
        const long long i = stop ? (long long)atomicAdd(head, 1u) : 0;
        if (i >= stop)
          break;
        const int b = a.order ? a.order[i] : (int)i;
        const bool mine = a.part == 0 || (batch_cost(a.m[b], a.n[b]) > widec) == (a.part == 1);
        if (mine && !(split && i < (long long)end && large(b))) {
          got = b;
          break;
        }
      }
      s_b[0] = got;
    }
    __syncthreads();
    const long long b = s_b[0];
    if (b < 0)
      break;
    svd_matrix<T>(a, sh, (int)b, Team{0, 1}, &sh);
  }
  // (the launch ends when the one before has, too; one CTA waits for it, the others make room)
  if ((a.part == 2 || a.fill) && blockIdx.x == 0)
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// the call's launches (occ 0: the default's parts)
template <typename T> static vj_fint batch_launch(BatchArgs<T> a, int block, int occ, cudaStream_t s)
{
  const long long count = a.count;
  const bool parts = !occ;
  if (parts)
    occ = 2;
  a.part = parts ? 1 : 0;
  a.fill = 0;
  void (*k)(BatchArgs<T>) = (occ == 2)   ? k_batch<T, 2>
                            : (occ == 3) ? k_batch<T, 3>
                            : (occ == 4) ? k_batch<T, 4>
                            : (occ == 5) ? k_batch<T, 5>
                                         : k_batch<T, 6>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = BATCH_CS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(BATCH_CS);
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = s;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    clusters = 1;
  }
  const int slots = clusters * BATCH_CS;
  k_plan<T><<<1, 1024, 0, s>>>(a, clusters, slots, block / 32);
  // a cluster per matrix at most: every matrix may be large
  cfg.gridDim = dim3((unsigned)(((long long)clusters < count ? (long long)clusters : (long long)count) * BATCH_CS));
  if (cudaLaunchKernelEx(&cfg, k, a) != cudaSuccess)
    return VJ_ERR_CUDA;
  // The SMs that no cluster fits on (their number in a processing cluster is not always a multiple of
  // four) get single CTAs, in a launch that starts beside the first: 152 equal matrices otherwise find
  // 148 SMs and take two rounds (FP64 128 x 64: 42 ms).
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, block, 0) != cudaSuccess) {
    cudaGetLastError();
    per = 0;
  }
  const long long room = (long long)per * a.sms - slots;
  if (room > 0 && count > clusters) {
    a.fill = 1;
    if (host::launch_pdl(k, dim3((unsigned)(room < count ? room : (long long)count)), dim3((unsigned)block), 0, s, a) !=
        cudaSuccess)
      return VJ_ERR_CUDA;
    a.fill = 0;
  }
  if (parts) {
    // the others: these CTAs start as the first launch's end
    a.part = 2;
    void (*const k2)(BatchArgs<T>) = k_batch<T, 4>;
    per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k2, block, 0) != cudaSuccess || per < 1) {
      cudaGetLastError();
      per = 1;
    }
    const long long most = (long long)per * a.sms;
    if (host::launch_pdl(k2, dim3((unsigned)(most < count ? most : (long long)count)), dim3((unsigned)block), 0, s, a) !=
        cudaSuccess)
      return VJ_ERR_CUDA;
  }
  return (cudaGetLastError() == cudaSuccess) ? 0 : VJ_ERR_CUDA;
}

template <typename T>
static vj_fint batch_dev(vj_fint count, const long long *m, const long long *n, T *G, const long long *offG, T *V,
                         const long long *offV, T *eS, T *fS, const long long *offS, const int *order,
                         long strategy, unsigned swp, long long *info, int block, int occ, void *stream)
{
  if (count < 0 || (strategy != 2l && strategy != 4l))
    return VJ_ERR_ARG;
  if (!count)
    return 0;
  if (!host::gpu_ready())
    return VJ_ERR_NO_GPU;
  if (block != 64 && block != 128 && block != 256)
    block = 128;
  cudaStream_t s = (cudaStream_t)stream;
  host::BatchPlanSlot slot;
  if (!host::batch_plan_take(sizeof(BatchPlan), s, slot))
    return VJ_ERR_NOMEM;
  BatchArgs<T> a;
  a.count = count;
  a.m = m; a.n = n; a.offG = offG; a.offV = offV; a.offS = offS; a.order = order;
  a.G = G; a.V = V; a.eS = eS; a.fS = fS; a.info = info;
  a.plan = reinterpret_cast<BatchPlan *>(slot.ptr);
  a.strategy = (int)strategy;
  a.swp = swp;
  a.sms = host::sm_count();
  const vj_fint r = batch_launch<T>(a, block, (occ < 2 || occ > 6) ? 0 : occ, s);
  return (!host::batch_plan_done(slot, s) && !r) ? VJ_ERR_CUDA : r;
}

}  // namespace vj

extern "C" {

vj_fint vj_dvjsvd_batch_dev(vj_fint count, const long long *m, const long long *n, double *G, const long long *offG,
                            double *V, const long long *offV, double *eS, double *fS, const long long *offS,
                            const int *order, long strategy, unsigned swp, long long *info, int block, void *stream)
{
  return vj::batch_dev<double>(count, m, n, G, offG, V, offV, eS, fS, offS, order, strategy, swp, info, block, 0,
                               stream);
}

vj_fint vj_svjsvd_batch_dev(vj_fint count, const long long *m, const long long *n, float *G, const long long *offG,
                            float *V, const long long *offV, float *eS, float *fS, const long long *offS,
                            const int *order, long strategy, unsigned swp, long long *info, int block, void *stream)
{
  return vj::batch_dev<float>(count, m, n, G, offG, V, offV, eS, fS, offS, order, strategy, swp, info, block, 0,
                              stream);
}

vj_fint vj_dvjsvd_batch_tuned_dev(vj_fint count, const long long *m, const long long *n, double *G,
                                  const long long *offG, double *V, const long long *offV, double *eS, double *fS,
                                  const long long *offS, const int *order, long strategy, unsigned swp,
                                  long long *info, int block, int occupancy, void *stream)
{
  return vj::batch_dev<double>(count, m, n, G, offG, V, offV, eS, fS, offS, order, strategy, swp, info, block,
                               occupancy, stream);
}

vj_fint vj_svjsvd_batch_tuned_dev(vj_fint count, const long long *m, const long long *n, float *G,
                                  const long long *offG, float *V, const long long *offV, float *eS, float *fS,
                                  const long long *offS, const int *order, long strategy, unsigned swp,
                                  long long *info, int block, int occupancy, void *stream)
{
  return vj::batch_dev<float>(count, m, n, G, offG, V, offV, eS, fS, offS, order, strategy, swp, info, block,
                              occupancy, stream);
}

}  // extern "C"
