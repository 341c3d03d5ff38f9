// FP64 matrix products on the BF16 tensor cores by exact digit products.
//
// GB300's FP64 unit forms 0.3e12 products and sums per second and its DGEMM reaches 1.1
// TFLOP/s, against 1.9 PFLOP/s in BF16. Each row of an operand is scaled by a power of two to
// magnitudes below 1/2 and cut into signed base-256 digits, x = sum_s d_s 2^(-8 (s+1)), |d_s| <=
// 128, which BF16 holds exactly; the product is the sum over the digit pairs of the integer
// products sum_k a_s b_t 2^(-8 (s+t+2)) (K. Ozaki et al., "Error-free transformations of matrix
// multiplication by using fast routines of matrix multiplication and its applications", Numer.
// Algorithms 59, 2012; on tensor cores D. Mukunoki et al., ISC 2020). The pairs of one weight w =
// s + t < nd share an FP32 accumulator in TMEM: its integers stay below 2^24 for 128 elements
// of K (at most 8 pairs of products up to 2^14), so every sum is exact; then the accumulators
// are read out into 64-bit integers, which hold the sums of up to MAX_K elements of K exactly, and the two halves of the weights are joined and rounded once at the end. What is
// left out, the pairs of weight nd and above and the digits past the last, is below 2^-54.9 (nd = 7) or
// 2^-62.8 (nd = 8; OMITTED8 of gram_bound.cuh) of K times the two rows' scales (the powers of two by
// which they are divided, at most four times their largest entries).
//
// k_gemm: a CTA forms a 128 x 64 tile of C: eight accumulators of 64 columns fill the 512 columns
// of TMEM. Two operand stages of KB = 32 (up to 96 KiB each) come by bulk copies; one thread
// issues copies and MMAs; all eight warps read out. The operands' blocks come from L2 (84 KiB
// per 56 MMAs of 128 x 64 x 16 with nd = 7), which bounds it. Where the tiles are fewer than half of the
// SMs and K is long (the Gram matrix of a tall matrix: one tile up to n = 64), several CTAs take a
// stretch of K each and leave their integers, which k_gemm_sum adds up: still exact, so the same bits.
#include "fp64tc.cuh"

#include <algorithm>
#include <cstdint>

#include "tc.cuh"
#include "vj_host.h"

namespace vj {
namespace oz {

constexpr int THREADS = 256;
constexpr int LBO = 128;              // bytes between core matrices adjacent in K
constexpr int SBO = (KB / 8) * 128;   // bytes between groups of 8 rows
constexpr int APLANE = 2 * PLANE;     // a digit of the 128-row tile of A
constexpr int STAGE = DIGITS * (APLANE + PLANE);
constexpr size_t SMEM = 2 * (size_t)STAGE + 1024;
constexpr int GROUP = 128 / KB;       // K blocks per read-out
constexpr uint32_t IDESC = tc::idesc_bf16<128, ROWB>::value;
constexpr long long WAIT_CYCLES = 4000000000LL;  // ~2 s: a wait that long has failed
constexpr int NOEXP = -(1 << 30);     // "exponent" of zero

// exponent of a finite double (ilogb), NOEXP for zero; infinities and NaN count as large
__device__ __forceinline__ int expo(double x)
{
  const unsigned long long u = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
  if (!u)
    return NOEXP;
  const int be = (int)(u >> 52);
  return be ? be - 1023 : -1011 - __clzll((long long)u);
}

__device__ __forceinline__ double element(const Source &s, int h, int r, int p, int k)
{
  if (s.mode == ROWS)
    return p ? s.im[(long long)k * s.ldi + r] : s.re[(long long)k * s.ldr + r];
  const bool im = h != p;
  const double v = im ? s.im[(long long)r * s.ldi + k] : s.re[(long long)r * s.ldr + k];
  const bool neg = (s.mode == COLS) ? (h && p) : (!h && p);
  return neg ? -v : v;
}

__global__ void k_fill_int(int *x, int n, int v)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] = v;
}

// e: the power of two by which row r is scaled (magnitudes below 1/2) from its largest exponent, for
// every half of np rows
__device__ __forceinline__ void put_exponent(int *e, int r, int np, int halves, int m)
{
  const int v = (m == NOEXP) ? 0 : m + 2;
  for (int h = 0; h < halves; ++h)
    e[h * np + r] = v;
}

// the operand's row exponents. COLS, PROD: a warp per row
__global__ void __launch_bounds__(256) k_expo_cols(Source s, int *e, int np, int halves)
{
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= np)
    return;
  int m = NOEXP;
  for (int k = lane; k < s.len && r < s.rows; k += 32) {
    const int a = s.ek ? s.esign * s.ek[k] : 0;
    int x = expo(s.re[(long long)r * s.ldr + k]);
    m = max(m, x == NOEXP ? x : x + a);
    if (s.im) {
      x = expo(s.im[(long long)r * s.ldi + k]);
      m = max(m, x == NOEXP ? x : x + a);
    }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0)
    put_exponent(e, r, np, halves, m);
}
// ROWS: threads along the rows, blockIdx.y along K; several of them collect the largest exponents, for
// k_expo_final
__global__ void __launch_bounds__(256) k_expo_rows(Source s, int *e, int np)
{
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= s.rows) {
    if (gridDim.y == 1 && r < np)
      e[r] = 0;
    return;
  }
  int m = NOEXP;
#pragma unroll 8
  for (int k = blockIdx.y; k < s.len; k += gridDim.y) {
    const int a = s.ek ? s.esign * s.ek[k] : 0;
    int x = expo(s.re[(long long)k * s.ldr + r]);
    m = max(m, x == NOEXP ? x : x + a);
    if (s.im) {
      x = expo(s.im[(long long)k * s.ldi + r]);
      m = max(m, x == NOEXP ? x : x + a);
    }
  }
  if (gridDim.y == 1)
    put_exponent(e, r, np, 1, m);
  else
    atomicMax(e + r, m);
}
__global__ void k_expo_final(int *e, int rows, int np)
{
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < np; r += gridDim.x * blockDim.x)
    put_exponent(e, r, np, 1, (r < rows) ? e[r] : NOEXP);
}

// x 2^-64 2^... as a 64-bit integer: round(x 2^(64 - e)), |x| < 2^(e - 1)
__device__ __forceinline__ long long fixed64(double x, int e)
{
  const unsigned long long u = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
  if (!u)
    return 0;
  int be = (int)(u >> 52);
  unsigned long long m = u & 0xfffffffffffffull;
  if (be)
    m |= 1ull << 52;
  else
    be = 1;
  // x = m 2^(be - 1075)
  const int sh = be - 1075 + 64 - e;
  long long q;
  if (sh >= 0)
    q = (long long)(m << (sh & 63));
  else if (sh > -55)
    q = (long long)((m + (1ull << (-sh - 1))) >> -sh);
  else
    q = 0;
  return (x < 0) ? -q : q;
}

// the digits of one 64 x 32 block: a thread cuts eight consecutive K elements of a row, one 16-byte
// row of a core matrix per digit
__global__ void __launch_bounds__(256) k_digits(Source s, Operand o)
{
  const int tid = threadIdx.x;
  const int kb = blockIdx.x, rb = blockIdx.y;
  const int nkb1 = o.kp / KB, nrb1 = o.np / ROWB;
  const int p = kb / nkb1, h = rb / nrb1;
  // (threads along whichever index is contiguous in memory)
  const int rl = (s.mode == ROWS) ? (tid & 63) : (tid >> 2), g = (s.mode == ROWS) ? (tid >> 6) : (tid & 3);
  const int r = (rb - h * nrb1) * ROWB + rl, k0 = (kb - p * nkb1) * KB + g * 8;
  const int e = o.e[h * o.np + r];
  long long q[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = k0 + i;
    q[i] = 0;
    if (r < s.rows && k < s.len)
      q[i] = fixed64(element(s, h, r, p, k), e - ((s.ek != nullptr) ? s.esign * s.ek[k] : 0));
  }
  unsigned char *const base =
      o.d + ((long long)rb * (nkb1 * o.parts) + kb) * (DIGITS * PLANE) + (rl >> 3) * SBO + g * LBO + (rl & 7) * 16;
#pragma unroll
  for (int d = DIGITS - 1; d >= 0; --d) {
    unsigned w[4];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      unsigned b[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int v = (int)(signed char)(q[i + j] & 255);  // (the last digit: what is left, |.| <= 128)
        const int dv = d ? v : (int)q[i + j];
        q[i + j] = (q[i + j] - v) >> 8;
        b[j] = __float_as_uint((float)dv) >> 16;
      }
      w[i >> 1] = b[0] | (b[1] << 16);
    }
    *reinterpret_cast<uint4 *>(base + d * PLANE) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, unsigned bytes, unsigned long long *bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(tc::saddr(bar))
               : "memory");
}

// 2^n x for a normal or zero x and any n (exact while the result is normal)
__device__ __forceinline__ double scaled(double x, int n) { return scalbn(x, n); }

// entry (r, j) of C's half from its sums of weights 0-3 and 4-7
__device__ __forceinline__ void put_entry(const Operand &A, const Operand &B, const Result &C, int half, int r, int j,
                                          int er, long long hi, long long lo)
{
  double *const out = half ? C.im : C.re;
  const long long ld = half ? C.ldi : C.ldr;
  // (hi 2^32 + lo) 2^-72
  double v = fma((double)hi, 4294967296.0, (double)lo);
  v = scaled(v, -72 + (C.scaled ? er + B.e[half * B.np + j] + (C.ej ? C.ej[j] : 0) : 0));
  double *const to = out + (long long)j * ld + r;
  *to = C.add ? *to + v : v;
}

// column tiles per half of C
__host__ __device__ inline int col_tiles(const Result &C) { return (C.cols + ROWB - 1) / ROWB; }

// where the sums of slice blockIdx.z of tile (cb, rb) begin: 64 columns of 128 rows
__device__ __forceinline__ size_t part_tile(int cb, int rb)
{
  return (((size_t)blockIdx.z * gridDim.y + rb) * gridDim.x + cb) * (size_t)(128 * ROWB);
}

// ND: digits used, a template so that the issue of the MMAs is straight-line code with constant
// descriptor offsets (computed in loops, the issuing thread took three times the MMAs' own time)
template <int ND>
__global__ void __launch_bounds__(THREADS, 1) k_gemm(Operand A, Operand B, Result C, int nkb_all, longlong2 *part,
                                                       unsigned *err)
{
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *const smem = smem_raw + ((1024u - (tc::saddr(smem_raw) & 1023u)) & 1023u);
  __shared__ unsigned long long full[2], freed[2], ready;
  __shared__ uint32_t tslot;
  __shared__ int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cb = blockIdx.x, rb = blockIdx.y;  // 64 columns, 128 rows
  const int half = cb / col_tiles(C), j0 = (cb - half * col_tiles(C)) * ROWB;
  if (C.lower && rb * 128 + 127 < j0)
    return;
  if (tid == 0) {
    tc::mbar_init1(&full[0]);
    tc::mbar_init1(&full[1]);
    tc::mbar_init1(&freed[0]);
    tc::mbar_init1(&freed[1]);
    tc::mbar_init1(&ready);
    tc::mbar_init_fence();
    s_fail = 0;
  }
  __syncwarp();
  if (warp == 0)
    tc::tmem_alloc(&tslot, 512);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tslot;
  // this CTA's stretch of K
  const int per = (nkb_all + (int)gridDim.z - 1) / (int)gridDim.z, kb0 = (int)blockIdx.z * per,
            nkb = min(per, nkb_all - kb0);
  const long long blk = (long long)DIGITS * PLANE;  // bytes between K blocks
  const unsigned char *const a0 = A.d + ((long long)(2 * rb) * nkb_all + kb0) * blk,
                            *const a1 = a0 + (long long)nkb_all * blk,
                            *const b0 = B.d + ((long long)((half * B.np + j0) / ROWB) * nkb_all + kb0) * blk;
  auto load = [&](int kb) {
    const int st = kb & 1;
    const uint32_t s0 = tc::saddr(smem) + st * STAGE;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::saddr(&full[st])),
                 "r"((unsigned)(ND * 3 * PLANE))
                 : "memory");
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      bulk_load(s0 + d * APLANE, a0 + kb * blk + d * PLANE, PLANE, &full[st]);
      bulk_load(s0 + d * APLANE + PLANE, a1 + kb * blk + d * PLANE, PLANE, &full[st]);
    }
    bulk_load(s0 + DIGITS * APLANE, b0 + kb * blk, (unsigned)(ND * PLANE), &full[st]);
  };
  long long hi[32], lo[32];  // this thread's row, 32 columns: weights 0-3 and 4-7
#pragma unroll
  for (int c = 0; c < 32; ++c)
    hi[c] = lo[c] = 0;
  int loaded = 0;
  if (tid == 0) {
    load(0);
    loaded = 1;
    if (nkb > 1) {
      load(1);
      loaded = 2;
    }
  }
  bool ok = true;
  uint32_t phase = 0;  // of `ready` that the last group entered ends
  const int groups = (nkb + GROUP - 1) / GROUP;
  for (int g = 0; g < groups; ++g) {
    const int k1 = min(nkb, (g + 1) * GROUP);
    phase = (uint32_t)(g & 1);
    if (tid == 0) {
      for (int kb = g * GROUP; kb < k1 && ok; ++kb) {
        const int st = kb & 1;
        ok = tc::mbar_wait(&full[st], (uint32_t)((kb >> 1) & 1), WAIT_CYCLES);
        if (!ok)
          break;
        tc::fence_after();
        const uint32_t s0 = tc::saddr(smem) + st * STAGE;
        // (a descriptor's address field counts 16 bytes: offsets are added to it)
        const uint64_t da = tc::sdesc(s0, LBO, SBO), db = tc::sdesc(s0 + DIGITS * APLANE, LBO, SBO);
        const uint32_t more = (kb > g * GROUP) ? 1u : 0u;
#pragma unroll
        for (int kk = 0; kk < KB / 16; ++kk)
#pragma unroll
          for (int w = 0; w < ND; ++w)
#pragma unroll
            for (int s = 0; s <= w; ++s)
              tc::mma_bf16(tmem + w * ROWB, da + (uint64_t)((s * APLANE + kk * 2 * LBO) >> 4),
                           db + (uint64_t)(((w - s) * PLANE + kk * 2 * LBO) >> 4), IDESC, (kk > 0 || s > 0) ? 1u : more);
        tc::commit(&freed[st]);
        // the other stage's next block, once its MMAs are done
        if (kb >= 1 && kb + 1 < nkb) {
          ok = tc::mbar_wait(&freed[st ^ 1], (uint32_t)(((kb - 1) >> 1) & 1), WAIT_CYCLES);
          if (ok) {
            load(kb + 1);
            loaded = kb + 2;
          }
        }
      }
      if (!ok)
        s_fail = 1;
      tc::commit(&ready);
    }
    const bool w = tc::mbar_wait(&ready, phase, WAIT_CYCLES);
    if (__syncthreads_or(!w || (tid == 0 && s_fail))) {
      ok = false;
      break;
    }
    tc::fence_after();
    const uint32_t t0 = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * 32);
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      uint32_t v[32];
      tc::tmem_ld32(t0 + d * ROWB, v);
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const int x = __float2int_rn(__uint_as_float(v[c]));
        long long &to = (d < 4) ? hi[c] : lo[c];
        to += (long long)x * (1 << (8 * (3 - (d & 3))));
      }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
  }
  if (!ok) {
    // (nothing may be in flight when shared memory and TMEM are given back)
    if (tid == 0) {
      atomicOr(err, 1u);
      for (int kb = (loaded >= 2) ? loaded - 2 : 0; kb < loaded; ++kb)
        (void)tc::mbar_wait(&full[kb & 1], (uint32_t)((kb >> 1) & 1), WAIT_CYCLES);
    }
    (void)tc::mbar_wait(&ready, phase, WAIT_CYCLES);
  }
  else if (gridDim.z > 1) {
    longlong2 *const to = part + part_tile(blockIdx.x, blockIdx.y) + (warp >> 2) * 32 * 128 + (warp & 3) * 32 + lane;
#pragma unroll
    for (int c = 0; c < 32; ++c)
      to[c * 128] = make_longlong2(hi[c], lo[c]);
  }
  else {
    const int r = rb * 128 + (warp & 3) * 32 + lane;
    if (r < C.rows) {
      const int er = C.scaled ? A.e[r] : 0;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const int j = j0 + (warp >> 2) * 32 + c;
        if (j < C.cols)
          put_entry(A, B, C, half, r, j, er, hi[c], lo[c]);
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  __syncwarp();
  if (warp == 0)
    tc::tmem_dealloc(tmem, 512);
}

// C from the slices' sums: a CTA per tile, a thread per row and column
__global__ void __launch_bounds__(256) k_gemm_sum(Operand A, Operand B, Result C, int slices, const longlong2 *part)
{
  const int cb = blockIdx.x, rb = blockIdx.y;
  const int half = cb / col_tiles(C), j0 = (cb - half * col_tiles(C)) * ROWB;
  if (C.lower && rb * 128 + 127 < j0)
    return;
  const size_t slice = (size_t)gridDim.x * gridDim.y * (size_t)(128 * ROWB);
  for (int q = threadIdx.x; q < 128 * ROWB; q += 256) {
    const int r = rb * 128 + (q & 127), j = j0 + (q >> 7);
    if (r >= C.rows || j >= C.cols)
      continue;
    long long hi = 0, lo = 0;
    const longlong2 *p = part + part_tile(cb, rb) + q;
#pragma unroll 4
    for (int z = 0; z < slices; ++z, p += slice) {
      hi += p->x;
      lo += p->y;
    }
    put_entry(A, B, C, half, r, j, C.scaled ? A.e[r] : 0, hi, lo);
  }
}

Operand shape(const Source &s, bool cplx)
{
  Operand o;
  o.d = nullptr;
  o.e = nullptr;
  o.np = (int)pad(s.rows, 128);
  o.halves = (cplx && s.mode != ROWS) ? 2 : 1;
  o.kp = (int)pad(s.len, KB);
  o.parts = cplx ? 2 : 1;
  return o;
}

cudaError_t row_exponents(const Source &s, int *e, cudaStream_t st)
{
  k_expo_cols<<<(s.rows + 7) / 8, 256, 0, st>>>(s, e, s.rows, 1);
  return cudaGetLastError();
}

cudaError_t split_exponents(const Source &s, const Operand &o, cudaStream_t st)
{
  if (s.mode != ROWS)
    k_expo_cols<<<(o.np + 7) / 8, 256, 0, st>>>(s, o.e, o.np, o.halves);
  else if (s.len <= 32)  // (a thread goes along all of K: no largest exponents to collect)
    k_expo_rows<<<(o.np + 255) / 256, 256, 0, st>>>(s, o.e, o.np);
  else {
    k_fill_int<<<(s.rows + 255) / 256, 256, 0, st>>>(o.e, s.rows, NOEXP);
    k_expo_rows<<<dim3((unsigned)((s.rows + 255) / 256), 32u), 256, 0, st>>>(s, o.e, o.np);
    k_expo_final<<<(o.np + 255) / 256, 256, 0, st>>>(o.e, s.rows, o.np);
  }
  return cudaGetLastError();
}

cudaError_t split_digits(const Source &s, const Operand &o, cudaStream_t st)
{
  k_digits<<<dim3((unsigned)(o.kp / KB * o.parts), (unsigned)(o.np / ROWB * o.halves)), 256, 0, st>>>(s, o);
  return cudaGetLastError();
}

cudaError_t split(const Source &s, const Operand &o, cudaStream_t st)
{
  const cudaError_t e = split_exponents(s, o, st);
  return (e != cudaSuccess) ? e : split_digits(s, o, st);
}

// K blocks of a slice at least (1000 x 16 real 1.57 ms with 4, 1.68 with 16; 512 x 512 real 9.3 and 9.7)
constexpr long long MIN_SLICE = 4;

// (slices x tiles <= SMs)
size_t part_bytes() { return (size_t)host::sm_count() * 128 * ROWB * sizeof(longlong2); }

cudaError_t gemm(const Operand &A, const Operand &B, const Result &C, int nd, unsigned *err, unsigned char *part,
                 cudaStream_t st)
{
  void (*const k)(Operand, Operand, Result, int, longlong2 *, unsigned *) = (nd <= 3)   ? k_gemm<3>
                                                                           : (nd == 4) ? k_gemm<4>
                                                                           : (nd == 5) ? k_gemm<5>
                                                                           : (nd == 6) ? k_gemm<6>
                                                                           : (nd == 7) ? k_gemm<7>
                                                                                       : k_gemm<8>;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
  if (e != cudaSuccess)
    return e;
  const long long nkb = (long long)(A.kp / KB) * A.parts;
  if (nkb > MAX_K / KB)
    return cudaErrorInvalidValue;
  // (with lower, the tiles above the diagonal return at once)
  dim3 grid((unsigned)(col_tiles(C) * B.halves), (unsigned)((C.rows + 127) / 128));
  const long long tiles = (long long)grid.x * grid.y;
  long long slices = std::min((long long)host::sm_count() / tiles, nkb / MIN_SLICE);
  if (slices > 1)  // (none of them empty)
    slices = (nkb + (nkb + slices - 1) / slices - 1) / ((nkb + slices - 1) / slices);
  grid.z = (unsigned)std::max(slices, 1ll);
  longlong2 *const sums = reinterpret_cast<longlong2 *>(part);
  k<<<grid, THREADS, SMEM, st>>>(A, B, C, (int)nkb, sums, err);
  if (grid.z > 1)
    k_gemm_sum<<<dim3(grid.x, grid.y), 256, 0, st>>>(A, B, C, (int)grid.z, sums);
  return cudaGetLastError();
}

}  // namespace oz
}  // namespace vj
