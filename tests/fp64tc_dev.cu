// Device harness for the digit products (vecjac_gb300/csrc/fp64tc.cu): X^H Y of random complex or real
// matrices with nd digits against long double sums, as columns by columns (scaled, or in the
// columns' units, its lower tiles only) and as rows by columns added to what is there.
//   fp64tc_dev KIND ND M N1 N2 SEED -> per product: largest error in units of the stated bound, and
//   whether entries that are no part of the result were left alone
// The bound per real sum: K (nd + 1) 2^(14 - 8 (nd + 2)) 201/200 (nd = 8: K OMITTED8) of the rows'
// powers of two, and four roundings of the result.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "../vecjac_gb300/csrc/fp64tc.cu"
#include "../vecjac_gb300/csrc/gram_bound.cuh"
#include "../vecjac_gb300/csrc/host.cu"

using namespace vj;
typedef long double ld;

static bool ok(cudaError_t e)
{
  if (e != cudaSuccess)
    std::printf("cuda: %s\n", cudaGetErrorString(e));
  return e == cudaSuccess;
}
template <typename T> static T *dev(const std::vector<T> &h)
{
  T *p = nullptr;
  if (!ok(cudaMalloc(&p, h.size() * sizeof(T))) ||
      !ok(cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice)))
    std::exit(2);
  return p;
}

struct Matrix {  // column-major planes with a leading dimension of their own
  int m, n, ldm;
  std::vector<double> re, im;
  Matrix(int m_, int n_, int pad) : m(m_), n(n_), ldm(m_ + pad), re((size_t)ldm * n_), im((size_t)ldm * n_) {}
};

static int power(double mx)  // the row's power of two: entries below 1/2 of it
{
  return mx > 0 ? std::ilogb(mx) + 2 : 0;
}

int main(int argc, char **argv)
{
  if (argc != 7)
    return 1;
  const bool cplx = argv[1][0] == 'z';
  const int nd = std::atoi(argv[2]), K = std::atoi(argv[3]), n1 = std::atoi(argv[4]), n2 = std::atoi(argv[5]);
  std::mt19937_64 rng((unsigned long long)std::atoi(argv[6]));
  std::normal_distribution<double> nrm;
  std::uniform_real_distribution<double> uni(-20.0, 20.0);
  auto fill = [&](Matrix &X) {
    for (int j = 0; j < X.n; ++j) {
      const double c = std::exp2(std::floor(uni(rng)));
      for (int i = 0; i < X.m; ++i) {
        // (graded entries: low digits without high ones)
        const double g = (i % 3 == 0) ? std::exp2(uni(rng) / 2 - 10.0) : 1.0;
        X.re[(size_t)j * X.ldm + i] = c * g * nrm(rng);
        X.im[(size_t)j * X.ldm + i] = cplx ? c * g * nrm(rng) : 0.0;
      }
    }
  };
  const int P = cplx ? 2 : 1;
  const ld one = nd == 8 ? (ld)oz::OMITTED8 : (ld)(nd + 1) * std::ldexp((ld)1.005, 14 - 8 * (nd + 2));
  unsigned *err = dev(std::vector<unsigned>(1, 0u));
  unsigned char *part = nullptr;
  if (!ok(cudaMalloc(&part, oz::part_bytes())))
    return 2;
  auto operand = [&](const oz::Source &s) {
    oz::Operand o = oz::shape(s, cplx);
    if (!ok(cudaMalloc(&o.d, (size_t)o.bytes())) || !ok(cudaMalloc(&o.e, (size_t)2 * o.np * 4)) ||
        !ok(oz::split(s, o, nullptr)))
      std::exit(2);
    return o;
  };
  // mode 0: X^H Y scaled; 1: X^H X in the columns' units, lower tiles; 2: C + Z Y (Z: n1 x K)
  for (int mode = 0; mode < 3; ++mode) {
    Matrix X(mode == 2 ? n1 : K, mode == 2 ? K : n1, 3), Y(K, n2, 5);
    fill(X);
    fill(Y);
    if (mode == 1)
      Y = X;
    const int nc = mode == 1 ? n1 : n2, ldc = n1 + 2;
    std::vector<double> C0((size_t)ldc * nc * 2);
    for (double &c : C0)
      c = nrm(rng) * 1e-3;
    const double *Xr = dev(X.re), *Xi = cplx ? dev(X.im) : nullptr, *Yr = dev(Y.re), *Yi = cplx ? dev(Y.im) : nullptr;
    double *C = dev(C0);
    oz::Operand A, B;
    if (mode == 2) {
      A = operand(oz::Source{Xr, Xi, X.ldm, X.ldm, n1, K, nullptr, 0, oz::ROWS});
      B = operand(oz::Source{Yr, Yi, Y.ldm, Y.ldm, n2, K, nullptr, 0, oz::PROD});
    }
    else {
      A = operand(oz::Source{Xr, Xi, X.ldm, X.ldm, n1, K, nullptr, 0, oz::COLS});
      A.halves = 1;
      B = operand(oz::Source{Yr, Yi, Y.ldm, Y.ldm, nc, K, nullptr, 0, oz::COLS});
    }
    const oz::Result R{C, C + (size_t)ldc * nc, ldc, ldc, n1, nc, nullptr, mode != 1, mode == 2, mode == 1};
    std::vector<double> H(C0.size());
    unsigned he = 1;
    if (!ok(oz::gemm(A, B, R, nd, err, part, nullptr)) || !ok(cudaDeviceSynchronize()) ||
        !ok(cudaMemcpy(H.data(), C, H.size() * 8, cudaMemcpyDeviceToHost)) ||
        !ok(cudaMemcpy(&he, err, 4, cudaMemcpyDeviceToHost)) || he)
      return 2;
    // the exponents of X's (Z's) and Y's rows as operands
    std::vector<int> ea((size_t)n1), eb((size_t)nc);
    for (int i = 0; i < n1; ++i) {
      double mx = 0;
      for (int k = 0; k < K; ++k) {
        const size_t o = mode == 2 ? (size_t)k * X.ldm + i : (size_t)i * X.ldm + k;
        mx = std::max(mx, std::max(std::fabs(X.re[o]), std::fabs(X.im[o])));
      }
      ea[(size_t)i] = power(mx);
    }
    for (int j = 0; j < nc; ++j) {
      double mx = 0;
      for (int k = 0; k < K; ++k) {
        const size_t o = (size_t)j * Y.ldm + k;
        mx = std::max(mx, std::max(std::fabs(Y.re[o]), std::fabs(Y.im[o])));
      }
      eb[(size_t)j] = power(mx);
    }
    ld worst = 0;
    bool kept = true;
    for (int j = 0; j < nc; ++j)
      for (int i = 0; i < ldc; ++i)
        for (int h = 0; h < 2; ++h) {
          const size_t at = (size_t)h * ldc * nc + (size_t)j * ldc + i;
          if (i >= n1 || (h && !cplx)) {
            kept = kept && H[at] == C0[at];
            continue;
          }
          if (mode == 1 && i < j)
            continue;  // (above the diagonal: some tiles are formed, some not)
          ld s = 0;
          for (int k = 0; k < K; ++k) {
            const size_t x = mode == 2 ? (size_t)k * X.ldm + i : (size_t)i * X.ldm + k, y = (size_t)j * Y.ldm + k;
            const ld xr = X.re[x], xi = mode == 2 ? X.im[x] : -X.im[x], yr = Y.re[y], yi = Y.im[y];
            s += h ? xr * yi + xi * yr : xr * yr - xi * yi;
          }
          const int e = mode == 1 ? 0 : ea[(size_t)i] + eb[(size_t)j];
          if (mode == 1)
            s = std::ldexp(s, -(ea[(size_t)i] + eb[(size_t)j]));
          const ld want = (mode == 2 ? (ld)C0[at] : 0) + s;
          const ld lim = std::ldexp((ld)P * K * one, e) + (std::fabs(s) + std::fabs(want)) * std::ldexp((ld)1, -51);
          worst = std::max(worst, std::fabs((ld)H[at] - want) / lim);
        }
    std::printf("%d %.6Lf %d\n", mode, worst, kept ? 1 : 0);
  }
  return 0;
}
