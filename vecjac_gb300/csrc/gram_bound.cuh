// What a Gram matrix from digit products (fp64tc.cu) says about the cosines of the columns: the
// error of its entries and the bound that the mixed SVD's certificate is made of (mixed.cu). Apart,
// so that a host harness can compile it.
#pragma once

namespace vj {
namespace oz {

// What the products with 8 digits of each factor leave out of a real sum, per element of K and in
// units of the two rows' powers of two (which bound each element by 1/2): the digit pairs of weight
// 8, seven of at most 2^14 2^-80, those of weight 9 and above, below a 200th of that, and the two
// roundings to 64 bits, half of 2^-65 each: 9.05 2^-66 = 1.2265e-19.
constexpr double OMITTED8 = 1.25e-19;

// An upper bound of |h_ij| / sqrt(h_ii h_jj) from computed entries: a = |h_ij|, ri and rj the
// reciprocal roots of h_ii and h_jj. Each real sum among them is within hb of its own; h_ij of
// complex columns is two of them, each hb away at most: sqrt(2) hb. The diagonal entries may be hb
// too large, and 1 / sqrt(1 - d) <= 1 + d up to d = 1/2 (no bound beyond). The factors 1 + 1e-14
// take the relative roundings of the entries and of this formula, some twenty units. (The four
// products that a pair costs beyond its cosine are not seen in a refinement's time.)
#ifdef __CUDACC__
__host__ __device__
#endif
inline double cosine_bound(double a, double ri, double rj, double hb, bool cplx)
{
  const double di = hb * ri * ri, dj = hb * rj * rj, r = 1.0 + 1e-14;
  if (!(di <= 0.5 && dj <= 0.5))
    return 2.0;
  return (a * r + (cplx ? 1.4142135623730952 : 1.0) * hb) * (ri * rj) * ((1.0 + di) * (1.0 + dj)) * r;
}

}  // namespace oz
}  // namespace vj
