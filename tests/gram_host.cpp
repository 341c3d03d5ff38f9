// Host harness for the bound of a cosine from a digit-product Gram matrix
// (vecjac_gb300/csrc/gram_bound.cuh). Reads lines "a hii hjj hb cplx" (hexadecimal doubles) and
// prints the bound of each; first the constant of the omitted products.
#include <cmath>
#include <cstdio>

#include "../vecjac_gb300/csrc/gram_bound.cuh"

int main()
{
  std::printf("%a\n", vj::oz::OMITTED8);
  double a, hi, hj, hb;
  int cplx;
  while (std::scanf("%la %la %la %la %d", &a, &hi, &hj, &hb, &cplx) == 5)
    std::printf("%a\n", vj::oz::cosine_bound(a, 1.0 / std::sqrt(hi), 1.0 / std::sqrt(hj), hb, cplx != 0));
  return 0;
}
