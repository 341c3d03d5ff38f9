// FP64 matrix products on the BF16 tensor cores (fp64tc.cu), for the mixed-precision SVD
// (mixed.cu): real and split-plane complex products as one real product of operands cut into
// digits.
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

namespace vj {
namespace oz {

constexpr int ROWB = 64;   // operand rows of a block
constexpr int KB = 32;     // K elements of a block
constexpr int DIGITS = 8;  // digits kept per element
constexpr int PLANE = ROWB * KB * 2;  // bytes of one digit of a block

inline long long pad(long long x, long long to) { return (x + to - 1) / to * to; }

// What an operand's element (row r of half h, part p of K, index k) is, from a planar complex
// matrix X (im null: real data, one half and one part):
//   COLS: X's columns against its rows k, for X^H Y:  h 0: re, im;  h 1: im, -re
//   ROWS: X's rows against its columns k, for X Y:    re, im
//   PROD: X's columns against its rows k, as Y of X Y: h 0: re, -im; h 1: im, re
// times 2^(esign * ek[k]) (ROWS, PROD; ek may be null).
enum { COLS = 0, ROWS = 1, PROD = 2 };
struct Source {
  const double *re, *im;
  long long ldr, ldi;
  int rows;       // operand rows per half
  int len;        // K elements per part
  const int *ek;
  int esign;
  int mode;
};

// Digits of an operand: rows per half padded to np, K per part to kp; block (row block, K block)
// holds DIGITS planes of ROWB x KB BF16 in the tensor core's K-major core-matrix order. e:
// the power of two of every row (per half the same).
struct Operand {
  unsigned char *d;
  int *e;
  int np, halves, kp, parts;
  long long bytes() const { return (long long)(np / ROWB) * halves * (kp / KB) * parts * DIGITS * PLANE; }
};

// the operand's shape for a source (d and e left null): np is a multiple of 128
Operand shape(const Source &s, bool cplx);
// exponents of the source's columns (COLS; 0 for a zero column), rows entries
cudaError_t row_exponents(const Source &s, int *e, cudaStream_t st);
// row exponents and digits of a source: both, or apart, where the digits are those of a part of the K
// over which the exponents were taken (e of o; its K does not matter to the exponents)
cudaError_t split(const Source &s, const Operand &o, cudaStream_t st);
cudaError_t split_exponents(const Source &s, const Operand &o, cudaStream_t st);
cudaError_t split_digits(const Source &s, const Operand &o, cudaStream_t st);
// most rows of operands of rows, and most elements of K over all parts, that the launches and the
// 64-bit sums take at once
constexpr long long MAX_ROWS = 1ll << 21, MAX_K = 1ll << 22;

// Where a product goes: column j of half 0 to re, of half 1 to im. Scaled: times the rows'
// powers of two and 2^ej[j] (ej may be null). add: added to what is there. lower: only the
// tiles that reach row >= column are formed.
struct Result {
  double *re, *im;
  long long ldr, ldi;
  int rows, cols;
  const int *ej;
  int scaled, add, lower;
};
// C (+)= A B^T over the operands' K (A one half, K up to MAX_K), with digits 0..nd-1 of each (3 <= nd <= 8); err is set
// nonzero when a wait inside the kernel gave up. part: part_bytes() of scratch for products whose K is
// split over CTAs (the same bits as unsplit).
size_t part_bytes();
cudaError_t gemm(const Operand &A, const Operand &B, const Result &C, int nd, unsigned *err, unsigned char *part,
                 cudaStream_t st);

}  // namespace oz
}  // namespace vj
