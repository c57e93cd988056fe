// FP64-accurate residual products on the tensor cores by exact slicing
// (the Ozaki scheme; Ozaki, Ogita, Oishi, Rump, "Error-free transformations
// of matrix multiplication by using fast routines of matrix
// multiplication", Numer. Algorithms 59, 2012).
//
// Every FP64 operand is scaled by a power of two per group (a row of U or of
// a leaf block D; 64-row chunks of a column of V, X; a column of the small
// coupling blocks T') and cut into kOzSlices signed 7-bit digits
//     a = 2^E * sum_s d_s 2^(-7(s+1)),   |d_s| <= 127,
// each exactly representable in bf16.  A product of two digits is an integer
// below 2^14, so a bf16 MMA with FP32 accumulation sums up to 1024 of them
// (7 digit pairs x up to 128 terms here) exactly; the pairs of one diagonal
// s + t = d share an accumulator and the seven diagonals are combined in
// double-word (FP32 pair) arithmetic with their exact power-of-two weights.
// The truncation (diagonals d >= 7 and the digits' remainder) is below
// 2^-48 of the row's largest |a| times the column's largest |x| per term --
// the accuracy of the double-word arithmetic it replaces -- at an eighth of
// its FP32-pipe cost (mma.sync bf16 runs at ~8x the FFMA rate here).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace hodlr {

constexpr int kOzSlices = 7;   // digits per operand (49 bits)
constexpr int kOzChunk = 64;   // rows per exponent group of the column-scaled operands

#ifdef __CUDACC__
// ------------------------------------------------------------------ digits
// All on the integer pipes (GB300 issues FP64 at 1/58 of the FP32 rate):
// magnitudes compare as their bit patterns, and a value's 49-bit fixed-point
// image F = trunc(|a| 2^(49-E)) is its 53-bit significand shifted right by
// E - e + 3 (e its unbiased exponent); the digits are F's 7-bit groups.
__device__ __forceinline__ unsigned long long abs_bits(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}

// E with max|a| / 2^E in [0.5, 1) from the largest magnitude's bit pattern (0 for zero)
__device__ __forceinline__ int oz_exponent_bits(unsigned long long maxbits) {
  if (maxbits == 0) return 0;
  const int ef = (int)(maxbits >> 52);
  if (ef == 0) return -1010 - __clzll((long long)maxbits);  // subnormal: top bit p = 63 - clz, E = p - 1073
  return ef - 1022;
}

// F of a value and its sign (1: negative).
__device__ __forceinline__ unsigned long long oz_fixed(double v, int E, unsigned &neg) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
  const int ef = (int)((bits >> 52) & 0x7ff);
  const unsigned long long frac = bits & 0xfffffffffffffull;
  const unsigned long long M = ef ? (frac | (1ull << 52)) : frac;  // |v| = M 2^(e - 52)
  const int e = ef ? ef - 1023 : -1022;
  const int sh = E - e + 3;  // >= 4 for normal v; a subnormal group may need a left shift
  const unsigned long long F = (M == 0 || sh >= 64) ? 0ull : (sh >= 0 ? (M >> sh) : (M << -sh));
  neg = (unsigned)(bits >> 63);
  return F;
}

template <typename Store>
__device__ __forceinline__ void oz_digits(double v, int E, Store store) {
  unsigned neg;
  const unsigned long long F = oz_fixed(v, E, neg);
#pragma unroll
  for (int s = 0; s < kOzSlices; ++s) {
    const int d = (int)((F >> (42 - 7 * s)) & 127ull);
    store(s, __int2bfloat16_rn(neg ? -d : d));
  }
}

// The digits of eight values, d[s] the eight of slice s: two values at a time,
// 0x4300 | digit the bf16 128 + digit, and one packed multiply-add
// +-(128 + digit) -+ 128 (a conversion a digit runs at a quarter of that rate).
__device__ __forceinline__ void oz_digits8(const double (&v)[8], int E, uint4 (&d)[kOzSlices]) {
  unsigned long long F[8];
  unsigned neg[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) F[u] = oz_fixed(v[u], E, neg[u]);
  unsigned w[kOzSlices][4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const unsigned sg = neg[2 * p] << 15 | neg[2 * p + 1] << 31, f = 0x3f803f80u | sg, a = 0xc300c300u ^ sg;
#pragma unroll
    for (int s = 0; s < kOzSlices; ++s) {
      const unsigned t = (__byte_perm((unsigned)(F[2 * p] >> (42 - 7 * s)), (unsigned)(F[2 * p + 1] >> (42 - 7 * s)),
                                      0x5410) & 0x007f007fu) | 0x43004300u;
      const __nv_bfloat162 r = __hfma2(*reinterpret_cast<const __nv_bfloat162 *>(&t),
                                       *reinterpret_cast<const __nv_bfloat162 *>(&f),
                                       *reinterpret_cast<const __nv_bfloat162 *>(&a));
      w[s][p] = *reinterpret_cast<const unsigned *>(&r);
    }
  }
#pragma unroll
  for (int s = 0; s < kOzSlices; ++s) d[s] = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}
#endif

// Leaf size and rank the tensor-core residual supports (else the double-word one runs).
inline bool oz_supported(int m, int r) { return m % kOzChunk == 0 && m <= 256 && r >= 8 && r <= 64 && r % 8 == 0; }

// Row-scaled digits.  Row i's entries are A(i, q) = A[(i / rpb) * bstride +
// (i % rpb) * si + q * sq], q < cols; digit s of (i, q) goes to
// out[s * slice_stride + i * ld_out + q]; exps[i] = E_i.
cudaError_t launch_oz_slice_rows(const double *A, long long rpb, long long bstride, long long si, long long sq,
                                 long long rows, int cols, __nv_bfloat16 *out, long long ld_out,
                                 long long slice_stride, int *exps, cudaStream_t s);
// Column-scaled digits per 64-row chunk of an n x c column-major matrix
// (n a multiple of 64): digit s of (i, j) to out[s * slice_stride + j * ld_out
// + i]; exps[(i / 64) * c + j].  The sliced value is X (may be null: zero)
// plus the FP32 add (may be null); xout (may be null) receives it.
cudaError_t launch_oz_slice_cols(const double *X, long long ldx, long long n, int c, __nv_bfloat16 *out,
                                 long long ld_out, long long slice_stride, int *exps, const int *skip,
                                 cudaStream_t s, const float *add = nullptr, double *xout = nullptr);
// Digits of the coupling blocks T'_b = diag(scale) T_{b^1} (r x k blocks of
// T at T + b * r * k, ld r), scaled per column: digit s of (q, j) of block b
// to out[((b * kOzSlices + s) * k + j) * r + q]; exps[b * k + j].
cudaError_t launch_oz_slice_tprime(const double *T, const double *scale, int r, int k, int nb, __nv_bfloat16 *out,
                                   int *exps, const int *skip, cudaStream_t s);

// R2 = split(B) - D X on every leaf (m rows): D digits row-scaled (layout of
// launch_oz_slice_rows with ld_out = m, slice_stride = n m), X digits from
// launch_oz_slice_cols (ld n, slice stride n k).  R2 double-word, ld ldr.
cudaError_t launch_oz_leaf(const __nv_bfloat16 *Dsl, const int *Dexp, int m, int nleaf, const __nv_bfloat16 *Xsl,
                           const int *Xexp, long long n, int k, const double *B, long long ldb, float2 *R2,
                           long long ldr, const int *skip, cudaStream_t s);

// T_b = V_b^T X_b (r x k, FP64) for nb child blocks of `rows` rows from row 0.
// V digits column-scaled (column q of slice s at Vsl + s * vslice + q * n),
// exponents Vexp[(i / 64) * r + q].  Split over row chunks with a
// deterministic second pass.
size_t oz_reduce_workspace_doubles(long long rows, int nb, int r, int k);
cudaError_t launch_oz_reduce(const __nv_bfloat16 *Vsl, long long vslice, const int *Vexp, int r,
                             const __nv_bfloat16 *Xsl, const int *Xexp, long long n, int k, long long rows, int nb,
                             double *out, double *work, const int *skip, cudaStream_t s);

// R2_b -= U_b T'_b for nb child blocks of `rows` rows (U digits row-scaled:
// row i of slice s at Usl + s * uslice + i * r, exps Uexp[i]; T' digits from
// launch_oz_slice_tprime).
cudaError_t launch_oz_update(const __nv_bfloat16 *Usl, long long uslice, const int *Uexp, int r,
                             const __nv_bfloat16 *Tsl, const int *Texp, int k, long long rows, int nb, float2 *R2,
                             long long ldr, const int *skip, cudaStream_t s);

// The T' digits of every level in one launch, from every level's T blocks
// stored one level after another (level l at sum_{l' < l} nb(l') r k); out
// and exps laid out as the tcgen05 residual reads them (below).
constexpr int kOzMaxLevels = 32;
struct TprimeLevels {
  long long wpre[kOzMaxLevels + 1], toff[kOzMaxLevels], ooff[kOzMaxLevels], eoff[kOzMaxLevels];
  const double *scale[kOzMaxLevels];
  int L;
};
cudaError_t launch_oz_slice_tprime_all(const double *T, int r, int k, int L, const int *lev_nb,
                                       const double *const *scale, __nv_bfloat16 *out, int *exps, const int *skip,
                                       cudaStream_t s);

// R2 = split(B) - D X - sum_l U_l T'_l in one pass over 128-row tiles on
// the tcgen05 tensor cores (oz_tc.cu): leaf size 128 or 256, the T' digits
// of every level stored one level after another (level l's block b at line
// offset sum_{l' < l} 7 k nb(l') + 7 k b, exponents at sum_{l' < l} k nb(l')
// + k b); lev_nb / lev_rows: host arrays of the level geometry.
bool oz_tc_supported(int m, int r, int k);
cudaError_t launch_oz_tc_resid(const __nv_bfloat16 *Dsl, const int *Dexp, const __nv_bfloat16 *Xsl, const int *Xexp,
                               const __nv_bfloat16 *Usl, const int *Uexp, const __nv_bfloat16 *Tsl, const int *Texp,
                               long long n, int m, int L, int r, int k, const int *lev_nb, const long long *lev_rows,
                               const double *B, long long ldb, float2 *R2, long long ldr, const int *skip,
                               DevStatus *st, cudaStream_t s);

// T_l = V_l^T X for every level in one pass (oz_tc.cu): level l's blocks at
// T + sum_{l' < l} nb(l') r k (r x k each, ld r); P: partial sums of blocks
// longer than a reduction range, oz_tc_reduce_partials doubles.
size_t oz_tc_reduce_partials(long long n, int L, int r, int k, const int *lev_nb, const long long *lev_rows);
cudaError_t launch_oz_tc_reduce(const __nv_bfloat16 *Vsl, const int *Vexp, const __nv_bfloat16 *Xsl,
                                const int *Xexp, long long n, int L, int r, int k, const int *lev_nb,
                                const long long *lev_rows, double *T, double *P, const int *skip, DevStatus *st,
                                cudaStream_t s);

}  // namespace hodlr
