// FP64 products on the tensor cores, to FP64 accuracy.
//
// GB300 issues an FP64 FMA for half a lane per clock and SM sub-partition
// (1.2 TFLOP/s for the GPU, 1/1500 of its 16-bit tensor rate), so the FP64
// contractions of the sweeps run as exact integer products instead (the
// error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59,
// 2012).  Each operand is cut along the inner dimension into groups that
// share one power-of-two scale -- a row of A, a column of B -- and each value
// becomes a 55-bit signed integer, rounded to nearest at 2^-54 of the group's
// power-of-two bound, written as seven signed base-256 digits of magnitude at
// most 128 (exact in FP16).  The products of digits s of A and t of B with
// s + t = d accumulate in one FP32 tensor-memory accumulator per diagonal d,
// exactly: at most 7 pairs x 128 terms of at most 2^14 each stay below 2^24.
// Diagonals 0 .. 7 are kept (34 of the 49 pairs); what is dropped starts at
// 2^-59 of (largest |a|) x (largest |b|) per product, below the rounding of
// the operands.  The eight sums are combined in 64-bit integers and rounded
// to FP64.
//
// Why seven digits and eight diagonals: with the 28 pairs of diagonals 0 .. 6
// the dropped digits (2^-52 of the largest product) would make sums of 32
// products less accurate than FP64 FMAs; with 34 they are more accurate, since
// a chain of FMAs rounds at every step.  Relative errors (2-norm) of C - A B
// against quadruple precision, 32 terms of N(0,1): 1.1e-16, FMA chain 2.0e-16;
// uniform [0,1): 6.8e-17 against 1.6e-16.
//
// Bound.  What holds is relative to the groups, not to each product: with alpha the
// largest |A(i, .)| of a row and beta the largest |B(., j)| of a column, both balanced
// (below), and K inner values, |C - A B|(i, j) <= 1.5 K 2^-53 alpha beta + 2^-53 |C|(i, j).
// An operand at 2^-k of its group's bound keeps 55 - k bits.  An FP64 FMA chain is bound
// by K 2^-53 sum |a| |b| instead: the same where the values of a row, a column or a group
// of rows are within a few powers of two once balanced, as bases and right-hand sides
// are, and smaller where a row's large values meet zeros or small ones.  The products
// of the factorisations are split so that no tile mixes rows of two kinds (f64_gj.cu).
//
// Balance.  Inner index k of A is divided by the power of two of the largest
// |A(., k)| of the tile and the same index of B multiplied by it (exponents
// only), so that a factor on inner index k of A with its inverse on B --
// unknowns or equations in other units, which FP64 FMAs do not notice --
// leaves the digits as they are.
//
// Non-finite operands: a group holding an infinity or NaN is marked.  The update and
// the reduction go over the results it enters again at a CTA's end and form them by
// FP64 FMAs (in the loops the calls would cost the update's epilogue 60 %).  The leaf
// application, whose operand is overwritten by then, gives NaN; solves refuse such
// right-hand sides.  Subnormal operands count as zero.
#pragma once
#include <cuda_fp16.h>

#include <cstdint>

#include "tcgen05.cuh"

namespace hodlr {

constexpr int kDig = 7;          // digits of an operand
constexpr int kDiag = 8;         // diagonals kept
constexpr int kDigN = 32;        // columns of a B tile and of each diagonal's accumulator
constexpr int kDigK = 32;        // K values per plane (one 64-byte swizzled row)
constexpr int kDigAPlane = 128 * kDigK * 2, kDigBPlane = kDigN * kDigK * 2;
constexpr int kDigABytes = kDig * kDigAPlane, kDigBBytes = kDig * kDigBPlane;
constexpr unsigned kDigAccCols = kDiag * kDigN;  // tensor-memory columns of one accumulator set

// ------------------------------------------------------------ operand side
// A value's exponent is e + c: e its biased exponent, c the balance of its
// inner index (negative for A's entries).  A group's key is the largest; its
// scale, what the epilogue adds up, is the key, with groups of zeros and
// non-finite groups marked.
constexpr int kDigZero = -(1 << 20), kDigBad = 1 << 20;

__device__ __forceinline__ unsigned dig_ahi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
// The same word for the balance: a non-finite entry is left out of it (its own
// row is marked, the other rows keep their digits).
__device__ __forceinline__ unsigned dig_finite(unsigned h) { return h >= 0x7ff00000u ? 0u : h; }
__device__ __forceinline__ void dig_key(int &key, unsigned h, int c) {  // h: high word of |x|
  if (h >= 0x00100000u) key = max(key, (int)(h >> 20) + c);
}
__device__ __forceinline__ int dig_scale(int key, unsigned ahi_max, int zero) {
  return ahi_max >= 0x7ff00000u ? kDigBad : key == kDigZero ? zero : key;
}
// The mark of a group, from memory: n values, `stride` apart.
__device__ __forceinline__ bool dig_marked(const double *x, long long stride, int n) {
  bool finite = true;
  for (int k = 0; k < n; ++k) finite = finite && dig_ahi(x[k * stride]) < 0x7ff00000u;
  return !finite;
}
constexpr int kDigZeroA = 0, kDigZeroB = 2046;  // scales of groups of zeros (any usual one: their sums are 0)

// |x| as an integer in units of 2^-54 of its group's bound, rounded to
// nearest, plus 128 in each of its seven low bytes: byte 6 - s of the result
// is digit s of |x| plus 128.  Byte 7 is 0x64, the high byte of dig_pair's FP16.
__device__ __forceinline__ unsigned long long dig_fix(double x, int c, int key) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7ffu);
  const unsigned long long m =
      ((unsigned long long)((hi & 0x000fffffu) | 0x00100000u) << 32 | (unsigned long long)lo) << 10;
  unsigned long long v;
  const unsigned sh = e ? (unsigned)(key - c - e + 8) : 64u;
  asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(sh));  // shifts past 63 give 0
  return (v + 0xc901010101010101ull) >> 1;  // (v + 1) / 2 + 0x6480808080808080
}

// The signs of two values as the factor and addend of dig_pair.
struct DigSign {
  __half2 f, a;
};
__device__ __forceinline__ DigSign dig_sign(double x, double y) {
  const unsigned s = __byte_perm((unsigned)__double2hiint(x), (unsigned)__double2hiint(y), 0x7030) & 0x80008000u;
  const unsigned f = s | 0x3c003c00u, a = s ^ 0xe480e480u;  // +-1, -+1152
  DigSign r;
  r.f = *reinterpret_cast<const __half2 *>(&f);
  r.a = *reinterpret_cast<const __half2 *>(&a);
  return r;
}

// Digit s of two values as a packed FP16 pair (the first in the low half):
// 0x6400 | byte is 1024 + 128 + digit of |x|, and the signed addend removes
// the offset: +-(1024 + byte) -+ 1152.
__device__ __forceinline__ unsigned dig_pair(unsigned long long a, unsigned long long b, const DigSign &sg, int s) {
  const int j = kDig - 1 - s;
  const unsigned q = (unsigned)(j & 3);
  const unsigned t =
      j >= 4 ? __byte_perm((unsigned)(a >> 32), (unsigned)(b >> 32), q | 0x30u | ((q + 4) << 8) | 0x7000u)
             : (__byte_perm((unsigned)a, (unsigned)b, q | (q << 4) | ((q + 4) << 8) | ((q + 4) << 12)) & 0x00ff00ffu) |
                   0x64006400u;
  const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&t), sg.f, sg.a);
  return *reinterpret_cast<const unsigned *>(&r);
}

// The seven planes of 8 consecutive K values of one row (16 bytes each);
// c(e): the balance of value e.
template <typename F>
__device__ __forceinline__ void dig_put8(unsigned char *p0, int plane_bytes, int off, const double *x, F c, int key) {
  unsigned long long u[8];
  DigSign g[4];
#pragma unroll
  for (int e = 0; e < 8; ++e) u[e] = dig_fix(x[e], c(e), key);
#pragma unroll
  for (int e = 0; e < 4; ++e) g[e] = dig_sign(x[2 * e], x[2 * e + 1]);
#pragma unroll
  for (int s = 0; s < kDig; ++s)
    *reinterpret_cast<uint4 *>(p0 + s * plane_bytes + off) =
        make_uint4(dig_pair(u[0], u[1], g[0], s), dig_pair(u[2], u[3], g[1], s), dig_pair(u[4], u[5], g[2], s),
                   dig_pair(u[6], u[7], g[3], s));
}
// The same for 4 consecutive K values (8 bytes each).
template <typename F>
__device__ __forceinline__ void dig_put4(unsigned char *p0, int plane_bytes, int off, const double *x, F c, int key) {
  unsigned long long u[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) u[e] = dig_fix(x[e], c(e), key);
  const DigSign g0 = dig_sign(x[0], x[1]), g1 = dig_sign(x[2], x[3]);
#pragma unroll
  for (int s = 0; s < kDig; ++s)
    *reinterpret_cast<uint2 *>(p0 + s * plane_bytes + off) =
        make_uint2(dig_pair(u[0], u[1], g0, s), dig_pair(u[2], u[3], g1, s));
}

// ---------------------------------------------------------------- products
// kind::f16 instruction descriptor, A and B FP16 (type 0), D FP32.
__host__ __device__ constexpr unsigned dig_idesc(int n) {
  return (1u << 4) | ((unsigned)(n >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
}
// Issues the products of one K-chunk (`ksteps` steps of 16) into the
// accumulator set at tensor-memory column `acc`: diagonal d at acc + 32 d.
// A's planes at `pa`, B's seven planes (contiguous, so that one product of
// digit s of A spans the digits of B) at `pb`.  `first`: the set is written,
// not added to.
__device__ __forceinline__ void dig_mma_chunk(unsigned acc, unsigned pa, unsigned pb, int ksteps, bool first) {
  const uint64_t ad = desc_sw64(pa), bd = desc_sw64(pb);
  for (int kk = 0; kk < ksteps; ++kk) {
    const unsigned add = (!first || kk > 0) ? 1u : 0u;
    const uint64_t a = ad + 2 * kk, b = bd + 2 * kk;
    tc_mma(acc, a, b, dig_idesc(kDigN * kDig), add);  // digit 0: diagonals 0 .. 6
    // digit 1: diagonals 1 .. 6, and 7 apart (nothing wrote it yet on the first step)
    tc_mma(acc + kDigN, a + kDigAPlane / 16, b, dig_idesc(kDigN * (kDig - 1)), 1u);
    tc_mma(acc + kDigN * 7, a + kDigAPlane / 16, b + (kDig - 1) * kDigBPlane / 16, dig_idesc(kDigN), add);
#pragma unroll
    for (int s = 2; s < kDig; ++s)  // digit s: diagonals s .. 7
      tc_mma(acc + kDigN * s, a + s * kDigAPlane / 16, b, dig_idesc(kDigN * (kDiag - s)), 1u);
  }
}

// ------------------------------------------------------------- result side
// The exact integer of an accumulator below 2^22 in magnitude, plus 0x4b400000:
// the bits of its sum with 1.5 2^23 (one FP32 addition; conversions run at a
// quarter of that rate).  With 1.5 2^(23 + Q) the integer over 2^Q, rounded,
// plus 0x4b400000 + (Q << 23).
template <int Q> __device__ __forceinline__ unsigned dig_raw(unsigned v) {
  constexpr float magic = 12582912.f * (float)(1 << Q);
  return __float_as_uint(__uint_as_float(v) + magic);
}
__device__ __forceinline__ int dig_cvt(unsigned v) { return __float2int_rn(__uint_as_float(v)); }

// The eight exact diagonal sums of an output as an integer in units of 2^-55
// of the bound of |a| |b|, rounded at that unit, for groups of at most KM
// terms (32, 64 or 128).  Diagonal d is at most KM d 2^14 (a leading digit is
// at most 64, the others 128), which tells where dig_raw<0> is exact.
template <int KM, int W>
__device__ __forceinline__ long long dig_combine(const unsigned (&v)[kDiag][W], int c) {
  // f: the bits of dig_raw, the integer plus kRaw; pairs f_d + 256 f_(d-1) lose their
  // offset in one subtraction (mod 2^32: the pairs' true values fit 32 bits)
  constexpr unsigned kRaw = 0x4b400000u, kPair = kRaw + (kRaw << 8);
  constexpr int Q = KM <= 32 ? 0 : KM <= 64 ? 1 : 2;  // diagonals 6 and 7 only round into the unit
  const unsigned f0 = dig_raw<0>(v[0][c]), f1 = dig_raw<0>(v[1][c]), f2 = dig_raw<0>(v[2][c]);
  const int hi = (int)(f1 + (f0 << 8) - kPair);
  const int low =
      ((int)(dig_raw<Q>(v[6][c]) - (kRaw + (Q << 23)) + (16 >> Q)) + (((int)(dig_raw<Q>(v[7][c]) - (kRaw + (Q << 23)))) >> 8)) >>
      (5 - Q);
  long long acc;
  if (KM <= 64) {
    const int mid = (int)(dig_raw<0>(v[3][c]) + (f2 << 8) - kPair);
    const int p5 = KM <= 32 ? (int)(dig_raw<0>(v[5][c]) + (dig_raw<0>(v[4][c]) << 8) - kPair)
                            : dig_cvt(v[5][c]) + (int)((dig_raw<0>(v[4][c]) - kRaw) << 8);
    acc = (long long)p5 * 8 + low;
    acc += (long long)mid * (1 << 19);
  } else {
    const int mid = dig_cvt(v[3][c]) + (int)((f2 - kRaw) << 8);
    acc = (long long)dig_cvt(v[4][c]) * 2048 + (low + (dig_cvt(v[5][c]) << 3));
    acc += (long long)mid * (1 << 19);
  }
  return acc + (long long)((unsigned long long)(unsigned)(hi << 3) << 32);
}

// v 2^(t - 2099) rounded to FP64, t the sum of the two groups' scales: packed
// on the integer pipes (the FP64 pipe's conversion takes three times as long
// as its additions; with it the low-rank update took 7800 clocks a tile
// instead of 5000).  Out of line: results outside the normal range, and marked
// groups.
template <bool NAN_IF_MARKED = true> static __device__ __noinline__ double dig_value_any(long long v, int t) {
  if (t >= kDigBad / 2) return NAN_IF_MARKED ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
  return scalbn((double)v, t - 2099);
}
// `odd` is set when the result has to come from dig_value_any instead.
__device__ __forceinline__ double dig_value(long long v, int t, bool &odd) {
  const unsigned s = (unsigned)(v >> 32) & 0x80000000u;
  const unsigned long long mag = (unsigned long long)(v < 0 ? -v : v) | (v == 0);  // 0 becomes 1: undone below
  const int lz = __clzll((long long)mag);
  // mag << (lz - 1) has its top bit at 62; rounded to 53 bits (a carry moves into the exponent)
  const unsigned long long r = ((mag << (lz - 1)) + 0x200ull) >> 10;
  const int be = t - 1014 - lz;  // biased exponent, less one: r carries the leading bit
  odd |= (unsigned)(be - 1) > 2040u;
  const unsigned hi = (unsigned)(r >> 32) + ((unsigned)be << 20);
  return __hiloint2double(v == 0 ? 0 : (int)(hi | s), (int)(unsigned)r);  // r's low word is 0 for v = 0
}


// The other way, on the FP64 pipe: v rounded to FP64 by two additions -- its halves
// as the low words of 2^84 and 2^52, the first subtraction exact, the second
// rounding --, to be scaled in the FMA that adds it to its sum.  A dozen integer
// instructions less, and two FP64 issues of 64 clocks; dig_power is 2^(t - 2099).
__device__ __forceinline__ double dig_double(long long v) {
  const double a = __hiloint2double(0x45300000, (int)((unsigned)(v >> 32) ^ 0x80000000u));
  const double b = __hiloint2double(0x43300000, (int)(unsigned)v);
  return (a - __hiloint2double(0x45300000, (int)0x80100000u)) + b;  // 2^84 + 2^63 + 2^52
}
__device__ __forceinline__ double dig_power(int t, bool &odd) {
  const int e = t - 1076;
  odd |= (unsigned)(e - 1) > 2045u;
  return __hiloint2double(e << 20, 0);
}

}  // namespace hodlr
