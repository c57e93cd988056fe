// K1 in FP64 for leaves of 64, 128 and 256 rows whose factorisation only needs
// the explicit inverse: blocked Gauss-Jordan with partial pivoting, 32 columns
// a block, the O(m^3) part on the tensor cores.
//
// For the pivot rows K and columns K of a block (D = A_KK after the block's row
// interchanges, L11 U11 = D its LU), every other row I and column J:
//     A_KJ <- D^-1 A_KJ      A_IJ <- A_IJ - (A_IK D^-1) A_KJ
//     A_KK <- D^-1           A_IK <- -A_IK D^-1
// The panel kernel (one CTA a leaf, one thread a row) factors the block's
// columns with the pivot rule of dgetf2 (first row of largest |a| among the
// rows not pivoted yet, reciprocal scaling), forms W = A_IK D^-1 as (A_IK
// U11^-1) L11^-1 -- for the rows below, the multipliers of the LU times L11^-1,
// so that no product is larger than elimination makes it -- interchanges the
// rows of the other columns, moves the pivot rows out into R and leaves zeros
// in their place; then one batched product A <- A - W R over all leaves
// (f64_update_tc.cu, W's pivot rows -D^-1) does both updates.  The LU factors
// and pivots of these leaves are formed on request from the blocks themselves
// (leaf_factor_reg_kernel / leaf_blocked.cu).
//
// A leaf with a pivot below 2^-40 of the largest entry of its row and of its
// column of D -- singular, or so close to it that the two ways of rounding
// would differ -- is factored again by FP64 FMAs in DGETRF's order
// (leaf_gj_again_kernel), which decides on a zero pivot and gives its inverse.
//
// What bounds it: the FP64 pipe, by the panels: (m + 32) (32^2 - 32) FMAs each,
// 0.6 M for leaf 128 of the 2.1 M of its Gauss-Jordan sweep in one piece.  32
// columns a block: at 16 the panels would take half as long, but each of twice
// as many products reads and writes the whole matrix.  Measured with the digit
// images: 8192 leaves of 128 rows 15.2 ms, 69.7 by the register-resident sweep
// (leaf_factor_reg_kernel, at 39 % of the FP64 rate); 16 leaves of 256 rows 1.35
// ms, 2.50 by blocked LU and triangular solves.
#include <algorithm>

#include "dense_ops.cuh"
#include "kernels.cuh"

namespace hodlr {

bool f64_update_tc_try(const UpdateArgs &a, DevStatus *st, cudaStream_t s, cudaError_t &err);

namespace {
constexpr int kNb = 32;
}

// Rows [k0, k0 + 32) of block columns [k0, k0 + 32): see above.  A [leaf][m][m]
// is worked on in place; W [leaf][32][m] (column c at + c m), R [leaf][m][32]
// (column j at + 32 j), perm [leaf][m]: the original row at each position.
template <int M>
__global__ void __launch_bounds__(M + kNb) leaf_gj_panel_kernel(double *A, double *W, double *R, int *perm, int k0,
                                                                const unsigned *big, int *again) {
  constexpr int NT = M + kNb, NW = NT / 32;
  __shared__ double sU[2][kNb], sRcp[2], sL[kNb][kNb];
  __shared__ uint4 sBest[2][NW];  // |a| (high, low word), position, row of each warp's candidate
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long leaf = blockIdx.x;
  double *Al = A + leaf * M * M;
  const bool real = tid < M;  // the last warp's rows are those of the identity: they become D^-1
  int pos = tid;
  const int orig = real ? (k0 ? perm[leaf * M + tid] : tid) : 0;  // the row of D
  const unsigned *bl = big + leaf * 2 * M;                         // largest |D| of its rows, then its columns
  const unsigned brow = real ? bl[orig] : 0;
  bool open = real && tid >= k0;  // may still become a pivot row
  bool pivot_row = false;
  double a[kNb];
#pragma unroll
  for (int c = 0; c < kNb; ++c) a[c] = real ? Al[tid + (long long)(k0 + c) * M] : (c == lane ? 1.0 : 0.0);
#pragma unroll
  for (int c = 0; c < kNb; ++c) {
    const int buf = c & 1;
    // pivot: largest |a|, ties to the lowest position; NaN is never preferred
    unsigned hi = 0, lo = 0;
    if (open) {
      hi = (unsigned)__double2hiint(a[c]) & 0x7fffffffu;
      lo = (unsigned)__double2loint(a[c]);
      if (hi > 0x7ff00000u || (hi == 0x7ff00000u && lo)) hi = lo = 0;
    }
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    const unsigned mp = __reduce_min_sync(0xffffffffu, open && hi == mh && lo == ml ? (unsigned)pos : 0xffffu);
    if (mp == 0xffffu ? lane == 0 : (open && (unsigned)pos == mp)) sBest[buf][warp] = make_uint4(mh, ml, mp, tid);
    __syncthreads();
    uint4 b = sBest[buf][0];
#pragma unroll
    for (int w = 1; w < NW - 1; ++w) {
      const uint4 o = sBest[buf][w];
      const bool better = o.z != 0xffffu && (b.z == 0xffffu || o.x > b.x || (o.x == b.x && (o.y > b.y || (o.y == b.y && o.z < b.z))));
      if (better) b = o;
    }
    const int pp = (int)b.z, prow = (int)b.w;  // the pivot's position and row
    if (tid == prow) {
      const double pv = a[c];
      sRcp[buf] = pv != 0.0 ? 1.0 / pv : 0.0;
#pragma unroll
      for (int j = c; j < kNb; ++j) sU[buf][j] = a[j];
      pivot_row = true;
      open = false;
      // exponents: |pivot| against the smaller of its row's and column's largest
      const unsigned ph = (unsigned)__double2hiint(pv) & 0x7fffffffu;
      if (pv == 0.0 || ph + (40u << 20) < min(brow, bl[M + k0 + c])) again[leaf] = 1;
    } else if (real && pos == k0 + c) {
      pos = pp;
    }
    if (tid == prow) pos = k0 + c;
    __syncthreads();
    const double pv = sU[buf][c];
    if (!pivot_row) {  // pivot rows keep L11 and U11
      double l = a[c];
      if (pv != 0.0) l = dabs(pv) >= safe_min<double>() ? l * sRcp[buf] : l / pv;
      a[c] = l;
#pragma unroll
      for (int j = c + 1; j < kNb; ++j) a[j] -= l * sU[buf][j];
    }
  }
  if (pivot_row) {
#pragma unroll
    for (int c = 0; c < kNb; ++c) sL[pos - k0][c] = a[c];
  }
  __syncthreads();
  // times L11^-1 from the right
  if (!pivot_row)
#pragma unroll
    for (int t = kNb - 1; t > 0; --t)
#pragma unroll
      for (int c = 0; c < t; ++c) a[c] -= a[t] * sL[t][c];
  // W and the panel's new columns: the identity's rows are the pivot rows' D^-1
  double *Wl = W + leaf * M * kNb;
  const int row = real ? pos : k0 + lane;
  if (!pivot_row)
#pragma unroll
    for (int c = 0; c < kNb; ++c) {
      const double v = real ? a[c] : -a[c];
      Wl[row + (long long)c * M] = v;
      Al[row + (long long)(k0 + c) * M] = -v;
    }
  // the other columns: rows to their positions, the pivot rows into R
  double *Rl = R + leaf * M * kNb;
  const bool moves = real && (pos != tid || pivot_row);
  for (int j0 = 0; j0 < M; j0 += 8) {
    double x[8];
    if (moves)
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = Al[tid + (long long)(j0 + e) * M];
    __syncthreads();
    if (j0 >= k0 && j0 < k0 + kNb) {  // the panel itself: no update
      if (pivot_row)
#pragma unroll
        for (int e = 0; e < 8; ++e) Rl[(long long)(j0 + e) * kNb + pos - k0] = 0.0;
    } else if (moves) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        Al[pos + (long long)(j0 + e) * M] = pivot_row ? 0.0 : x[e];
        if (pivot_row) Rl[(long long)(j0 + e) * kNb + pos - k0] = x[e];
      }
    }
  }
  __syncthreads();
  if (real) perm[leaf * M + pos] = orig;
}

// A = D, the largest |D| of every row and column (high words), again = 0; the
// first non-finite leaf reported.
__global__ void __launch_bounds__(256) leaf_gj_copy_kernel(const double *__restrict__ D, long long d_ld,
                                                           long long d_stride, int m, double *A, unsigned *big,
                                                           int *again, DevStatus *st) {
  __shared__ unsigned srow[256], scol[256];
  const long long leaf = blockIdx.x;
  const double *Dl = D + leaf * d_stride;
  const int tid = threadIdx.x;
  srow[tid] = scol[tid] = 0;
  __syncthreads();
  unsigned mx = 0;
  for (int e = tid; e < m * m; e += 256) {  // m divides 256: the thread stays on row tid % m
    const double v = Dl[e % m + (long long)(e / m) * d_ld];
    const unsigned h = (unsigned)__double2hiint(v) & 0x7fffffffu;
    A[leaf * m * m + e] = v;
    mx = max(mx, h);
    const unsigned w = __reduce_max_sync(0xffffffffu, h);
    if ((tid & 31) == 0) atomicMax(&scol[e / m], w);
  }
  atomicMax(&srow[tid % m], mx);
  const int bad = __syncthreads_or(mx >= 0x7ff00000u);
  if (tid < m) {
    big[leaf * 2 * m + tid] = srow[tid];
    big[leaf * 2 * m + m + tid] = scol[tid];
  }
  if (tid == 0) {
    again[leaf] = 0;
    if (bad) report_error(st, HODLR_ERR_NONFINITE_INPUT, leaf * m);
  }
}

// The leaves marked `again`: LU by FP64 FMAs in the workspace A (DGETF2's
// order, a zero pivot reported), and Dinv from it, 8 columns at a time.
__global__ void __launch_bounds__(256) leaf_gj_again_kernel(const double *__restrict__ D, long long d_ld,
                                                            long long d_stride, int m, double *A, int *ipiv,
                                                            double *Dinv, const int *again, DevStatus *st) {
  const long long leaf = blockIdx.x;
  if (!again[leaf]) return;
  __shared__ double sX[256 * 8];
  __shared__ int spiv[256], s_info;
  const double *Dl = D + leaf * d_stride;
  double *Al = A + leaf * m * m, *O = Dinv + leaf * m * m;
  int bad = 0;
  for (int e = threadIdx.x; e < m * m; e += 256) {
    const double v = Dl[e % m + (long long)(e / m) * d_ld];
    bad |= !isfinite(v);
    Al[e] = v;
  }
  if (__syncthreads_or(bad)) return;  // reported by the copy
  block_getrf<double>(Al, m, m, ipiv + leaf * m, &s_info);
  __syncthreads();
  if (s_info && threadIdx.x == 0) report_error(st, HODLR_ERR_SINGULAR_LEAF, leaf);
  for (int i = threadIdx.x; i < m; i += 256) spiv[i] = ipiv[leaf * m + i];
  for (int c0 = 0; c0 < m; c0 += 8) {
    for (int e = threadIdx.x; e < m * 8; e += 256) sX[e] = e % m == c0 + e / m ? 1.0 : 0.0;
    __syncthreads();
    block_getrs<double, false>(Al, m, spiv, m, sX, m, 8);
    for (int e = threadIdx.x; e < m * 8; e += 256) O[(long long)c0 * m + e] = sX[e];
    __syncthreads();
  }
}

// Dinv's columns from the inverse of the interchanged rows.
__global__ void __launch_bounds__(256) leaf_gj_columns_kernel(const double *__restrict__ A, const int *__restrict__ perm,
                                                              int m, double *Dinv) {
  const long long leaf = blockIdx.x;
  const double *Al = A + leaf * m * m;
  double *O = Dinv + leaf * m * m;
  for (int e = threadIdx.x; e < m * m; e += 256) {
    const int i = e % m, p = e / m;
    O[i + (long long)perm[leaf * m + p] * m] = Al[e];
  }
}

// Bytes of scratch: W, R, perm, the largest entries and the marks.
size_t f64_leaf_gj_scratch(int m, int nleaf) {
  return (size_t)nleaf * (m * (2 * kNb * sizeof(double) + sizeof(int) + 2 * sizeof(unsigned)) + sizeof(int));
}

// Dinv = D^-1 for every leaf; A: an [nleaf][m][m] workspace, ipiv: [nleaf][m].
cudaError_t launch_f64_leaf_gj(const double *D, long long d_ld, long long d_stride, int m, int nleaf, double *A,
                               int *ipiv, double *Dinv, void *scratch, DevStatus *st, cudaStream_t s) {
  double *W = static_cast<double *>(scratch), *R = W + (size_t)nleaf * m * kNb;
  int *perm = reinterpret_cast<int *>(R + (size_t)nleaf * m * kNb);
  unsigned *big = reinterpret_cast<unsigned *>(perm + (size_t)nleaf * m);
  int *again = reinterpret_cast<int *>(big + (size_t)nleaf * 2 * m);
  HODLR_LAUNCH(leaf_gj_copy_kernel, nleaf, 256, 0, s, D, d_ld, d_stride, m, A, big, again, st);
  for (int k0 = 0; k0 < m; k0 += kNb) {
    if (m == 64) HODLR_LAUNCH(leaf_gj_panel_kernel<64>, nleaf, 64 + kNb, 0, s, A, W, R, perm, k0, big, again);
    else if (m == 128) HODLR_LAUNCH(leaf_gj_panel_kernel<128>, nleaf, 128 + kNb, 0, s, A, W, R, perm, k0, big, again);
    else if (m == 256) HODLR_LAUNCH(leaf_gj_panel_kernel<256>, nleaf, 256 + kNb, 0, s, A, W, R, perm, k0, big, again);
    else return cudaErrorInvalidValue;
    UpdateArgs ua{};
    ua.A = W;
    ua.lda = m;
    ua.a_bstride = (long long)m * kNb;
    ua.B = R;
    ua.ldb = kNb;
    ua.b_s1 = 2LL * m * kNb;
    ua.b_s2 = (long long)m * kNb;
    ua.C = A;
    ua.ldc = m;
    ua.c_bstride = (long long)m * m;
    ua.M = m;
    ua.N = m;
    ua.K = kNb;
    ua.nbatch = nleaf;
    ua.alpha = -1.0;
    cudaError_t e = cudaSuccess;
    if (!f64_update_tc_try(ua, st, s, e)) return cudaErrorInvalidValue;
    if (e != cudaSuccess) return e;
  }
  HODLR_LAUNCH(leaf_gj_columns_kernel, nleaf, 256, 0, s, A, perm, m, Dinv);
  HODLR_LAUNCH(leaf_gj_again_kernel, nleaf, 256, 0, s, D, d_ld, d_stride, m, A, ipiv, Dinv, again, st);
  return cudaGetLastError();
}

}  // namespace hodlr
