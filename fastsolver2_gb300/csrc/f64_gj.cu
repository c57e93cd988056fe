// K1 in FP64 for leaves of 64, 128 and 256 rows whose factorisation only needs
// the explicit inverse, and K4a in FP64, the capacitance systems' LU and
// inverse: elimination with partial pivoting, 32 columns a block, the O(m^3) part
// on the tensor cores.
//
// Up to 128 rows in one phase, Gauss-Jordan.  For the pivot rows K and columns K of a
// block (after the block's row interchanges A_KK = L11 U11), every other row I, W_I =
// A_IK U11^-1 (below the block the multipliers of the LU), W_K = -U11^-1, and all
// columns J, those of K begun anew as the identity's:
//     R_J = L11^-1 A_KJ      A_IJ <- A_IJ - W_I R_J      A_KJ <- -W_K R_J
// Leaves of 256 rows in two phases, the LU with L^-1 beside it (rows I below only, A_KJ
// <- R_J), then U^-1 times L^-1 from the last block up (R = U11^-1 Z_K, Z_I <- Z_I -
// U_IK R above).
//
// The panel kernel (one CTA a leaf, one thread a row) factors the block's
// columns with the pivot rule of dgetf2 (first row of largest |a| among the
// rows not pivoted yet, reciprocal scaling), interchanges the rows of the other
// columns, moves the pivot rows out into R and forms W and R; batched products over
// all leaves (f64_update_tc.cu) do the updates.  The LU factors and pivots of these
// leaves are formed on request from the blocks themselves (leaf_factor_reg_kernel /
// leaf_blocked.cu); those of a capacitance system (padded with the identity to 32, 64
// or 128 rows), and of leaves whose caller wants them in any case, are captured as they
// appear: L11, U11 and L21 in the panel, U12 = R right of the block, later interchanges
// applied to the columns of L already out.
//
// Backward error.  The sums are those of the sweeps before, entry by entry (reg_factor.cuh:
// Gauss-Jordan; leaf_blocked.cu: substitution on the identity), so that A x = b and
// A^T x = b keep their residuals.  Two orders that cost less do not: W_I L11^-1 in place
// of R makes the residual of A x = b grow with the condition (1e6: 60 times, 1e10 4000
// times, leaves of 64 rows), and one product for the rows above and in the block, whose
// W are as large as 1 / U11's pivots, and for those below, whose W are at most 1, that of
// A^T x = b: the digits of a row tile share the balance of an inner index.
//
// A leaf or system with a pivot below 2^-40 of the largest entry of its row and of its
// column of D -- singular, or so close to it that the two ways of rounding
// would differ -- is factored again by FP64 FMAs in DGETRF's order
// (leaf_gj_again_kernel, cap_factor_kernel), which decides on a zero pivot and
// gives its inverse.
//
// What bounds it: the FP64 pipe, by the panels: some (2 m + 32) 496 FMAs each in one
// phase, 0.57 M for leaf 128 of the 2.1 M of its Gauss-Jordan sweep in one piece.  32
// columns a block: at 16 the panels would take half as long, but each of twice
// as many products reads and writes the whole matrix.  Measured with the digit
// images: 8192 leaves of 128 rows 15.4 ms, 69.7 by the register-resident sweep
// (leaf_factor_reg_kernel, at 39 % of the FP64 rate); 16 leaves of 256 rows 1.34
// ms, 2.50 by blocked LU and triangular solves.  The capacitance systems of N =
// 2^20, rank 32 (8191 of 64 rows in 13 levels) with their applications to the transformed
// bases on the tensor cores 11.4 ms, 38 by the register-resident sweep
// (cap_factor_reg_kernel) and FMA applications; a lone system of 64 rows 190 us.
#include <algorithm>

#include "dense_ops.cuh"
#include "kernels.cuh"

namespace hodlr {

bool f64_update_tc_try(const UpdateArgs &a, DevStatus *st, cudaStream_t s, cudaError_t &err);
cudaError_t launch_cap_factor_marked(const CapFactorArgs &a, const int *only, cudaStream_t s);  // apply_kernels.cu

namespace {
constexpr int kNb = 32;
template <int M> constexpr bool kGjTwo = M == 256;  // see above

// Where a panel puts the LU factors (capacitance systems): n x n of the M x M
// padded system, DGETRF's layout, 1-based pivots.
struct LuOut {
  double *lu;
  int *ipiv, n;
};
}  // namespace

// Rows [k0, k0 + 32) of block columns [k0, k0 + 32): see above.  A [block][m][m]
// is worked on in place; W [block][32][m] (column c at + c m), R [block][m][32]
// (column j at + 32 j), perm [block][m]: the original row at each position.
//
// One thread a row, the panel's 32 columns in its registers; in one phase the
// identity's rows go along and become U11^-1.  An FP64 FMA holds its sub-partition's
// pipe for 64 clocks (and its result comes then), so a step is 64 clocks for
// each column left, plus some 900 for the pivot: one block barrier, every warp
// finding its best candidate for the next pivot as soon as that column is up to
// date, computing its reciprocal beside the other columns' FMAs, and leaving the
// whole row in shared memory, so that after the barrier every thread reads the
// winner's.  Then the threads take a column each of L11^-1 A_KJ.  A lone 64-row panel
// takes 66 us (74000 clocks the elimination, 32000 the columns); with two barriers, a
// division after the first and FP64 compares it took 87 to 108.
template <int M> __host__ __device__ constexpr int gj_threads() { return kGjTwo<M> ? M : M + kNb; }
template <int M, bool LU>
__global__ void __launch_bounds__(gj_threads<M>(), M == 128 ? (LU ? 3 : 4) : M == 64 ? 5 : 0)
gj_panel_kernel(double *A, double *W, double *R, int *perm, int k0, int nc, const unsigned *big, int *again, LuOut out) {
  constexpr bool kTwo = kGjTwo<M>, kOne = M == kNb;  // two phases; a single block
  constexpr int NW = M / 32;  // warps with rows of the block; the next has the identity's
  __shared__ double sU[2][NW][kNb], sRcp[2][NW], sL[kNb][kNb];
  __shared__ uint4 sBest[2][NW];  // |a| (high, low word), position, row of each warp's candidate
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long blk = blockIdx.x;
  double *Al = A + blk * M * M;
  const bool real = warp < NW, ident = warp == NW;
  int pos = tid;
  const int orig = real ? (k0 ? perm[blk * M + tid] : tid) : 0;  // the row of D
  const unsigned *bl = big + blk * 2 * M;                         // largest |D| of its rows, then its columns
  const unsigned brow = real ? bl[orig] : 0;
  // the identity's rows and columns that pad the block are their own pivots: no
  // steps for the panel's columns from nc on
  bool pivot_row = LU && real && tid >= k0 + nc && tid < k0 + kNb;
  bool open = real && tid >= k0 && !pivot_row;  // may still become a pivot row
  double a[kNb];
#pragma unroll
  for (int c = 0; c < kNb; ++c) a[c] = real ? Al[tid + (long long)(k0 + c) * M] : (c == lane ? 1.0 : 0.0);

  // the warp's candidate for column c: largest |a|, ties to the lowest
  // position, NaN never preferred; returns whether this lane holds it
  unsigned mh, ml, mp;
  auto candidate = [&](double v) {
    unsigned hi = 0, lo = 0;
    if (open) {
      hi = (unsigned)__double2hiint(v) & 0x7fffffffu;
      lo = (unsigned)__double2loint(v);
      if (hi > 0x7ff00000u || (hi == 0x7ff00000u && lo)) hi = lo = 0;
    }
    mh = __reduce_max_sync(0xffffffffu, hi);
    ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    mp = __reduce_min_sync(0xffffffffu, open && hi == mh && lo == ml ? (unsigned)pos : 0xffffu);
    return mp == 0xffffu ? lane == 0 : (open && (unsigned)pos == mp);
  };
  // the candidate's row, reciprocal and key into buffer b
#define HODLR_GJ_PUBLISH(c, b)                                                                    \
  if (real) {                                                                                     \
    if (cand) {                                                                                   \
      sBest[b][warp] = make_uint4(mh, ml, mp, tid);                                               \
      sRcp[b][warp] = rcp_usual(a[c]) ? rc : ((__double2hiint(a[c]) & 0x7fffffff) | __double2loint(a[c])) ? 1.0 / a[c] : 0.0; \
      _Pragma("unroll") for (int j = c; j < kNb; ++j) sU[b][warp][j] = a[j];                      \
    }                                                                                             \
  }
  bool cand = candidate(a[0]);
  double rc = newton_rcp(a[0]);
  HODLR_GJ_PUBLISH(0, 0)
  __syncthreads();
#pragma unroll
  for (int c = 0; c < kNb; ++c) {
    if (LU && c >= nc) continue;
    const int buf = c & 1;
    uint4 best = sBest[buf][0];
    int bw = 0;
#pragma unroll
    for (int w = 1; w < NW; ++w) {
      const uint4 o = sBest[buf][w];
      const bool better = o.z != 0xffffu && (best.z == 0xffffu || o.x > best.x ||
                                            (o.x == best.x && (o.y > best.y || (o.y == best.y && o.z < best.z))));
      if (better) {
        best = o;
        bw = w;
      }
    }
    const bool zero = (best.x | best.y) == 0;
    if (tid == (int)best.w) {
      pivot_row = true;
      open = false;
      pos = k0 + c;
      // exponents: |pivot| against the smaller of its row's and column's largest
      if (zero || best.x + (40u << 20) < min(brow, bl[M + k0 + c])) again[blk] = 1;
    } else if (real && pos == k0 + c) {
      pos = (int)best.z;
    }
    if (LU && tid == 0 && k0 + c < out.n) out.ipiv[blk * out.n + k0 + c] = (int)best.z + 1;
    const bool row = kTwo ? open : !pivot_row && (real || ident);  // pivot rows keep L11 and U11
    const double *u = sU[buf][bw];
    double l = 0.0;
    if (row) {
      l = a[c];
      if (!zero) l = best.x >= 0x00100000u ? l * sRcp[buf][bw] : l / u[c];
      a[c] = l;
      if (c + 1 < kNb) a[c + 1] -= l * u[c + 1];
    }
    if (c + 1 < (LU ? nc : kNb)) {
      cand = candidate(a[c + 1]);
      rc = newton_rcp(a[c + 1]);
      if (row) {
#pragma unroll
        for (int j = c + 2; j < kNb; ++j) a[j] -= l * u[j];
      }
      HODLR_GJ_PUBLISH(c + 1, buf ^ 1)
      __syncthreads();
    }
  }
#undef HODLR_GJ_PUBLISH
  if (pivot_row) {
#pragma unroll
    for (int c = 0; c < kNb; ++c) sL[pos - k0][c] = a[c];
  }
  double *lu = LU ? out.lu + blk * out.n * out.n : nullptr;
  if (LU && (pivot_row || open) && pos < out.n) {
#pragma unroll
    for (int c = 0; c < kNb; ++c)
      if (k0 + c < out.n) lu[pos + (long long)(k0 + c) * out.n] = a[c];
  }
  if (kOne) {  // D^-1 at once: the identity's rows times L11^-1 from the right
    __syncthreads();
    if (ident) {
#pragma unroll
      for (int t = kNb - 1; t > 0; --t) {
        if (t >= nc) continue;
#pragma unroll
        for (int c = 0; c < t; ++c) a[c] -= a[t] * sL[t][c];
      }
#pragma unroll
      for (int c = 0; c < kNb; ++c) Al[lane + (long long)c * M] = a[c];
    }
    if (real) perm[blk * M + pos] = orig;
    return;
  }
  // W: the multipliers of the rows, and -U11^-1 in one phase.  The block's own columns
  // begin anew, as those of the identity.
  double *Wl = W + blk * M * kNb;
  if (kTwo ? open : !pivot_row) {
    const int row = real ? pos : k0 + lane;
#pragma unroll
    for (int c = 0; c < kNb; ++c) Wl[row + (long long)c * M] = real ? a[c] : -a[c];
  }
  if (kTwo ? real && tid >= k0 + kNb : real) {
#pragma unroll
    for (int c = 0; c < kNb; ++c) Al[tid + (long long)(k0 + c) * M] = 0.0;
  }
  // the other columns: rows to their positions, the pivot rows into R, zeros in
  // their place; in the columns of L already out, the rows alone
  double *Rl = R + blk * M * kNb;
  const bool moves = real && (pos != tid || pivot_row);
  for (int j0 = 0; j0 < M; j0 += 8) {
    if (j0 >= k0 && j0 < k0 + kNb) continue;
    double x[8], y[8];
    const bool moves_l = LU && j0 < k0 && real && tid >= k0 && tid < out.n && pos != tid;
    if (moves)
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = Al[tid + (long long)(j0 + e) * M];
    if (moves_l)
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = lu[tid + (long long)(j0 + e) * out.n];
    __syncthreads();
    if (moves_l && pos < out.n)
#pragma unroll
      for (int e = 0; e < 8; ++e) lu[pos + (long long)(j0 + e) * out.n] = y[e];
    if (moves && !(kTwo && pivot_row))
#pragma unroll
      for (int e = 0; e < 8; ++e) Al[pos + (long long)(j0 + e) * M] = pivot_row ? 0.0 : x[e];
    if (pivot_row)
#pragma unroll
      for (int e = 0; e < 8; ++e) Rl[(long long)(j0 + e) * kNb + pos - k0] = x[e];
  }
  __syncthreads();
  if (!real) return;
  perm[blk * M + pos] = orig;
  // column tid of L11^-1 [A_KJ, I]; U12 and, in two phases, what the pivot rows hold from now on
  double *Rj = Rl + (long long)tid * kNb;
  const int jk = tid - k0;  // of the block's own columns, from 0 on
  const bool own = jk >= 0 && jk < kNb;
#pragma unroll
  for (int c = 0; c < kNb; ++c) a[c] = own ? (c == jk ? 1.0 : 0.0) : Rj[c];
#pragma unroll
  for (int c = 0; c < kNb; ++c) {
    if (LU && c >= nc) continue;
#pragma unroll
    for (int t = c + 1; t < kNb; ++t) a[t] -= sL[t][c] * a[c];
  }
#pragma unroll
  for (int c = 0; c < kNb; ++c) Rj[c] = a[c];
  if (LU && jk >= kNb && tid < out.n)
#pragma unroll
    for (int c = 0; c < kNb; ++c)
      if (k0 + c < out.n) lu[k0 + c + (long long)tid * out.n] = a[c];
  if (kTwo) {
#pragma unroll
    for (int c = 0; c < kNb; ++c) Al[k0 + c + (long long)tid * M] = own && c <= jk ? sL[c][jk] : a[c];
  }
}

// Two phases, the columns of Z, at their places in D^-1, from L^-1 (below the diagonal of A).
__global__ void __launch_bounds__(256) gj_split_kernel(const double *__restrict__ A, const int *__restrict__ perm, int m,
                                                       double *Z) {
  const long long leaf = blockIdx.x;
  const double *Al = A + leaf * m * m;
  double *Zl = Z + leaf * m * m;
  for (int e = threadIdx.x; e < m * m; e += 256) {
    const int i = e % m, p = e / m;
    Zl[i + (long long)perm[leaf * m + p] * m] = i > p ? Al[e] : i == p ? 1.0 : 0.0;
  }
}

// Rows K of Z times U11^-1 from the left, also into R: 32 columns a CTA (blockIdx.y),
// four neighbouring lanes a column, every fourth row each (one thread a column takes
// 32000 clocks, a leaf's 256 columns in one CTA 90000).
__global__ void __launch_bounds__(4 * kNb) gj_rows_kernel(const double *__restrict__ A, int m, double *Z, double *R, int k0) {
  constexpr int NC = kNb / 4;
  __shared__ double sU[kNb][kNb + 1], sRcp[kNb];
  const int tid = threadIdx.x, q = tid & 3, j = kNb * (int)blockIdx.y + (tid >> 2);
  const long long blk = blockIdx.x;
  const double *Akk = A + blk * m * m + (long long)k0 * (m + 1);
  double *z = Z + blk * m * m + k0 + (long long)j * m, *Rj = R + (blk * m + j) * kNb;
  for (int e = tid; e < kNb * kNb; e += 4 * kNb) sU[e % kNb][e / kNb] = Akk[e % kNb + (long long)(e / kNb) * m];
  double a[NC];
#pragma unroll
  for (int t = 0; t < NC; ++t) a[t] = z[4 * t + q];
  __syncthreads();
  if (tid < kNb) sRcp[tid] = rcp_usual(sU[tid][tid]) ? 1.0 / sU[tid][tid] : 0.0;
  __syncthreads();
#pragma unroll
  for (int c = kNb - 1; c >= 0; --c) {
    double w = a[c / 4];  // of the lane whose row it is
    w = sRcp[c] != 0.0 ? w * sRcp[c] : w / sU[c][c];
    w = __shfl_sync(0xffffffffu, w, c & 3, 4);
    if (q == (c & 3)) a[c / 4] = w;
    if (q < (c & 3)) a[c / 4] -= w * sU[c / 4 * 4 + q][c];
#pragma unroll
    for (int t = 0; t < c / 4; ++t) a[t] -= w * sU[4 * t + q][c];
  }
#pragma unroll
  for (int t = 0; t < NC; ++t) z[4 * t + q] = Rj[4 * t + q] = a[t];
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

// C[system](rows r0 .. r0 + rows) -= F[system](those rows, 32 columns) R[system].
static cudaError_t gj_product(int m, int count, const double *F, long long f_stride, const double *R, double *C, int r0,
                              int rows, DevStatus *st, cudaStream_t s) {
  if (rows <= 0) return cudaSuccess;
  UpdateArgs ua{};
  ua.A = F + r0;
  ua.lda = m;
  ua.a_bstride = f_stride;
  ua.B = R;
  ua.ldb = kNb;
  ua.b_s1 = 2LL * m * kNb;
  ua.b_s2 = (long long)m * kNb;
  ua.C = C + r0;
  ua.ldc = m;
  ua.c_bstride = (long long)m * m;
  ua.M = rows;
  ua.N = m;
  ua.K = kNb;
  ua.nbatch = count;
  ua.alpha = -1.0;
  cudaError_t e = cudaSuccess;
  return f64_update_tc_try(ua, st, s, e) ? e : cudaErrorInvalidValue;
}

// One phase: `count` m x m systems (m 64 and 128, or 32, 64 and 128 with the LU
// factors), worked on in place in A: on return A holds the inverses of the
// interchanged rows.  Rows and columns from n on are the identity's.
template <bool LU>
static cudaError_t gj_one(int m, int n, int count, double *A, double *W, double *R, int *perm, const unsigned *big,
                          int *again, const LuOut &out, DevStatus *st, cudaStream_t s) {
#define HODLR_GJ(MV)                                                                                            \
  HODLR_LAUNCH((gj_panel_kernel<MV, LU>), count, gj_threads<MV>(), 0, s, A, W, R, perm, k0, std::min(kNb, n - k0), big, again, \
               out)
  for (int k0 = 0; k0 < n; k0 += kNb) {
    if (m == 64) {
      HODLR_GJ(64);
    } else if (m == 128) {
      HODLR_GJ(128);
    } else {
      if (!LU || m != kNb) return cudaErrorInvalidValue;
      if constexpr (LU) HODLR_GJ(kNb);
      break;  // no other columns
    }
    cudaError_t e = gj_product(m, count, W, (long long)m * kNb, R, A, 0, k0 + kNb, st, s);
    if (e == cudaSuccess) e = gj_product(m, count, W, (long long)m * kNb, R, A, k0 + kNb, m - k0 - kNb, st, s);
    if (e != cudaSuccess) return e;
  }
#undef HODLR_GJ
  return cudaGetLastError();
}

// Two phases, leaves of 256 rows: Z = their inverses; A is worked on in place.
static cudaError_t gj_two(int count, double *A, double *Z, double *W, double *R, int *perm, const unsigned *big,
                          int *again, DevStatus *st, cudaStream_t s) {
  constexpr int M = 256;
  cudaError_t e;
  for (int k0 = 0; k0 < M; k0 += kNb) {
    HODLR_LAUNCH((gj_panel_kernel<M, false>), count, gj_threads<M>(), 0, s, A, W, R, perm, k0, kNb, big, again,
                 (LuOut{nullptr, nullptr, 0}));
    if ((e = gj_product(M, count, W, (long long)M * kNb, R, A, k0 + kNb, M - k0 - kNb, st, s)) != cudaSuccess) return e;
  }
  HODLR_LAUNCH(gj_split_kernel, count, 256, 0, s, A, perm, M, Z);
  for (int k0 = M - kNb; k0 >= 0; k0 -= kNb) {
    HODLR_LAUNCH(gj_rows_kernel, dim3(count, M / kNb), 4 * kNb, 0, s, A, M, Z, R, k0);
    if ((e = gj_product(M, count, A + (long long)k0 * M, (long long)M * M, R, Z, 0, k0, st, s)) != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

// Bytes of scratch: W, R, perm, the largest entries and the marks.
size_t f64_leaf_gj_scratch(int m, int nleaf) {
  return (size_t)nleaf * (m * (2 * kNb * sizeof(double) + sizeof(int) + 2 * sizeof(unsigned)) + sizeof(int));
}

// Dinv = D^-1 for every leaf; A: an [nleaf][m][m] workspace, ipiv: [nleaf][m].  With
// LU (m 64 and 128, not A) the factors and pivots of every leaf as well: hsolve of
// 8 leaves of 64 rows takes 0.88 ms so, 1.00 with the register-resident sweep.
cudaError_t launch_f64_leaf_gj(const double *D, long long d_ld, long long d_stride, int m, int nleaf, double *A,
                               int *ipiv, double *Dinv, double *LU, void *scratch, DevStatus *st, cudaStream_t s) {
  double *W = static_cast<double *>(scratch), *R = W + (size_t)nleaf * m * kNb;
  int *perm = reinterpret_cast<int *>(R + (size_t)nleaf * m * kNb);
  unsigned *big = reinterpret_cast<unsigned *>(perm + (size_t)nleaf * m);
  int *again = reinterpret_cast<int *>(big + (size_t)nleaf * 2 * m);
  HODLR_LAUNCH(leaf_gj_copy_kernel, nleaf, 256, 0, s, D, d_ld, d_stride, m, A, big, again, st);
  cudaError_t e = m == 256 ? gj_two(nleaf, A, Dinv, W, R, perm, big, again, st, s)
                  : LU     ? gj_one<true>(m, m, nleaf, A, W, R, perm, big, again, LuOut{LU, ipiv, m}, st, s)
                           : gj_one<false>(m, m, nleaf, A, W, R, perm, big, again, LuOut{nullptr, nullptr, 0}, st, s);
  if (e != cudaSuccess) return e;
  if (m != 256) HODLR_LAUNCH(leaf_gj_columns_kernel, nleaf, 256, 0, s, A, perm, m, Dinv);
  HODLR_LAUNCH(leaf_gj_again_kernel, nleaf, 256, 0, s, D, d_ld, d_stride, m, LU ? LU : A, ipiv, Dinv, again, st);
  return cudaGetLastError();
}

// ------------------------------------------------------ capacitance systems
// S = [I, s.T1u; s.T0u, I] of every node of a depth, padded with the identity
// to m x m; the largest |S| of its rows and columns; again = 0.
__global__ void __launch_bounds__(256) cap_gj_build_kernel(CapFactorArgs a, int m, double *A, unsigned *big,
                                                           int *again) {
  __shared__ unsigned srow[128], scol[128];
  const int p = blockIdx.x, tid = threadIdx.x, r = a.r, n2 = 2 * r;
  const long long o0 = (long long)(2 * p) * a.tb_stride + (long long)a.ucol * r, o1 = o0 + a.tb_stride;
  auto T = [&](long long off) -> double { return a.Tb32 ? (double)a.Tb32[off] : a.Tb[off]; };
  if (tid < m) srow[tid] = scol[tid] = 0;
  __syncthreads();
  unsigned mx = 0;
  for (int e = tid; e < m * m; e += 256) {
    const int i = e % m, j = e / m;
    double v = i == j ? 1.0 : 0.0;
    if (i >= r && i < n2 && j < r) v = (a.scale ? a.scale[i - r] : 1.0) * T(o0 + i - r + (long long)j * r);
    if (i < r && j >= r && j < n2) v = (a.scale ? a.scale[i] : 1.0) * T(o1 + i + (long long)(j - r) * r);
    A[(long long)p * m * m + e] = v;
    const unsigned h = (unsigned)__double2hiint(v) & 0x7fffffffu;
    mx = max(mx, h);
    const unsigned w = __reduce_max_sync(0xffffffffu, h);
    if ((tid & 31) == 0) atomicMax(&scol[j], w);
  }
  atomicMax(&srow[tid % m], mx);
  __syncthreads();
  if (tid < m) {
    big[(long long)p * 2 * m + tid] = srow[tid];
    big[(long long)p * 2 * m + m + tid] = scol[tid];
  }
  if (tid == 0) again[p] = 0;
}

// Sinv's columns from the inverse of the interchanged rows (FP32 if sinv32).
__global__ void __launch_bounds__(256) cap_gj_columns_kernel(const double *__restrict__ A, const int *__restrict__ perm,
                                                             int m, int n2, double *sinv, float *sinv32) {
  const long long p = blockIdx.x;
  for (int e = threadIdx.x; e < n2 * n2; e += 256) {
    const int i = e % n2, j = e / n2, c = perm[p * m + j];
    const double v = A[p * m * m + i + (long long)j * m];
    const long long o = p * n2 * n2 + i + (long long)c * n2;
    if (c >= n2) continue;
    if (sinv32)
      sinv32[o] = f64_to_f32_rn(v);
    else
      sinv[o] = v;
  }
}

static int cap_gj_rows(int r) { return r <= 16 ? 32 : r <= 32 ? 64 : 128; }

size_t f64_cap_gj_scratch(int r, int nnode) {
  const size_t m = cap_gj_rows(r);
  return (size_t)nnode * (m * (m + 2 * kNb) * sizeof(double) + m * (sizeof(int) + 2 * sizeof(unsigned)) + sizeof(int));
}

cudaError_t launch_f64_cap_gj(const CapFactorArgs &a, void *scratch, cudaStream_t s) {
  if (a.nnode <= 0) return cudaSuccess;
  const int m = cap_gj_rows(a.r), n2 = 2 * a.r;
  const size_t nn = a.nnode;
  double *A = static_cast<double *>(scratch), *W = A + nn * m * m, *R = W + nn * m * kNb;
  int *perm = reinterpret_cast<int *>(R + nn * m * kNb);
  unsigned *big = reinterpret_cast<unsigned *>(perm + nn * m);
  int *again = reinterpret_cast<int *>(big + nn * 2 * m);
  const LuOut out{a.cap_lu + (long long)a.node_base * n2 * n2, a.cap_ipiv + (long long)a.node_base * n2, n2};
  HODLR_LAUNCH(cap_gj_build_kernel, a.nnode, 256, 0, s, a, m, A, big, again);
  cudaError_t e = gj_one<true>(m, n2, a.nnode, A, W, R, perm, big, again, out, a.st, s);
  if (e != cudaSuccess) return e;
  const long long base = (long long)a.node_base * n2 * n2;
  HODLR_LAUNCH(cap_gj_columns_kernel, a.nnode, 256, 0, s, A, perm, m, n2, a.sinv ? a.sinv + base : nullptr,
               a.sinv32 ? a.sinv32 + base : nullptr);
  return launch_cap_factor_marked(a, again, s);
}

}  // namespace hodlr
