// K1 for leaves too large for one CTA's shared memory: batched right-looking
// blocked LU, the blocked order of LAPACK DGETRF (netlib_blas/dgetrf.f:109 --
// factor a panel of nb columns, apply its interchanges to the other columns
// (DLASWP), U12 = L11^{-1} A12 (DTRSM), A22 -= L21 U12 (DGEMM)): the panel of
// every leaf by one CTA, the interchanges and the triangular solve spread over
// (column tile, leaf) CTAs, the product in FP64 on the tensor cores
// (f64_update_tc.cu), in FP32 by FMAs.
//
// The result has the layout of the one-CTA kernels: LU [nleaf][m][m]
// column-major with the unit lower factor below the diagonal, 1-based pivots
// [nleaf][m], the first zero pivot reported as HODLR_ERR_SINGULAR_LEAF.
//
// The FP64 products round once where FMAs round 32 times, so a leaf whose
// elimination would cancel exactly may be left with a tiny pivot instead: a leaf
// with a pivot below 2^-40 of the largest entry of its row and of its column is
// factored again by FMAs in DGETRF's order (leaf_lu_again_kernel), which decides
// on a zero pivot.
#include <algorithm>
#include <cstdlib>

#include "dense_ops.cuh"
#include "kernels.cuh"

namespace hodlr {

bool f64_update_tc_try(const UpdateArgs &a, DevStatus *st, cudaStream_t s, cudaError_t &err);

constexpr int kPanelNb = 32;      // panel width
constexpr int kTrailCols = 32;    // columns per trailing-update CTA
constexpr int kTrailRows = 128;   // rows of L21 staged per pass

template <typename T>
static cudaError_t set_dyn_smem(T kernel, size_t bytes) {
  return allow_dyn_smem(kernel, bytes);
}

// LU[leaf] = (T) D[leaf]; the first non-finite entry is reported.
template <typename T>
__global__ void __launch_bounds__(256) leaf_blocked_init_kernel(const double *__restrict__ D, long long d_ld,
                                                                long long d_stride, int m, T *LU, DevStatus *st) {
  const int leaf = blockIdx.y;
  const double *Dg = D + (long long)leaf * d_stride;
  T *A = LU + (long long)leaf * m * m;
  const long long mm = (long long)m * m;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < mm; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % m), j = (int)(e / m);
    const double v = Dg[i + (long long)j * d_ld];
    if (!isfinite(v)) report_error(st, HODLR_ERR_NONFINITE_INPUT, (long long)leaf * m);
    A[e] = (T)v;
  }
}

// Panel [j0, j0 + jb) of every leaf (one CTA each): LU with partial pivoting
// of rows [j0, m) (the pivot is the first row of largest |a|, IDAMAX; the
// column under it scaled by the pivot's reciprocal), staged in shared memory
// when `staged`.  A zero pivot is reported unless `defer`.  For more rows than the
// kernel below takes.
template <typename T>
__global__ void __launch_bounds__(256) leaf_panel_kernel(T *LU, int m, int j0, int jb, int *ipiv, int staged,
                                                         int defer, DevStatus *st) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_p, s_info, s_piv[kPanelNb];
  __shared__ T s_pv;
  const int leaf = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x;
  T *A = LU + (long long)leaf * m * m;
  const int rows = m - j0;
  T *P = staged ? reinterpret_cast<T *>(smem_raw) : A + j0 + (long long)j0 * m;
  const long long ldp = staged ? rows : m;
  if (tid == 0) s_info = 0;
  if (staged)
    for (int e = tid; e < rows * jb; e += nt) {
      const int i = e % rows, j = e / rows;
      P[e] = A[(j0 + i) + (long long)(j0 + j) * m];
    }
  __syncthreads();
  for (int k = 0; k < jb; ++k) {
    if (warp == 0) {
      T best = T(-1);
      int bi = -1;
      for (int i = k + lane; i < rows; i += 32) {
        const T v = dabs(P[i + k * ldp]);
        if (v > best) {
          best = v;
          bi = i;
        }
      }
#pragma unroll
      for (int off = 16; off; off >>= 1) {
        const T ob = __shfl_down_sync(0xffffffffu, best, off);
        const int oi = __shfl_down_sync(0xffffffffu, bi, off);
        if (oi >= 0 && (bi < 0 || ob > best || (ob == best && oi < bi))) {
          best = ob;
          bi = oi;
        }
      }
      if (lane == 0) {
        const int p = bi < 0 ? k : bi;
        s_p = p;
        s_piv[k] = j0 + p;
        s_pv = P[p + k * ldp];
        if (s_pv == T(0) && s_info == 0) s_info = j0 + k + 1;
      }
    }
    __syncthreads();
    const int p = s_p;
    const T pv = s_pv;
    if (p != k)
      for (int j = tid; j < jb; j += nt) swap_vals(P[k + j * ldp], P[p + j * ldp]);
    __syncthreads();
    if (pv != T(0)) {
      if (dabs(pv) >= safe_min<T>()) {
        const T rcp = T(1) / pv;
        for (int i = k + 1 + tid; i < rows; i += nt) P[i + k * ldp] *= rcp;
      } else {
        for (int i = k + 1 + tid; i < rows; i += nt) P[i + k * ldp] /= pv;
      }
    }
    __syncthreads();
    const int nj = jb - k - 1;
    for (int e = tid; e < (rows - k - 1) * nj; e += nt) {
      const int i = k + 1 + e % (rows - k - 1), j = k + 1 + e / (rows - k - 1);
      P[i + j * ldp] -= P[i + k * ldp] * P[k + j * ldp];
    }
    __syncthreads();
  }
  if (staged)
    for (int e = tid; e < rows * jb; e += nt) {
      const int i = e % rows, j = e / rows;
      A[(j0 + i) + (long long)(j0 + j) * m] = P[e];
    }
  for (int k = tid; k < jb; k += nt) ipiv[(long long)leaf * m + j0 + k] = s_piv[k] + 1;
  if (tid == 0 && s_info && !defer) report_error(st, HODLR_ERR_SINGULAR_LEAF, leaf);
}

template <typename T> struct PanelBits;
template <> struct PanelBits<double> {
  static __device__ __forceinline__ void key(double v, unsigned &hi, unsigned &lo) {
    hi = (unsigned)__double2hiint(v) & 0x7fffffffu;
    lo = (unsigned)__double2loint(v);
    if (hi > 0x7ff00000u || (hi == 0x7ff00000u && lo)) hi = lo = 0;  // NaN: never preferred
  }
  static __device__ __forceinline__ double rcp(double v) {
    return rcp_usual(v) ? newton_rcp(v) : v != 0.0 ? 1.0 / v : 0.0;
  }
};
template <> struct PanelBits<float> {
  static __device__ __forceinline__ void key(float v, unsigned &hi, unsigned &lo) {
    hi = __float_as_uint(v) & 0x7fffffffu;
    lo = 0;
    if (hi > 0x7f800000u) hi = 0;
  }
  static __device__ __forceinline__ float rcp(float v) { return v != 0.0f ? 1.0f / v : 0.0f; }
};

template <typename T, int NW>  // NW: most warps with candidates
struct PanelShared {
  T u[2][NW][kPanelNb], rcp[2][NW];
  uint4 best[2][NW];  // |a| (high, low word), position, row of each warp's candidate
  unsigned top[3];    // the largest |a| (high word) published so far for a column
};

// Columns [0, nc) of the panel, one thread a row, in a: all threads of the block, of
// nw warps; pivot c moves to position c, `open`: the row may still become a pivot
// and is eliminated.  sh.top is zeroed before; pivot(c, best, value) is called in
// the thread of each pivot row.
//
// A step costs one block barrier: every warp finds its best candidate for the next
// pivot as soon as that column is up to date, and leaves its key, its whole row and,
// unless a larger candidate is there, its reciprocal in double-buffered shared
// memory; after the barrier every thread picks the best of the warps' candidates
// and reads its row.
template <typename T, int NW, typename F>
__device__ __forceinline__ void panel_eliminate(T (&a)[kPanelNb], PanelShared<T, NW> &sh, int nw, int nc, int &pos,
                                                bool &open, F pivot) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned mh = 0, ml = 0, mp = 0;
  auto candidate = [&](T v) {
    unsigned hi = 0, lo = 0;
    if (open) PanelBits<T>::key(v, hi, lo);
    mh = __reduce_max_sync(0xffffffffu, hi);
    ml = sizeof(T) == 8 ? __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u) : 0u;
    mp = __reduce_min_sync(0xffffffffu, open && hi == mh && lo == ml ? (unsigned)pos : 0xffffu);
    return mp == 0xffffu ? lane == 0 : (open && (unsigned)pos == mp);
  };
  auto publish = [&](int c, T v) {
    sh.best[c & 1][warp] = make_uint4(mh, ml, mp, tid);
    if (mh >= atomicMax(&sh.top[c % 3], mh)) sh.rcp[c & 1][warp] = PanelBits<T>::rcp(v);  // may be the pivot's
  };
  const bool first = candidate(a[0]);
  if (first) {
    publish(0, a[0]);
#pragma unroll
    for (int j = 0; j < kPanelNb; ++j) sh.u[0][warp][j] = a[j];
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < kPanelNb; ++c) {
    if (c >= nc) continue;
    const int buf = c & 1, c1 = c + 1 < kPanelNb ? c + 1 : c;
    if (tid == 0) sh.top[(c + 2) % 3] = 0;
    // the best candidate: lane w has warp w's
    const uint4 o = lane < nw ? sh.best[buf][lane] : make_uint4(0, 0, 0xffffu, 0);
    const unsigned hi = o.z == 0xffffu ? 0u : o.x + 1, bh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned bl = __reduce_max_sync(0xffffffffu, hi == bh ? o.y : 0u);
    const unsigned bz = __reduce_min_sync(0xffffffffu, hi == bh && o.y == bl ? o.z : 0xffffu);
    const int bw = __ffs(__ballot_sync(0xffffffffu, hi == bh && o.y == bl && o.z == bz)) - 1;
    const uint4 best = sh.best[buf][bw];
    const T *u = sh.u[buf][bw];
    const T pv = u[c];
    if (tid == (int)best.w) {
      open = false;
      pos = c;
      pivot(c, best, pv);
    } else if (pos == c) {
      pos = (int)best.z;
    }
    T l = T(0);
    if (open) {
      l = a[c];
      if (pv != T(0)) l = dabs(pv) >= safe_min<T>() ? l * sh.rcp[buf][bw] : l / pv;
      a[c] = l;
      if (c1 > c) a[c1] -= l * u[c1];
    }
    if (c + 1 < nc) {
      const bool cand = candidate(a[c1]);
      if (open) {
#pragma unroll
        for (int j = c + 2; j < kPanelNb; ++j) a[j] -= l * u[j];
      }
      if (cand) {
        publish(c1, a[c1]);
#pragma unroll
        for (int j = c1; j < kPanelNb; ++j) sh.u[buf ^ 1][warp][j] = a[j];
      }
      __syncthreads();
    }
  }
}

// The same panel with one thread a row and the panel's columns in registers
// (panel_eliminate), for up to kPanelMaxRows rows.  With the kernel below, four leaves of
// 400 rows take 1.2 ms in FP64 by 13 panels, 2.9 before; 512 of 300 rows 4.0 ms,
// 13.3; bound by the FP64 pipe, a panel's 496 FMAs a row, and for a few leaves by
// the steps' latency.
constexpr int kPanelMaxRows = 640;
template <typename T, int MT>  // MT: most threads
__global__ void __launch_bounds__(MT) leaf_panel_rows_kernel(T *LU, int m, int j0, int jb, int *ipiv, int defer,
                                                            DevStatus *st) {
  constexpr int NB = kPanelNb;
  __shared__ PanelShared<T, MT / 32> sh;
  __shared__ int sBad;
  const int leaf = blockIdx.x, tid = threadIdx.x;
  T *A = LU + (long long)leaf * m * m + j0 + (long long)j0 * m;
  const bool real = tid < m - j0;
  int pos = tid;
  bool open = real;
  T a[NB];
#pragma unroll
  for (int c = 0; c < NB; ++c) a[c] = real && c < jb ? A[tid + (long long)c * m] : T(0);
  if (tid == 0) sBad = sh.top[0] = sh.top[1] = sh.top[2] = 0;
  __syncthreads();
  panel_eliminate(a, sh, blockDim.x / 32, jb, pos, open, [&](int c, const uint4 &best, T pv) {
    ipiv[(long long)leaf * m + j0 + c] = j0 + (int)best.z + 1;
    if (pv == T(0)) sBad = 1;
  });
  if (real) {
#pragma unroll
    for (int c = 0; c < NB; ++c)
      if (c < jb) A[pos + (long long)c * m] = a[c];
  }
  __syncthreads();
  if (tid == 0 && sBad && !defer) report_error(st, HODLR_ERR_SINGULAR_LEAF, leaf);
}

// The panel's interchanges on 32 of the other columns, and in those right of it
// U12 = L11^{-1} A12 in DTRSM's order: CTA (tile, leaf), lane = column, each of
// the four warps with every fourth row of U12 in registers, row c passed through
// shared memory once it is done.  At most 64 rows of a column move: a thread
// follows each back through the interchanges.
template <typename T>
__global__ void __launch_bounds__(128) leaf_rows_kernel(T *LU, int m, int j0, int jb, const int *__restrict__ ipiv) {
  constexpr int NB = kPanelNb;
  __shared__ T sM[2 * NB][33], sL[NB][NB], sX[2][32];
  __shared__ int sPiv[NB], sTo[2 * NB], sFrom[2 * NB];
  const int leaf = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T *A = LU + (long long)leaf * m * m;
  if (tid < jb) sPiv[tid] = ipiv[(long long)leaf * m + j0 + tid] - 1;
  for (int e = tid; e < jb * jb; e += 128) sL[e % jb][e / jb] = A[j0 + e % jb + (long long)(j0 + e / jb) * m];
  __syncthreads();
  if (tid < 2 * jb) {
    const int to = tid < jb ? j0 + tid : sPiv[tid - jb];
    int from = to;
    for (int k = jb - 1; k >= 0; --k) {
      const int p = sPiv[k];
      from = from == j0 + k ? p : from == p ? j0 + k : from;
    }
    sTo[tid] = to;
    sFrom[tid] = from;
  }
  __syncthreads();
  auto column = [&](int c) {  // of the matrix; m from the last on
    const int o = 32 * (int)blockIdx.x + c;
    return o >= m - jb ? m : o < j0 ? o : o + jb;
  };
  for (int e = tid; e < 2 * jb * 32; e += 128) {
    const int k = e % (2 * jb), c = e / (2 * jb), col = column(c);
    sM[k][c] = col < m ? A[sFrom[k] + (long long)col * m] : T(0);
  }
  __syncthreads();
  for (int e = tid; e < jb * 32; e += 128) {  // below the panel's rows (a row met twice gets the same value)
    const int k = jb + e % jb, c = e / jb, col = column(c);
    if (col < m && sTo[k] >= j0 + jb) A[sTo[k] + (long long)col * m] = sM[k][c];
  }
  if (32 * (int)blockIdx.x + 31 >= j0) {
    T x[NB / 4];
#pragma unroll
    for (int q = 0; q < NB / 4; ++q) x[q] = 4 * q + warp < jb ? sM[4 * q + warp][lane] : T(0);
#pragma unroll
    for (int c = 0; c < NB; ++c) {
      if (c >= jb) continue;
      if (warp == (c & 3)) sX[c & 1][lane] = x[c / 4];
      __syncthreads();
      const T xc = sX[c & 1][lane];
#pragma unroll
      for (int q = c / 4; q < NB / 4; ++q)
        if (4 * q + warp > c && 4 * q + warp < jb) x[q] -= xc * sL[4 * q + warp][c];
    }
    if (column(lane) > j0)
#pragma unroll
      for (int q = 0; q < NB / 4; ++q)
        if (4 * q + warp < jb) sM[4 * q + warp][lane] = x[q];
    __syncthreads();
  }
  for (int e = tid; e < jb * 32; e += 128) {
    const int k = e % jb, c = e / jb, col = column(c);
    if (col < m) A[j0 + k + (long long)col * m] = sM[k][c];
  }
}

// Trailing update after panel [j0, j0 + jb) by FMAs: CTA (tile, leaf) owns columns
// [c0, c0 + 32) right of the panel: A22 -= L21 U12 in passes of 128 rows, the
// products of each entry summed in panel-column order.
template <typename T>
__global__ void __launch_bounds__(256) leaf_trail_kernel(T *LU, int m, int j0, int jb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *sU = reinterpret_cast<T *>(smem_raw);            // jb x 32, ld kPanelNb
  T *sL21 = sU + kPanelNb * kTrailCols;               // 128 x jb, element (r, k) at [k * 128 + r]
  const int leaf = blockIdx.y, tid = threadIdx.x, nt = blockDim.x;
  T *A = LU + (long long)leaf * m * m;
  const int c0 = j0 + jb + blockIdx.x * kTrailCols;
  const int nc = min(kTrailCols, m - c0);
  for (int e = tid; e < jb * nc; e += nt) {
    const int i = e % jb, c = e / jb;
    sU[i + c * kPanelNb] = A[(j0 + i) + (long long)(c0 + c) * m];
  }
  // A22 -= L21 U12: thread (lane, group) owns rows lane + 32a (a < 4) and columns 4 group + b (b < 4)
  const int lane = tid & 31, grp = tid >> 5;
  for (int r0 = j0 + jb; r0 < m; r0 += kTrailRows) {
    const int nr = min(kTrailRows, m - r0);
    __syncthreads();
    for (int e = tid; e < kTrailRows * jb; e += nt) {
      const int r = e % kTrailRows, k = e / kTrailRows;
      sL21[k * kTrailRows + r] = r < nr ? A[(r0 + r) + (long long)(j0 + k) * m] : T(0);
    }
    __syncthreads();
    T acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int r = lane + 32 * a, c = 4 * grp + b;
        acc[a][b] = (r < nr && c < nc) ? A[(r0 + r) + (long long)(c0 + c) * m] : T(0);
      }
    for (int k = 0; k < jb; ++k) {
      T l[4], u[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) l[a] = sL21[k * kTrailRows + lane + 32 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) u[b] = sU[k + (4 * grp + b) * kPanelNb];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] -= l[a] * u[b];
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int r = lane + 32 * a, c = 4 * grp + b;
        if (r < nr && c < nc) A[(r0 + r) + (long long)(c0 + c) * m] = acc[a][b];
      }
  }
}

// Explicit inverses D^{-1} = U^{-1} L^{-1} P from the LU factors of every leaf:
// CTA (tile, leaf) owns columns [c0, c0 + 32) of the inverse, all m rows in
// shared memory, a row's 32 columns side by side.  The identity's columns get
// the interchanges, then a blocked unit-lower solve (32-row diagonal blocks, the
// rows below updated by the block's L panel in passes of 256 rows) and a blocked
// upper solve from the bottom (diagonal blocks by division, the rows above
// updated by the block's U panel) -- the DGETRS order on the identity.  (For
// solves with a few right-hand sides launch_leaf_getrs, which spreads the columns
// over every SM, is faster.)
//
// A diagonal block takes no barrier: a warp has four of the columns, lane = row, a
// step a shuffle and an FMA a column.  In a pass a thread has 4 rows x 8 columns:
// 6 shared-memory wavefronts a warp for 32 FMAs.  1024 FP32 leaves of 256 rows take
// 3.7 ms, 4.1 with 4 x 4 a thread.
constexpr int kInvRows = 256;  // rows of a pass
template <typename T>
__global__ void __launch_bounds__(256) leaf_inverse_blocked_kernel(const T *__restrict__ LU,
                                                                   const int *__restrict__ ipiv, int m, T *Dinv) {
  constexpr int NB = kPanelNb, LD = kTrailCols + 4;
  struct alignas(16) Four {
    T v[4];
  };
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *sX = reinterpret_cast<T *>(smem_raw);  // m x 32, column c of row i at [i * LD + c]
  T *sP = sX + (size_t)m * LD;              // panel pass: 256 x 32, [k * 256 + r]
  int *spiv = reinterpret_cast<int *>(sP);  // (before the first pass)
  const int leaf = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T *A = LU + (long long)leaf * m * m;
  const int c0 = blockIdx.x * kTrailCols, nc = min(kTrailCols, m - c0);
  T *out = Dinv + (long long)leaf * m * m + (long long)c0 * m;
  for (int i = tid; i < m; i += 256) spiv[i] = ipiv[(long long)leaf * m + i] - 1;
  __syncthreads();
  for (int i = tid; i < m; i += 256) {
    int from = i;  // row i of P I
    for (int k = m - 1; k >= 0; --k) {
      const int p = spiv[k];
      from = from == k ? p : from == p ? k : from;
    }
    for (int c = 0; c < kTrailCols; ++c) sX[i * LD + c] = from == c0 + c ? T(1) : T(0);
  }
  // rows [r0, r1) -= A(rows, kb block) X(kb block rows, :)
  auto panel_update = [&](int kb0, int kbn, int r0, int r1) {
    const int g = warp & 3, h = warp >> 2;  // columns 8 g + (0..7), rows 128 h + lane + 32 (0..3) of a pass
    for (int p0 = r0; p0 < r1; p0 += kInvRows) {
      const int nr = min(kInvRows, r1 - p0);
      __syncthreads();
#pragma unroll
      for (int k = 0; k < NB; ++k)
        sP[k * kInvRows + tid] = tid < nr && k < kbn ? A[(p0 + tid) + (long long)(kb0 + k) * m] : T(0);
      __syncthreads();
      if (128 * h >= nr) continue;
      T acc[4][8];
      T *Xr = sX + (p0 + 128 * h + lane) * LD + 8 * g;
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          Four f{};
          if (128 * h + lane + 32 * a < nr) f = *reinterpret_cast<const Four *>(Xr + 32 * a * LD + 4 * q);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[a][4 * q + e] = f.v[e];
        }
      for (int k = 0; k < kbn; ++k) {
        T l[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) l[a] = sP[k * kInvRows + 128 * h + lane + 32 * a];
        const Four u0 = *reinterpret_cast<const Four *>(sX + (kb0 + k) * LD + 8 * g);
        const Four u1 = *reinterpret_cast<const Four *>(sX + (kb0 + k) * LD + 8 * g + 4);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            acc[a][e] -= l[a] * u0.v[e];
            acc[a][4 + e] -= l[a] * u1.v[e];
          }
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          Four f;
#pragma unroll
          for (int e = 0; e < 4; ++e) f.v[e] = acc[a][4 * q + e];
          if (128 * h + lane + 32 * a < nr) *reinterpret_cast<Four *>(Xr + 32 * a * LD + 4 * q) = f;
        }
    }
  };
  // a diagonal block: the block's rows of the factors in registers
  T d[NB];
  Four x;
  auto load = [&](int kb0, int kbn) {
#pragma unroll
    for (int k = 0; k < NB; ++k)
      d[k] = lane < kbn && k < kbn ? A[(kb0 + lane) + (long long)(kb0 + k) * m] : T(k == lane);
    __syncthreads();
    x = Four{};
    if (lane < kbn) x = *reinterpret_cast<const Four *>(sX + (kb0 + lane) * LD + 4 * warp);
  };
  auto store = [&](int kb0, int kbn) {
    if (lane < kbn) *reinterpret_cast<Four *>(sX + (kb0 + lane) * LD + 4 * warp) = x;
  };
  for (int kb0 = 0; kb0 < m; kb0 += NB) {  // L Y = P X
    const int kbn = min(NB, m - kb0);
    load(kb0, kbn);
#pragma unroll
    for (int k = 0; k + 1 < NB; ++k)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const T xk = __shfl_sync(0xffffffffu, x.v[c], k);
        if (lane > k) x.v[c] -= xk * d[k];
      }
    store(kb0, kbn);
    if (kb0 + kbn < m) panel_update(kb0, kbn, kb0 + kbn, m);
  }
  for (int kb0 = (m - 1) / NB * NB; kb0 >= 0; kb0 -= NB) {  // U X = Y
    const int kbn = min(NB, m - kb0);
    load(kb0, kbn);
    T u = T(1);  // the lane's pivot
#pragma unroll
    for (int k = 0; k < NB; ++k)
      if (k == lane) u = d[k];
#pragma unroll
    for (int k = NB - 1; k >= 0; --k) {
      if (k >= kbn) continue;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (lane == k) x.v[c] /= u;
        const T xk = __shfl_sync(0xffffffffu, x.v[c], k);
        if (lane < k) x.v[c] -= xk * d[k];
      }
    }
    store(kb0, kbn);
    if (kb0 > 0) panel_update(kb0, kbn, 0, kb0);
  }
  __syncthreads();
  for (int c = warp; c < nc; c += 8)
    for (int i = lane; i < m; i += 32) out[i + (long long)c * m] = sX[i * LD + c];
}

size_t leaf_inverse_blocked_smem(int m, int elem_bytes) {
  return (size_t)elem_bytes * ((size_t)m * (kTrailCols + 4) + (size_t)kInvRows * kPanelNb);
}

template <typename T>
cudaError_t launch_leaf_inverse_blocked(const T *LU, const int *ipiv, int m, int nleaf, T *Dinv, cudaStream_t s) {
  const size_t bytes = leaf_inverse_blocked_smem(m, sizeof(T));
  cudaError_t e = set_dyn_smem(leaf_inverse_blocked_kernel<T>, bytes);
  if (e != cudaSuccess) return e;
  dim3 grid(ceil_div(m, kTrailCols), nleaf);
  HODLR_LAUNCH(leaf_inverse_blocked_kernel<T>, grid, 256, bytes, s, LU, ipiv, m, Dinv);
  return cudaGetLastError();
}

template cudaError_t launch_leaf_inverse_blocked<double>(const double *, const int *, int, int, double *,
                                                         cudaStream_t);
template cudaError_t launch_leaf_inverse_blocked<float>(const float *, const int *, int, int, float *, cudaStream_t);


// The leaves with a pivot below 2^-40 of the largest entry of its row and of its
// column in D (exponents): LU again by FMAs in DGETF2's order, a zero pivot
// reported.  Leaves with non-finite entries are left as they are (reported by
// the copy).
constexpr int kAgainMaxRows = 2048;
__global__ void __launch_bounds__(512) leaf_lu_again_kernel(const double *__restrict__ D, long long d_ld,
                                                            long long d_stride, int m, double *LU, int *ipiv,
                                                            DevStatus *st) {
  __shared__ unsigned srow[kAgainMaxRows], scol[kAgainMaxRows];
  __shared__ int spiv[kAgainMaxRows], s_info;
  const long long leaf = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double *Dl = D + leaf * d_stride;
  double *A = LU + leaf * m * m;
  for (int i = tid; i < m; i += 512) {
    srow[i] = scol[i] = 0;
    spiv[i] = ipiv[leaf * m + i] - 1;
  }
  __syncthreads();
  for (int j0 = 8 * warp; j0 < m; j0 += 8 * 16) {  // a warp takes 8 columns at a time
    unsigned cm[8] = {};
    for (int i0 = 0; i0 < m; i0 += 32) {
      const int i = i0 + lane;
      unsigned h[8], rm = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e)
        h[e] = i < m && j0 + e < m ? (unsigned)__double2hiint(Dl[i + (j0 + e) * d_ld]) & 0x7fffffffu : 0u;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        cm[e] = max(cm[e], h[e]);
        rm = max(rm, h[e]);
      }
      if (i < m) atomicMax(&srow[i], rm);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const unsigned w = __reduce_max_sync(0xffffffffu, cm[e]);
      if (lane == 0 && j0 + e < m) scol[j0 + e] = w;
    }
  }
  __syncthreads();
  bool bad = false, again = false;
  for (int k = tid; k < m; k += 512) {
    int from = k;  // the row of D whose elimination left row k of U
    for (int t = m - 1; t >= 0; --t) {
      const int p = spiv[t];
      from = from == t ? p : from == p ? t : from;
    }
    const double pv = A[k + (long long)k * m];
    const unsigned h = (unsigned)__double2hiint(pv) & 0x7fffffffu;
    bad |= scol[k] >= 0x7ff00000u;
    again |= pv == 0.0 || h + (40u << 20) < min(srow[from], scol[k]);
  }
  bad = __syncthreads_or(bad);
  again = __syncthreads_or(again);
  if (bad || !again) return;
  for (int e = tid; e < m * m; e += 512) A[e] = Dl[e % m + (long long)(e / m) * d_ld];
  __syncthreads();
  block_getrf<double>(A, m, m, ipiv + leaf * m, &s_info);
  if (tid == 0 && s_info) report_error(st, HODLR_ERR_SINGULAR_LEAF, leaf);
}

template <typename T>
cudaError_t launch_leaf_getrf_blocked(const double *D, long long d_ld, long long d_stride, T *LU, int *ipiv, int m,
                                      int nleaf, DevStatus *st, cudaStream_t s) {
  if (m < 1 || nleaf < 1) return cudaSuccess;
  {
    const long long per = ((long long)m * m + 255) / 256;
    dim3 grid((unsigned)std::min<long long>(per, 64), nleaf);
    HODLR_LAUNCH(leaf_blocked_init_kernel<T>, grid, 256, 0, s, D, d_ld, d_stride, m, LU, st);
  }
  const size_t trail_bytes = sizeof(T) * ((size_t)kPanelNb * kTrailCols + (size_t)kTrailRows * kPanelNb);
  cudaError_t e = set_dyn_smem(leaf_trail_kernel<T>, trail_bytes);
  if (e != cudaSuccess) return e;
  constexpr size_t kPanelSmemCap = 200 * 1024;
  const char *no_tc = getenv("HODLR_NO_TCGEN05");
  const bool tc = sizeof(T) == 8 && m <= kAgainMaxRows && !(no_tc && no_tc[0] == '1');
  const long long mm = (long long)m * m;
  for (int j0 = 0; j0 < m; j0 += kPanelNb) {
    const int jb = std::min(kPanelNb, m - j0), rows = m - j0, rest = rows - jb;
    const int threads = ceil_div(rows, 32) * 32;
    const size_t pbytes = sizeof(T) * (size_t)rows * jb;
    if (threads <= kPanelMaxRows / 2) {
      HODLR_LAUNCH((leaf_panel_rows_kernel<T, kPanelMaxRows / 2>), nleaf, threads, 0, s, LU, m, j0, jb, ipiv, (int)tc,
                   st);
    } else if (threads <= kPanelMaxRows) {
      HODLR_LAUNCH((leaf_panel_rows_kernel<T, kPanelMaxRows>), nleaf, threads, 0, s, LU, m, j0, jb, ipiv, (int)tc, st);
    } else {
      const bool staged = pbytes <= kPanelSmemCap;
      if (staged && (e = set_dyn_smem(leaf_panel_kernel<T>, pbytes)) != cudaSuccess) return e;
      HODLR_LAUNCH(leaf_panel_kernel<T>, nleaf, 256, staged ? pbytes : 0, s, LU, m, j0, jb, ipiv, (int)staged, (int)tc,
                   st);
    }
    if (m > jb) {
      dim3 grid(ceil_div(m - jb, 32), nleaf);
      HODLR_LAUNCH(leaf_rows_kernel<T>, grid, 128, 0, s, LU, m, j0, jb, ipiv);
    }
    if (rest < 1) break;
    if (tc) {
      UpdateArgs ua{};
      ua.A = LU + (j0 + jb) + (long long)j0 * m;
      ua.lda = m;
      ua.a_bstride = mm;
      ua.B = reinterpret_cast<const double *>(LU) + j0 + (long long)(j0 + jb) * m;
      ua.ldb = m;
      ua.b_s1 = 2 * mm;
      ua.b_s2 = mm;
      ua.C = LU + (j0 + jb) + (long long)(j0 + jb) * m;
      ua.ldc = m;
      ua.c_bstride = mm;
      ua.M = ua.N = rest;
      ua.K = jb;
      ua.nbatch = nleaf;
      ua.alpha = -1.0;
      if (!f64_update_tc_try(ua, st, s, e)) return cudaErrorInvalidValue;
      if (e != cudaSuccess) return e;
    } else {
      dim3 grid(ceil_div(rest, kTrailCols), nleaf);
      HODLR_LAUNCH(leaf_trail_kernel<T>, grid, 256, trail_bytes, s, LU, m, j0, jb);
    }
  }
  if constexpr (sizeof(T) == 8)
    if (tc) HODLR_LAUNCH(leaf_lu_again_kernel, nleaf, 512, 0, s, D, d_ld, d_stride, m, LU, ipiv, st);
  return cudaGetLastError();
}

template cudaError_t launch_leaf_getrf_blocked<double>(const double *, long long, long long, double *, int *, int,
                                                       int, DevStatus *, cudaStream_t);
template cudaError_t launch_leaf_getrf_blocked<float>(const double *, long long, long long, float *, int *, int,
                                                      int, DevStatus *, cudaStream_t);

}  // namespace hodlr
