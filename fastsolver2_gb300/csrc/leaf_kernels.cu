// K1 / K2: batched leaf LU and leaf triangular solves.
//
// Replaces the leaf case of fastSolver2's hsolve, one dgesv per leaf on the
// CPU (src/tasks/leaf_solve.cc:80-92): here every leaf of the tree is
// factorised by one launch (one CTA per leaf, the block staged in shared
// memory when it fits) and the solves against all right-hand-side columns
// are one launch over (leaf, column tile).
#include <algorithm>
#include <cstdlib>

#include "dense_ops.cuh"
#include "kernels.cuh"
#include "reg_factor.cuh"

namespace hodlr {

bool f64_update_tc_try(const UpdateArgs &a, DevStatus *st, cudaStream_t s, cudaError_t &err);

template <typename T, bool SMEM>
__global__ void __launch_bounds__(256)
leaf_getrf_kernel(const double *__restrict__ D, long long d_ld, long long d_stride, T *LU, int *ipiv,
                  int m, DevStatus *st, T *Dinv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_bad;
  __shared__ int s_info;
  const int leaf = blockIdx.x;
  const double *Dg = D + (long long)leaf * d_stride;
  T *LUg = LU + (long long)leaf * m * m;
  T *A = SMEM ? reinterpret_cast<T *>(smem_raw) : LUg;
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
  int bad = 0;
  for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
    const int i = e % m, j = e / m;
    const double v = Dg[i + (long long)j * d_ld];
    if (!isfinite(v)) bad = 1;
    A[e] = (T)v;
  }
  if (bad) atomicOr(&s_bad, 1);
  __syncthreads();
  if (s_bad) {
    if (threadIdx.x == 0) report_error(st, HODLR_ERR_NONFINITE_INPUT, (long long)leaf * m);
    return;
  }
  block_getrf<T>(A, m, m, ipiv + (long long)leaf * m, &s_info);
  if (s_info && threadIdx.x == 0) report_error(st, HODLR_ERR_SINGULAR_LEAF, leaf);
  if (SMEM) {
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) LUg[e] = A[e];
    if (Dinv) {  // explicit inverse: Gauss-Jordan on a fresh copy of the block
      __syncthreads();
      for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
        const int i = e % m, j = e / m;
        A[e] = (T)Dg[i + (long long)j * d_ld];
      }
      __syncthreads();
      T *fcol = A + (size_t)m * m;
      int *perm = reinterpret_cast<int *>(fcol + m);
      block_gj_inverse<T>(A, m, m, fcol, perm, &s_info);
      T *out = Dinv + (long long)leaf * m * m;
      for (int e = threadIdx.x; e < m * m; e += blockDim.x) out[e] = A[e];
    }
  }
}

// Leaf LU (+ optional explicit inverse) with the block resident in registers
// (reg_factor.cuh), for M in {32, 64, 128}.
template <typename T, int M>
__global__ void __launch_bounds__(256, (sizeof(T) == 4 && M == 128) ? 2 : 1)
leaf_factor_reg_kernel(const double *__restrict__ D, long long d_ld, long long d_stride, T *LU, int *ipiv,
                       DevStatus *st, T *Dinv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_bad, s_info;
  T *buf = reinterpret_cast<T *>(smem_raw);
  const int leaf = blockIdx.x;
  const double *Dg = D + (long long)leaf * d_stride;
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
  int bad = 0;
  for (int e = threadIdx.x; e < M * M; e += blockDim.x)
    if (!isfinite(Dg[(e % M) + (long long)(e / M) * d_ld])) bad = 1;
  if (bad) atomicOr(&s_bad, 1);
  __syncthreads();
  if (s_bad) {
    if (threadIdx.x == 0) report_error(st, HODLR_ERR_NONFINITE_INPUT, (long long)leaf * M);
    return;
  }
  T *inv = Dinv ? Dinv + (long long)leaf * M * M : nullptr;
  auto load = [&](int i, int j) -> T { return (T)Dg[i + (long long)j * d_ld]; };
  auto store = [&](int i, int j, T v) { inv[i + j * M] = v; };
  reg_factor<T, M>(load, buf, LU + (long long)leaf * M * M, ipiv + (long long)leaf * M, store, inv != nullptr,
                   &s_info);
  if (s_info && threadIdx.x == 0) report_error(st, HODLR_ERR_SINGULAR_LEAF, leaf);
}

// FAR: block_getrs's, for that many CTAs an SM (0: not).
template <typename T, bool TRANS, bool LU_SMEM, int FAR>
__global__ void __launch_bounds__(256, FAR == 2 ? 2 : 0)
leaf_getrs_kernel(const T *__restrict__ LU, const int *__restrict__ ipiv, int m, T *X, long long ldx,
                  int ncols, int ct, const int *skip) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int leaf = blockIdx.y;
  const int c0 = blockIdx.x * ct;
  const int nc = min(ct, ncols - c0);
  T *sX = reinterpret_cast<T *>(smem_raw);
  int *spiv = reinterpret_cast<int *>(sX + (size_t)m * ct);
  T *sLU = reinterpret_cast<T *>(reinterpret_cast<uintptr_t>(spiv + m + 3) & ~uintptr_t(15));
  const T *gLU = LU + (long long)leaf * m * m;
  for (int i = threadIdx.x; i < m; i += blockDim.x) spiv[i] = ipiv[(long long)leaf * m + i];
  if (LU_SMEM)
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) sLU[e] = gLU[e];
  T *Xg = X + (long long)leaf * m + (long long)c0 * ldx;
  for (int e = threadIdx.x; e < m * nc; e += blockDim.x) {
    const int i = e % m, j = e / m;
    sX[e] = Xg[i + (long long)j * ldx];
  }
  __syncthreads();
  block_getrs<T, TRANS, FAR != 0>(LU_SMEM ? sLU : gLU, m, spiv, m, sX, m, nc);
  for (int e = threadIdx.x; e < m * nc; e += blockDim.x) {
    const int i = e % m, j = e / m;
    Xg[i + (long long)j * ldx] = sX[e];
  }
}

// X := D^{-1} X for many columns: 32-row diagonal blocks in launches of their own --
// 32 columns a CTA, lane = column, each of the four warps with every fourth row in
// registers, row k passed through shared memory once it is done, a step a barrier
// and up to eight FMAs --, the updates of the other rows in FP64 on the tensor cores
// (f64_update_tc.cu), in FP32 by FMAs (update_nn_kernel).  FP64 is bound by its pipe
// in the diagonal blocks (2 x 496 FMAs a column and block) and by the updates, half
// each: 2048 leaves of 100 rows, 143 columns and then 5: 5.0 ms, 22.1 with one CTA a
// leaf and column tile doing it all; 512 leaves of 300 rows, 122 columns 4.1 ms,
// 22.2.  FP32: 1024 leaves of 286 rows, 636 columns and 16 a correction 13.7 ms, 84.
template <typename T>
__global__ void __launch_bounds__(256) leaf_interchange_kernel(const int *__restrict__ ipiv, int m, T *X,
                                                               long long ldx, int ncols, int ct, const int *skip) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *sX = reinterpret_cast<T *>(smem_raw);  // [ct][m]
  int *sfrom = reinterpret_cast<int *>(sX + (size_t)m * ct), *spiv = sfrom + m;
  const int leaf = blockIdx.y, c0 = blockIdx.x * ct, nc = min(ct, ncols - c0), tid = threadIdx.x;
  T *Xg = X + (long long)leaf * m + (long long)c0 * ldx;
  for (int i = tid; i < m; i += 256) spiv[i] = ipiv[(long long)leaf * m + i] - 1;
  __syncthreads();
  for (int i = tid; i < m; i += 256) {
    int from = i;  // row i of P X
    for (int k = m - 1; k >= 0; --k) {
      const int p = spiv[k];
      from = from == k ? p : from == p ? k : from;
    }
    sfrom[i] = from;
  }
  for (int c = tid >> 5; c < nc; c += 8)
    for (int i = tid & 31; i < m; i += 32) sX[c * m + i] = Xg[i + (long long)c * ldx];
  __syncthreads();
  for (int c = tid >> 5; c < nc; c += 8)
    for (int i = tid & 31; i < m; i += 32)
      if (sfrom[i] != i) Xg[i + (long long)c * ldx] = sX[c * m + sfrom[i]];
}

template <typename T, bool UPPER>
__global__ void __launch_bounds__(128) leaf_diag_kernel(const T *__restrict__ LU, int m, int k0, T *X,
                                                        long long ldx, int ncols, const int *skip) {
  if (skip && *skip) return;
  __shared__ T sA[32][32], sX[32][33], sK[2][32];  // sA[column][row], sX[column][row]
  __shared__ Quotient<T> sR[32];
  const int leaf = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kb = min(32, m - k0);
  const int c0 = blockIdx.x * 32;
  const T *A = LU + (long long)leaf * m * m + k0 + (long long)k0 * m;
  T *Xg = X + (long long)leaf * m + k0 + (long long)c0 * ldx;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = warp + 4 * i;
    sA[c][lane] = lane < kb && c < kb ? A[lane + (long long)c * m] : c == lane ? T(1) : T(0);
    sX[c][lane] = lane < kb && c0 + c < ncols ? Xg[lane + (long long)c * ldx] : T(0);
  }
  __syncthreads();
  if (UPPER) {
    if (tid < 32) sR[tid] = Quotient<T>::by(sA[tid][tid]);
    __syncthreads();
  }
  T x[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) x[q] = sX[lane][4 * q + warp];
#pragma unroll
  for (int step = 0; step < 32; ++step) {
    const int k = UPPER ? 31 - step : step;
    if (warp == (k & 3)) {
      if (UPPER) x[k / 4] = sR[k].of(x[k / 4]);
      sK[k & 1][lane] = x[k / 4];
    }
    __syncthreads();
    const T xk = sK[k & 1][lane];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (UPPER ? 4 * q > k : 4 * q + 3 < k) continue;
      if (UPPER ? 4 * q + warp < k : 4 * q + warp > k) x[q] -= sA[k][4 * q + warp] * xk;
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) sX[lane][4 * q + warp] = x[q];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = warp + 4 * i;
    if (lane < kb && c0 + c < ncols) Xg[lane + (long long)c * ldx] = sX[c][lane];
  }
}

// The line: 4 m / 32 launches of some 10 us each against the one of
// leaf_getrs_kernel, whose time grows with the elements: 16 leaves of 180 rows, 20
// columns 0.19 ms there and 0.25 here; 32 leaves of 100 rows, 32 columns 0.16 and
// 0.16; 32 of 180 rows, 70 columns 0.77 and 0.44; 64 of 50 rows, 50 columns 0.19
// and 0.12.  In FP32, where the one kernel's FMAs cost less, from eight times the
// elements on: 64 leaves of 100 rows, 83 columns and 11 times 5 0.26 and 0.27 ms, 512
// of 72 rows, 122 columns 0.56 and 0.36.  Up to 8 columns would fill a quarter of a
// tile: 2048 leaves of 100 rows, 5 columns 0.91 and 1.10.
template <typename T> static bool leaf_getrs_by_blocks(int m, int nleaf, int ncols) {
  const char *no_tc = getenv("HODLR_NO_TCGEN05");
  if (sizeof(T) == 8 && no_tc && no_tc[0] == '1') return false;
  return m > 32 && m <= 4096 && nleaf <= 65535 && ncols > 8 && (long long)nleaf * ncols * m >= (sizeof(T) == 8 ? 1 << 17 : 1 << 20);
}

template <typename T>
static cudaError_t leaf_getrs_blocked(const T *LU, const int *ipiv, int m, int nleaf, T *X, long long ldx,
                                      int ncols, const int *skip, DevStatus *st, cudaStream_t s) {
  const int ct = std::max(1, std::min(8, (int)(96 * 1024 / ((size_t)m * sizeof(T)))));
  const size_t bytes = (size_t)m * (ct * sizeof(T) + 2 * sizeof(int));
  cudaError_t e = allow_dyn_smem(leaf_interchange_kernel<T>, bytes);
  if (e != cudaSuccess) return e;
  HODLR_LAUNCH(leaf_interchange_kernel<T>, dim3(ceil_div(ncols, ct), nleaf), 256, bytes, s, ipiv, m, X, ldx, ncols, ct,
               skip);
  const dim3 grid(ceil_div(ncols, 32), nleaf);
  auto update = [&](int k0, int r0, int r1) {  // rows [r0, r1) -= A(rows, block) X(block)
    UpdateArgs ua{};
    ua.A = LU + r0 + (long long)k0 * m;
    ua.lda = m;
    ua.a_bstride = (long long)m * m;
    if constexpr (sizeof(T) == 8)
      ua.B = X + k0;
    else
      ua.B32 = X + k0;
    ua.ldb = ldx;
    ua.b_s1 = 2LL * m;
    ua.b_s2 = m;
    ua.C = X + r0;
    ua.ldc = ldx;
    ua.c_bstride = m;
    ua.M = r1 - r0;
    ua.N = ncols;
    ua.K = std::min(32, m - k0);
    ua.nbatch = nleaf;
    ua.alpha = -1.0;
    ua.skip = skip;
    if constexpr (sizeof(T) == 4) return launch_update_fma_f32(ua, s);
    return f64_update_tc_try(ua, st, s, e) ? e : cudaErrorInvalidValue;
  };
  const int last = (m - 1) / 32 * 32;
  for (int k0 = 0; k0 <= last; k0 += 32) {
    HODLR_LAUNCH((leaf_diag_kernel<T, false>), grid, 128, 0, s, LU, m, k0, X, ldx, ncols, skip);
    if (k0 < last && (e = update(k0, k0 + 32, m)) != cudaSuccess) return e;
  }
  for (int k0 = last; k0 >= 0; k0 -= 32) {
    HODLR_LAUNCH((leaf_diag_kernel<T, true>), grid, 128, 0, s, LU, m, k0, X, ldx, ncols, skip);
    if (k0 > 0 && (e = update(k0, 0, k0)) != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

static constexpr size_t kSmemCap = 220 * 1024;

template <typename K>
static cudaError_t set_smem(K kernel, size_t bytes) {
  return allow_dyn_smem(kernel, bytes);
}

static bool reg_leaf(int m) { return m == 32 || m == 64 || m == 128; }

bool leaf_getrf_fused_inverse(int m, int elem_bytes) {
  return reg_leaf(m) || (size_t)m * (m + 1) * elem_bytes + (size_t)m * 4 <= kSmemCap;
}

template <typename T, int M>
static cudaError_t launch_reg(const double *D, long long d_ld, long long d_stride, T *LU, int *ipiv, int nleaf,
                              DevStatus *st, T *Dinv, cudaStream_t s) {
  const size_t bytes = (size_t)M * M * sizeof(T);
  auto k = leaf_factor_reg_kernel<T, M>;
  cudaError_t e = set_smem(k, bytes);
  if (e != cudaSuccess) return e;
  HODLR_LAUNCH(k, nleaf, 256, bytes, s, D, d_ld, d_stride, LU, ipiv, st, Dinv);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_leaf_getrf(const double *D, long long d_ld, long long d_stride, T *LU, int *ipiv,
                              int m, int nleaf, DevStatus *st, T *Dinv, cudaStream_t s) {
  if (m == 32) return launch_reg<T, 32>(D, d_ld, d_stride, LU, ipiv, nleaf, st, Dinv, s);
  if (m == 64) return launch_reg<T, 64>(D, d_ld, d_stride, LU, ipiv, nleaf, st, Dinv, s);
  if (m == 128) return launch_reg<T, 128>(D, d_ld, d_stride, LU, ipiv, nleaf, st, Dinv, s);
  const size_t bytes = (size_t)m * (m + 1) * sizeof(T) + (size_t)m * 4;
  // In FP64 the panels of leaf_blocked.cu from 96 rows on, where the one CTA of
  // leaf_getrf_kernel spends a leaf's time on barriers and FMAs: 2048 leaves of 100
  // rows 1.88 ms by panels and 3.06 here, 1024 of 150 rows 1.76 and 5.46, 4 of 100
  // rows 0.25 and 0.35; 256 of 72 rows 0.29 and 0.25.
  const char *no_tc = getenv("HODLR_NO_TCGEN05");
  const bool panels = sizeof(T) == 8 && m >= 96 && !Dinv && !(no_tc && no_tc[0] == '1');
  if (bytes <= kSmemCap && !panels) {
    auto k = leaf_getrf_kernel<T, true>;
    cudaError_t e = set_smem(k, bytes);
    if (e != cudaSuccess) return e;
    HODLR_LAUNCH(k, nleaf, 256, bytes, s, D, d_ld, d_stride, LU, ipiv, m, st, Dinv);
  } else {
    if (Dinv) return cudaErrorInvalidValue;  // caller forms the inverse separately
    return launch_leaf_getrf_blocked<T>(D, d_ld, d_stride, LU, ipiv, m, nleaf, st, s);
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_leaf_getrs(const T *LU, const int *ipiv, int m, int nleaf, T *X, long long ldx,
                              int ncols, bool trans, const int *skip, DevStatus *st, cudaStream_t s) {
  if (ncols <= 0 || nleaf <= 0) return cudaSuccess;
  if (!trans && leaf_getrs_by_blocks<T>(m, nleaf, ncols))
    return leaf_getrs_blocked<T>(LU, ipiv, m, nleaf, X, ldx, ncols, skip, st, s);
  const size_t lu_bytes = (size_t)m * m * sizeof(T);
  const size_t piv_bytes = (size_t)m * sizeof(int) + 16;
  // FP32: keep two CTAs per SM; FP64 is DFMA-bound, one CTA per SM suffices.
  const size_t cap = sizeof(T) == 4 ? 110 * 1024 : kSmemCap;
  bool lu_smem = lu_bytes + piv_bytes + (size_t)m * 8 * sizeof(T) <= cap;
  // FP64 factors for up to 8 columns are not worth staging where that leaves an SM
  // one leaf at a time, or many leaves in turn: 512 leaves of 129 rows, 6 columns 0.38
  // ms from the caches, 0.55 staged; 2048 of 100 rows, 5 columns 0.75 and 0.91, one
  // column 0.42 and 0.57; 32 of 100 rows 0.078 and 0.072, 2048 of 50 0.33 both.
  // Transposed (nothing is loaded ahead there) 64 of 129 rows 0.13 and 0.18, 32 of 150
  // rows 0.12 and 0.11.
  if (sizeof(T) == 8 && ncols <= 8 && m >= 64 && ((m > 128 && nleaf >= (trans ? 64 : 1)) || nleaf > 2 * kNumSMs))
    lu_smem = false;
  size_t avail = cap - piv_bytes - (lu_smem ? lu_bytes : 0);
  int ct_max = (int)std::min<size_t>(avail / ((size_t)m * sizeof(T)), 128);
  if (ct_max < 1) return cudaErrorInvalidValue;
  // enough column tiles to give every SM a CTA when the leaves are few and large
  int ntile = std::max(ceil_div(ncols, ct_max), std::min(ncols, ceil_div(kNumSMs, nleaf)));
  // Factors far away loaded ahead (block_getrs) while no SM has more than two CTAs, 128
  // registers a thread, or in FP64 more than one, 160: one column on each of 4 leaves
  // of 400 rows 0.28 ms, 0.39 without, of 256 leaves of 300 rows 0.27 and 0.49, of 512
  // leaves 0.53 and 0.52; in FP32 22 times 2 columns on 1024 leaves of 182 rows 1.7 ms
  // loaded ahead, 1.4 without.
  int far = !trans && !lu_smem ? 2 : 0;
  if (far && (long long)ntile * nleaf > 2 * kNumSMs) far = 0;
  if (!trans && !lu_smem && sizeof(T) == 8) {
    const int nt = std::max(ceil_div(ncols, ct_max), std::min(ncols, std::max(1, kNumSMs / nleaf)));
    if ((long long)nt * nleaf <= kNumSMs) {
      far = 1;
      ntile = nt;
    }
  }
  int ct = ceil_div(ncols, ntile);
  ntile = ceil_div(ncols, ct);
  size_t bytes = (size_t)m * ct * sizeof(T) + piv_bytes + (lu_smem ? lu_bytes : 0);
  dim3 grid(ntile, nleaf);
  cudaError_t e = cudaSuccess;
#define HODLR_GETRS_CASE(TR, LS, FA)                                                 \
  {                                                                                  \
    auto k = leaf_getrs_kernel<T, TR, LS, FA>;                                       \
    e = set_smem(k, bytes);                                                          \
    if (e != cudaSuccess) return e;                                                  \
    HODLR_LAUNCH(k, grid, 256, bytes, s, LU, ipiv, m, X, ldx, ncols, ct, skip);      \
  }
  if (!trans) {
    if (lu_smem) HODLR_GETRS_CASE(false, true, 0)
    else if (far == 2) HODLR_GETRS_CASE(false, false, 2)
    else if (sizeof(T) == 8 && far == 1) HODLR_GETRS_CASE(false, false, 1)
    else HODLR_GETRS_CASE(false, false, 0)
  } else {
    if (lu_smem) HODLR_GETRS_CASE(true, true, 0) else HODLR_GETRS_CASE(true, false, 0)
  }
#undef HODLR_GETRS_CASE
  return cudaGetLastError();
}

template cudaError_t launch_leaf_getrf<double>(const double *, long long, long long, double *, int *, int,
                                               int, DevStatus *, double *, cudaStream_t);
template cudaError_t launch_leaf_getrf<float>(const double *, long long, long long, float *, int *, int,
                                              int, DevStatus *, float *, cudaStream_t);
template cudaError_t launch_leaf_getrs<double>(const double *, const int *, int, int, double *, long long,
                                               int, bool, const int *, DevStatus *, cudaStream_t);
template cudaError_t launch_leaf_getrs<float>(const float *, const int *, int, int, float *, long long, int,
                                              bool, const int *, DevStatus *, cudaStream_t);

}  // namespace hodlr
