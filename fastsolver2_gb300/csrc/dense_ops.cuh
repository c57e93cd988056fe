// Block-wide dense LU and triangular solves on one small column-major matrix
// (shared or global memory).  One CTA owns the matrix; all threads of the
// block must call these functions.  These are the per-block arithmetic of
// LAPACK DGETRF / DGETRS (netlib_blas/dgetrf.f, dgetrs.f), reorganised for a
// CTA: warp-shuffle pivot search, 32-row diagonal blocks solved one warp per
// right-hand side, the rest as block-wide multiply-subtracts.
#pragma once
#include <cfloat>

#include "common.cuh"

namespace hodlr {

template <typename T> __device__ __forceinline__ T safe_min();
template <> __device__ __forceinline__ double safe_min<double>() { return DBL_MIN; }
template <> __device__ __forceinline__ float safe_min<float>() { return FLT_MIN; }

template <typename T> __device__ __forceinline__ void swap_vals(T &a, T &b) {
  T t = a;
  a = b;
  b = t;
}

// 1 / x within 0.52 ulp for |x| in 2^-960 .. 2^961 (rcp_usual): the hyperpower
// iteration of order three (Altman, Pacific J. Math. 10, 1960), y <- y (1 + e + e^2)
// with e = 1 - x y, on the hardware's approximation.  Its 20 correct bits become 60:
// 2^-7 ulp, and the last FMA rounds once.  Three FMAs where a division takes 440 clocks.
__device__ __forceinline__ double newton_rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ bool rcp_usual(double x) {
  return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 63u < 1921u;
}

// Quotients by one divisor, in FP64 by its reciprocal in two parts, hi + lo = 1 / u to
// 2^-104: x hi + x lo with one rounding of the sum, so within 0.5 + 2^-40 ulp of x / u
// and another value than the division's only that close to the middle of two; within
// an ulp where the quotient or its second part is subnormal.  Extreme divisors,
// infinities and NaNs are left to the division.
template <typename T> struct Quotient {
  T u;
  __device__ __forceinline__ static Quotient by(T u) { return Quotient{u}; }
  __device__ __forceinline__ T of(T x) const { return x / u; }
};
template <> struct Quotient<double> {
  double u, hi, lo;
  int ok;
  __device__ __forceinline__ static Quotient by(double u) {
    const double hi = 1.0 / u;
    return Quotient{u, hi, fma(-u, hi, 1.0) * hi, fabs(u) > 1e-280 && fabs(u) < 1e280};
  }
  __device__ __forceinline__ double of(double x) const {  // x / u
    const double q = fma(x, hi, x * lo);
    return ok && isfinite(q) ? q : x / u;
  }
};

// In-place LU with partial pivoting of the m x m matrix A (lda).  piv gets the
// 1-based LAPACK pivots.  *info = 0, or k+1 for the first zero pivot k.  The
// pivot is the first row of maximal |a| (IDAMAX, netlib_blas/idamax.f:52).
// piv and info may live in shared or global memory.
template <typename T>
__device__ void block_getrf(T *A, int lda, int m, int *piv, int *info) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5;
  __shared__ int s_p;
  __shared__ T s_pv;
  __shared__ int s_info;
  if (tid == 0) s_info = 0;
  const int ti = tid & 31, tj = tid >> 5, ntj = nt >> 5;
  for (int k = 0; k < m; ++k) {
    if (warp == 0) {
      T best = T(-1);
      int bi = -1;
      for (int i = k + lane; i < m; i += 32) {
        T v = dabs(A[i + (long long)k * lda]);
        if (v > best) {
          best = v;
          bi = i;
        }
      }
#pragma unroll
      for (int off = 16; off; off >>= 1) {
        T ob = __shfl_down_sync(0xffffffffu, best, off);
        int oi = __shfl_down_sync(0xffffffffu, bi, off);
        if (oi >= 0 && (bi < 0 || ob > best || (ob == best && oi < bi))) {
          best = ob;
          bi = oi;
        }
      }
      if (lane == 0) {
        int p = bi < 0 ? k : bi;
        piv[k] = p + 1;
        s_p = p;
        T pv = A[p + (long long)k * lda];
        s_pv = pv;
        if (pv == T(0) && s_info == 0) s_info = k + 1;
      }
    }
    __syncthreads();
    const int p = s_p;
    const T pv = s_pv;
    if (p != k)
      for (int j = tid; j < m; j += nt) swap_vals(A[k + (long long)j * lda], A[p + (long long)j * lda]);
    __syncthreads();
    if (pv != T(0)) {
      if (dabs(pv) >= safe_min<T>()) {
        const T rcp = T(1) / pv;
        for (int i = k + 1 + tid; i < m; i += nt) A[i + (long long)k * lda] *= rcp;
      } else {
        for (int i = k + 1 + tid; i < m; i += nt) A[i + (long long)k * lda] /= pv;
      }
    }
    __syncthreads();
    for (int j = k + 1 + tj; j < m; j += ntj) {
      const T akj = A[k + (long long)j * lda];
      T *Aj = A + (long long)j * lda;
      const T *Ak = A + (long long)k * lda;
      for (int i = k + 1 + ti; i < m; i += 32) Aj[i] -= Ak[i] * akj;
    }
    __syncthreads();
  }
  if (tid == 0) *info = s_info;
  __syncthreads();
}

// In-place inverse of the n x n matrix A by Gauss-Jordan elimination with
// the partial-pivoting rule of block_getrf (first row of maximal |a|; the
// rows searched are the Schur complement rows, so the pivot sequence is the
// LU's).  Every step is a full 2-D rank-1 update over the block, so all
// threads stay busy: n^3 multiply-adds at 4 block barriers per column.
// fcol: n scratch entries, perm: n ints (shared memory).  Returns the first
// zero pivot (k+1) or 0 in *info.
template <typename T>
__device__ void block_gj_inverse(T *A, int lda, int n, T *fcol, int *perm, int *info) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int ti = tid & 31, tj = tid >> 5, ntj = nt >> 5;
  __shared__ int s_p, s_info;
  if (tid == 0) s_info = 0;
  for (int k = 0; k < n; ++k) {
    if (warp == 0) {
      T best = T(-1);
      int bi = -1;
      for (int i = k + lane; i < n; i += 32) {
        const T v = dabs(A[i + (long long)k * lda]);
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
        perm[k] = p;
        if (A[p + (long long)k * lda] == T(0) && s_info == 0) s_info = k + 1;
      }
    }
    __syncthreads();
    const int p = s_p;
    if (p != k)
      for (int j = tid; j < n; j += nt) swap_vals(A[k + (long long)j * lda], A[p + (long long)j * lda]);
    __syncthreads();
    const T akk = A[k + (long long)k * lda];
    const T d = akk != T(0) ? T(1) / akk : T(0);
    // scale row k (its diagonal becomes d) and save column k
    for (int j = tid; j < n; j += nt) {
      T *x = A + k + (long long)j * lda;
      *x = (j == k) ? d : *x * d;
    }
    for (int i = tid; i < n; i += nt) fcol[i] = A[i + (long long)k * lda];
    __syncthreads();
    for (int j = tj; j < n; j += ntj) {
      const T akj = A[k + (long long)j * lda];
      T *Aj = A + (long long)j * lda;
      for (int i = ti; i < n; i += 32) {
        if (i == k) continue;
        Aj[i] = (j == k) ? -fcol[i] * akj : Aj[i] - fcol[i] * akj;
      }
    }
    __syncthreads();
  }
  // the row interchanges become column interchanges of the inverse, in reverse
  for (int i = tid; i < n; i += nt)
    for (int k = n - 1; k >= 0; --k) {
      const int p = perm[k];
      if (p != k) swap_vals(A[i + (long long)k * lda], A[i + (long long)p * lda]);
    }
  if (tid == 0) *info = s_info;
  __syncthreads();
}

// In-place inverse from the LU factors and pivots of block_getrf, in the
// order of LAPACK DGETRI's unblocked path: inv(U) column by column (DTRTI2),
// then inv(A) inv(L)... solved right to left, then the column interchanges
// undone in reverse.  work: n scratch entries (shared memory).
template <typename T>
__device__ void block_getri(T *A, int lda, int n, const int *piv, T *work) {
  const int tid = threadIdx.x, nt = blockDim.x;
  auto a = [&](int i, int j) -> T & { return A[i + (long long)j * lda]; };
  // 1. inv(U): A[0:j, j] = -inv(U)[j,j] * inv(U)[0:j,0:j] * A[0:j, j]
  for (int j = 0; j < n; ++j) {
    for (int i = tid; i < j; i += nt) work[i] = a(i, j);
    __syncthreads();
    const T dj = T(1) / a(j, j);
    for (int i = tid; i < j; i += nt) {
      T acc = T(0);
      for (int k = i; k < j; ++k) acc += a(i, k) * work[k];
      a(i, j) = -dj * acc;
    }
    __syncthreads();
    if (tid == 0) a(j, j) = dj;
    __syncthreads();
  }
  // 2. solve X L = inv(U) for X, columns n-2 .. 0
  for (int j = n - 2; j >= 0; --j) {
    for (int i = j + 1 + tid; i < n; i += nt) work[i] = a(i, j);
    __syncthreads();
    for (int i = tid; i < n; i += nt) {
      T acc = (i > j) ? T(0) : a(i, j);
      for (int k = j + 1; k < n; ++k) acc -= a(i, k) * work[k];
      a(i, j) = acc;
    }
    __syncthreads();
  }
  // 3. undo the row interchanges of P as column interchanges, in reverse
  for (int i = tid; i < n; i += nt)
    for (int j = n - 2; j >= 0; --j) {
      const int jp = piv[j] - 1;
      if (jp != j) swap_vals(a(i, j), a(i, jp));
    }
  __syncthreads();
}

// Row interchanges of a column tile, in LAPACK DLASWP order (forward) or
// reversed (backward).
template <typename T>
__device__ void block_laswp(const int *piv, int m, T *X, int ldx, int nc, bool forward) {
  for (int j = threadIdx.x; j < nc; j += blockDim.x) {
    T *x = X + (long long)j * ldx;
    if (forward) {
      for (int i = 0; i < m; ++i) {
        int p = piv[i] - 1;
        if (p != i) swap_vals(x[i], x[p]);
      }
    } else {
      for (int i = m - 1; i >= 0; --i) {
        int p = piv[i] - 1;
        if (p != i) swap_vals(x[i], x[p]);
      }
    }
  }
  __syncthreads();
}

// X := A^{-1} X (TRANS = false) or A^{-T} X (TRANS = true) for the LU
// factors LU (lda) and pivots piv of A, X an m x nc tile (ldx).  FAR (A^{-1}, factors
// in global memory): a lane's row of a diagonal block is loaded ahead into
// registers and a row's 32 factors of an update together, instead of one wait of
// the caches a step.
template <typename T, bool TRANS, bool FAR = false>
__device__ void block_getrs(const T *LU, int lda, const int *piv, int m, T *X, int ldx, int nc) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarp = nt >> 5;
  auto lu = [&](int i, int j) -> T { return LU[i + (long long)j * lda]; };
  if (!TRANS) {
    T d[FAR ? 32 : 1];
    auto load_diag = [&](int k0, int kb) {
#pragma unroll
      for (int k = 0; k < (FAR ? 32 : 0); ++k) d[k] = lane < kb && k < kb ? lu(k0 + lane, k0 + k) : T(0);
    };
    // x_i - sum over the block's rows k of A(i, k) x_k
    auto row_update = [&](T acc, int i, int k0, int kb, const T *x) {
      if (FAR) {
        T l[32];
#pragma unroll
        for (int kk = 0; kk < 32; ++kk) l[kk] = kk < kb ? lu(i, k0 + kk) : T(0);
#pragma unroll
        for (int kk = 0; kk < 32; ++kk)
          if (kk < kb) acc -= l[kk] * x[k0 + kk];
      } else {
        for (int kk = 0; kk < kb; ++kk) acc -= lu(i, k0 + kk) * x[k0 + kk];
      }
      return acc;
    };
    block_laswp(piv, m, X, ldx, nc, true);
    // L y = P b, L unit lower: 32-row blocks, forward
    for (int k0 = 0; k0 < m; k0 += 32) {
      const int kb = min(32, m - k0);
      if (FAR) {
        if (warp < nc) load_diag(k0, kb);
        for (int j = warp; j < nc; j += nwarp) {
          T *x = X + (long long)j * ldx + k0;
          T v = lane < kb ? x[lane] : T(0);
#pragma unroll
          for (int kk = 0; kk < 31; ++kk) {
            const T xk = __shfl_sync(0xffffffffu, v, kk);
            if (lane > kk && lane < kb) v -= d[kk] * xk;
          }
          if (lane < kb) x[lane] = v;
        }
      } else {
        for (int j = warp; j < nc; j += nwarp) {
          T *x = X + (long long)j * ldx + k0;
          T v = lane < kb ? x[lane] : T(0);
          for (int kk = 0; kk < kb - 1; ++kk) {
            T xk = __shfl_sync(0xffffffffu, v, kk);
            if (lane > kk && lane < kb) v -= lu(k0 + lane, k0 + kk) * xk;
          }
          if (lane < kb) x[lane] = v;
        }
      }
      __syncthreads();
      const int rows = m - k0 - kb;
      if (rows > 0) {
        for (int e = tid; e < rows * nc; e += nt) {
          const int i = k0 + kb + e % rows, j = e / rows;
          T *x = X + (long long)j * ldx;
          x[i] = row_update(x[i], i, k0, kb, x);
        }
      }
      __syncthreads();
    }
    // U x = y, U non-unit upper: 32-row blocks, backward
    for (int k1 = m; k1 > 0; k1 -= 32) {
      const int k0 = max(0, k1 - 32), kb = k1 - k0;
      if (FAR) {
        T u = T(1);  // the lane's pivot
        if (warp < nc) {
          load_diag(k0, kb);
          if (lane < kb) u = lu(k0 + lane, k0 + lane);
        }
        for (int j = warp; j < nc; j += nwarp) {
          T *x = X + (long long)j * ldx + k0;
          T v = lane < kb ? x[lane] : T(0);
#pragma unroll
          for (int kk = 31; kk >= 0; --kk) {
            if (kk >= kb) continue;
            if (lane == kk) v = v / u;
            const T xk = __shfl_sync(0xffffffffu, v, kk);
            if (lane < kk) v -= d[kk] * xk;
          }
          if (lane < kb) x[lane] = v;
        }
      } else {
        for (int j = warp; j < nc; j += nwarp) {
          T *x = X + (long long)j * ldx + k0;
          T v = lane < kb ? x[lane] : T(0);
          for (int kk = kb - 1; kk >= 0; --kk) {
            if (lane == kk) v = v / lu(k0 + kk, k0 + kk);
            T xk = __shfl_sync(0xffffffffu, v, kk);
            if (lane < kk) v -= lu(k0 + lane, k0 + kk) * xk;
          }
          if (lane < kb) x[lane] = v;
        }
      }
      __syncthreads();
      if (k0 > 0) {
        for (int e = tid; e < k0 * nc; e += nt) {
          const int i = e % k0, j = e / k0;
          T *x = X + (long long)j * ldx;
          x[i] = row_update(x[i], i, k0, kb, x);
        }
      }
      __syncthreads();
    }
  } else {
    // U^T y = b, U^T non-unit lower: forward
    for (int k0 = 0; k0 < m; k0 += 32) {
      const int kb = min(32, m - k0);
      for (int j = warp; j < nc; j += nwarp) {
        T *x = X + (long long)j * ldx + k0;
        T v = lane < kb ? x[lane] : T(0);
        for (int kk = 0; kk < kb; ++kk) {
          if (lane == kk) v = v / lu(k0 + kk, k0 + kk);
          T xk = __shfl_sync(0xffffffffu, v, kk);
          if (lane > kk && lane < kb) v -= lu(k0 + kk, k0 + lane) * xk;
        }
        if (lane < kb) x[lane] = v;
      }
      __syncthreads();
      const int rows = m - k0 - kb;
      if (rows > 0) {
        for (int e = tid; e < rows * nc; e += nt) {
          const int i = k0 + kb + e % rows, j = e / rows;
          T *x = X + (long long)j * ldx;
          T acc = x[i];
          for (int kk = 0; kk < kb; ++kk) acc -= lu(k0 + kk, i) * x[k0 + kk];
          x[i] = acc;
        }
      }
      __syncthreads();
    }
    // L^T z = y, L^T unit upper: backward
    for (int k1 = m; k1 > 0; k1 -= 32) {
      const int k0 = max(0, k1 - 32), kb = k1 - k0;
      for (int j = warp; j < nc; j += nwarp) {
        T *x = X + (long long)j * ldx + k0;
        T v = lane < kb ? x[lane] : T(0);
        for (int kk = kb - 1; kk > 0; --kk) {
          T xk = __shfl_sync(0xffffffffu, v, kk);
          if (lane < kk) v -= lu(k0 + kk, k0 + lane) * xk;
        }
        if (lane < kb) x[lane] = v;
      }
      __syncthreads();
      if (k0 > 0) {
        for (int e = tid; e < k0 * nc; e += nt) {
          const int i = e % k0, j = e / k0;
          T *x = X + (long long)j * ldx;
          T acc = x[i];
          for (int kk = 0; kk < kb; ++kk) acc -= lu(k0 + kk, i) * x[k0 + kk];
          x[i] = acc;
        }
      }
      __syncthreads();
    }
    block_laswp(piv, m, X, ldx, nc, false);
  }
}

}  // namespace hodlr
