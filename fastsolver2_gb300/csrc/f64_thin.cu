// The FP64 steps of a solve for few right-hand sides (up to 8 columns), and the
// outer products of the gradients (inner dimension up to 4).
//
// With a handful of columns every value of U, V, the leaf inverses and the
// capacitance inverses is read once and used a few times: at one column a
// value's 8 bytes take 0.34 clocks of an SM's share of HBM and its FMA 0.48 of
// its FP64 pipe, so both count and none may be spent on padding (the tiled
// kernels these replace pad the columns to 32 or 64, and multiplied mostly
// zeros).  No shared-memory tiles of the matrices: each thread streams its row
// or its lanes' rows straight from memory, the few columns sit in shared memory
// or registers.  Measured at N = 2^18, leaf 128, rank 16: a solve for one
// column 14.5 -> 0.40 ms forward and 0.42 transposed (2.5 TB/s of factors; the
// upper levels are short launches), four columns 0.99, eight 1.84 (the FP64
// rate).  The updates and gradients of an adjoint step at N = 2^18, rank 24, one
// column: 22.0 -> 2.6 ms.
#include <algorithm>

#include "kernels.cuh"

namespace hodlr {

namespace {

// Sum of CNT (a power of two up to 32) values a lane over the 32 lanes; the
// lane keeps value `index`.  Halves the values while it halves the distance:
// CNT - 1 + log2(32 / CNT) additions instead of 5 CNT.
template <int CNT>
__device__ __forceinline__ double lanes_sum(double (&v)[CNT], int lane, int &index) {
  index = 0;
  int n = CNT;
#pragma unroll
  for (int off = 16; off; off >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = lane & off;
#pragma unroll
      for (int k = 0; k < CNT / 2; ++k)
        if (k < n) {
          const double keep = up ? v[k + n] : v[k], give = up ? v[k] : v[k + n];
          v[k] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
      if (up) index += n;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    }
  }
  return v[0];
}

constexpr int kBChunk = 64;  // inner values of B staged at a time

}  // namespace

// C_b += alpha A_b diag(scale) op(B_b), N <= NC columns, A not transposed: one
// thread a row.
template <int NC>
__global__ void __launch_bounds__(256) f64_thin_update_kernel(UpdateArgs a, int nrt) {
  if (a.skip && *a.skip) return;
  __shared__ double sB[kBChunk * NC];
  const int b = (int)(blockIdx.x / nrt), i = (int)(blockIdx.x % nrt) * blockDim.x + threadIdx.x;
  const double *A = static_cast<const double *>(a.A) + (long long)b * a.a_bstride + i;
  const double *B = a.B + (long long)(b >> 1) * a.b_s1 + (long long)((b & 1) ^ a.b_flip) * a.b_s2;
  double *C = static_cast<double *>(a.C) + (long long)b * a.c_bstride + i;
  const bool in = i < a.M;
  // two chains of sums a column: an FP64 FMA's result is a long time coming
  double acc[2][NC], c[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    acc[0][j] = acc[1][j] = 0.0;
    c[j] = in && j < a.N ? C[(long long)j * a.ldc] : 0.0;
  }
  for (int q0 = 0; q0 < a.K; q0 += kBChunk) {
    const int kb = min(kBChunk, a.K - q0);
    if (q0) __syncthreads();
    for (int e = threadIdx.x; e < kBChunk * NC; e += blockDim.x) {
      const int q = e / NC, j = e % NC;
      double v = 0.0;
      if (q < kb && j < a.N) {
        v = a.b_trans ? B[j + (long long)(q0 + q) * a.ldb] : B[(q0 + q) + (long long)j * a.ldb];
        if (a.scale) v *= a.scale_cols ? a.scale[j] : a.scale[q0 + q];
      }
      sB[e] = v;
    }
    __syncthreads();
    if (in) {
      const double *Aq = A + (long long)q0 * a.lda;
      int q = 0;
      for (; q + 8 <= kb; q += 8) {
        double x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = Aq[(long long)(q + e) * a.lda];
#pragma unroll
        for (int e = 0; e < 8; ++e)
#pragma unroll
          for (int j = 0; j < NC; ++j) acc[e & 1][j] = fma(x[e], sB[(q + e) * NC + j], acc[e & 1][j]);
      }
      for (; q < kb; ++q) {
        const double x = Aq[(long long)q * a.lda];
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[q & 1][j] = fma(x, sB[q * NC + j], acc[q & 1][j]);
      }
    }
  }
  if (!in) return;
#pragma unroll
  for (int j = 0; j < NC; ++j)
    if (j < a.N) C[(long long)j * a.ldc] = fma(a.alpha, acc[0][j] + acc[1][j], c[j]);
}

// The same for an inner dimension K <= KC and any number of columns: one thread
// a row and kOutCols columns, its K values of A in registers.
constexpr int kOutCols = 32;
template <int KC>
__global__ void __launch_bounds__(256) f64_thin_outer_kernel(UpdateArgs a, int nrt, int nct) {
  if (a.skip && *a.skip) return;
  __shared__ double sB[kOutCols * KC];
  long long u = blockIdx.x;
  const int j0 = (int)(u % nct) * kOutCols;
  u /= nct;
  const int i = (int)(u % nrt) * blockDim.x + threadIdx.x, b = (int)(u / nrt);
  const double *B = a.B + (long long)(b >> 1) * a.b_s1 + (long long)((b & 1) ^ a.b_flip) * a.b_s2;
  for (int e = threadIdx.x; e < kOutCols * KC; e += blockDim.x) {
    const int q = e % KC, j = j0 + e / KC;
    double v = 0.0;
    if (q < a.K && j < a.N) {
      v = a.b_trans ? B[j + (long long)q * a.ldb] : B[q + (long long)j * a.ldb];
      if (a.scale) v *= a.scale_cols ? a.scale[j] : a.scale[q];
    }
    sB[e] = v;
  }
  __syncthreads();
  if (i >= a.M) return;
  const double *A = static_cast<const double *>(a.A) + (long long)b * a.a_bstride + i;
  double *C = static_cast<double *>(a.C) + (long long)b * a.c_bstride + i + (long long)j0 * a.ldc;
  double x[KC];
#pragma unroll
  for (int q = 0; q < KC; ++q) x[q] = q < a.K ? A[(long long)q * a.lda] : 0.0;
  const int nj = min(kOutCols, a.N - j0);
  int j = 0;
  for (; j + 4 <= nj; j += 4) {
    double c[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) c[e] = a.overwrite ? 0.0 : C[(long long)(j + e) * a.ldc];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < KC; ++q) s = fma(x[q], sB[(j + e) * KC + q], s);
      C[(long long)(j + e) * a.ldc] = a.overwrite ? a.alpha * s : fma(a.alpha, s, c[e]);
    }
  }
  for (; j < nj; ++j) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < KC; ++q) s = fma(x[q], sB[j * KC + q], s);
    C[(long long)j * a.ldc] = a.overwrite ? a.alpha * s : fma(a.alpha, s, C[(long long)j * a.ldc]);
  }
}

// Out_b = A_b^T X_b for C <= NC columns: a CTA takes a chunk of rows, its warp w
// the ranks w, w + W, ... (RQ of them), a lane every 32nd row; the lanes are
// summed at the end.
template <int RQ, int NC, int W>
__global__ void __launch_bounds__(32 * W) f64_thin_reduce_kernel(const double *__restrict__ A, long long lda,
                                                                const double *__restrict__ X, long long ldx,
                                                                long long nrows, int r, int C, int chunk_rows,
                                                                int nchunks, double *out, const int *skip) {
  if (skip && *skip) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunk = (int)(blockIdx.x % nchunks);
  const long long b = blockIdx.x / nchunks, row0 = b * nrows + (long long)chunk * chunk_rows;
  const int rows = (int)min((long long)chunk_rows, nrows - (long long)chunk * chunk_rows);
  const double *Ab = A + row0, *Xb = X + row0;
  double acc[RQ * NC];
#pragma unroll
  for (int k = 0; k < RQ * NC; ++k) acc[k] = 0.0;
  constexpr int UN = RQ * NC <= 4 ? 4 : 2;
  for (int i0 = lane; i0 < rows; i0 += 32 * UN) {
    double av[UN][RQ], xv[UN][NC];
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const int i = i0 + 32 * u;
      const bool in = i < rows;
#pragma unroll
      for (int q = 0; q < RQ; ++q) av[u][q] = in && warp + W * q < r ? Ab[i + (long long)(warp + W * q) * lda] : 0.0;
#pragma unroll
      for (int j = 0; j < NC; ++j) xv[u][j] = in && j < C ? Xb[i + (long long)j * ldx] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < UN; ++u)
#pragma unroll
      for (int q = 0; q < RQ; ++q)
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[q * NC + j] = fma(av[u][q], xv[u][j], acc[q * NC + j]);
  }
  int k;
  const double s = lanes_sum<RQ * NC>(acc, lane, k);
  constexpr int kSame = 32 / (RQ * NC);  // lanes left with the same value
  const int q = warp + W * (k / NC), j = k % NC;
  if ((lane & (kSame - 1)) == 0 && q < r && j < C) out[(long long)blockIdx.x * r * C + q + (long long)j * r] = s;
}

// X_i := op(Dinv_i) X_i in place for C <= NC columns, leaves of m = 64, 128 or
// 256 rows: one CTA a leaf, thread t the row t % m and the inner indices
// congruent to t / m.  The transposed inverse passes through shared memory 32
// of its rows at a time.
template <int NC, bool TRANS>
__global__ void __launch_bounds__(256) f64_thin_leaf_kernel(const double *__restrict__ Dinv, int m, double *X,
                                                            long long ldx, int C, const int *skip) {
  if (skip && *skip) return;
  extern __shared__ double sm[];
  double *sX = sm;              // [m][NC]
  double *sP = sm + m * NC;     // partial sums [groups][m][NC], or the staged rows [32][m + 1]
  const int leaf = blockIdx.x, tid = threadIdx.x, i = tid % m, g = tid / m, G = 256 / m;
  const double *A = Dinv + (long long)leaf * m * m;
  double *Xg = X + (long long)leaf * m;
  for (int e = tid; e < m * NC; e += 256) {
    const int k = e % m, j = e / m;
    sX[k * NC + j] = j < C ? Xg[k + (long long)j * ldx] : 0.0;
  }
  __syncthreads();
  double acc[2][NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) acc[0][j] = acc[1][j] = 0.0;
  if (!TRANS) {
    for (int k0 = g; k0 < m; k0 += 8 * G) {
      double x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = A[i + (long long)(k0 + e * G) * m];
#pragma unroll
      for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[e & 1][j] = fma(x[e], sX[(k0 + e * G) * NC + j], acc[e & 1][j]);
    }
  } else {
    const int warp = tid >> 5, lane = tid & 31;
    for (int k0 = 0; k0 < m; k0 += 32) {
      for (int c = warp; c < m; c += 8) sP[lane * (m + 1) + c] = A[k0 + lane + (long long)c * m];
      __syncthreads();
      for (int k = g; k < 32; k += 2 * G)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int j = 0; j < NC; ++j)
            acc[e][j] = fma(sP[(k + e * G) * (m + 1) + i], sX[(k0 + k + e * G) * NC + j], acc[e][j]);
      __syncthreads();
    }
  }
#pragma unroll
  for (int j = 0; j < NC; ++j) sP[(g * m + i) * NC + j] = acc[0][j] + acc[1][j];
  __syncthreads();
  for (int e = tid; e < m * NC; e += 256) {
    const int k = e % m, j = e / m;
    if (j >= C) continue;
    double s = sP[k * NC + j];
    for (int q = 1; q < G; ++q) s += sP[(q * m + k) * NC + j];
    Xg[k + (long long)j * ldx] = s;
  }
}

// eta_p = op(Sinv_p) RHS_p for C <= NC columns (cap_apply_kernel's contract,
// FP64): one CTA a node, NP rows (2r padded), the inner index split over the
// 256 / NP groups.
template <int NP, int NC>
__global__ void __launch_bounds__(256) f64_thin_cap_kernel(CapApplyArgs a) {
  if (a.skip && *a.skip) return;
  constexpr int G = 256 / NP;
  __shared__ double sR[NP * NC], sP[G][NP * NC];
  const int r = a.r, n2 = 2 * r, p = blockIdx.x, tid = threadIdx.x, i = tid % NP, g = tid / NP;
  const double *S = a.sinv + (long long)(a.node_base + p) * n2 * n2;
  const double *T0 = a.Tb + (long long)(2 * p) * a.tb_stride, *T1 = a.Tb + (long long)(2 * p + 1) * a.tb_stride;
  for (int e = tid; e < NP * NC; e += 256) {
    const int q = e % NP, j = e / NP;
    double v = 0.0;
    if (q < n2 && j < a.C) {
      const bool first = q < r;
      const int qq = first ? q : q - r;
      if (!a.trans)
        v = (a.scale ? a.scale[qq] : 1.0) * (first ? T1 : T0)[qq + (long long)j * r];
      else
        v = (first ? T0 : T1)[qq + (long long)j * r];
    }
    sR[q * NC + j] = v;
  }
  __syncthreads();
  double acc[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) acc[j] = 0.0;
  if (i < n2)
#pragma unroll 4
    for (int q = g; q < n2; q += G) {
      const double s = a.trans ? S[q + (long long)i * n2] : S[i + (long long)q * n2];
#pragma unroll
      for (int j = 0; j < NC; ++j) acc[j] = fma(s, sR[q * NC + j], acc[j]);
    }
#pragma unroll
  for (int j = 0; j < NC; ++j) sP[g][i * NC + j] = acc[j];
  __syncthreads();
  for (int e = tid; e < NP * NC; e += 256) {
    const int k = e % NP, j = e / NP;
    if (k >= n2 || j >= a.C) continue;
    double s = sP[0][k * NC + j];
#pragma unroll
    for (int q = 1; q < G; ++q) s += sP[q][k * NC + j];
    const long long o = (long long)p * n2 * a.C + k + (long long)j * n2;
    if (a.eta32)
      a.eta32[o] = (float)(a.out_scale ? s * a.out_scale[k % r] : s);
    else
      a.eta[o] = s;
  }
}

cudaError_t launch_f64_thin_update(const UpdateArgs &a, cudaStream_t s) {
  const int bt = std::min(256, (a.M + 31) / 32 * 32), nrt = ceil_div(a.M, bt);
  const unsigned grid = (unsigned)((long long)nrt * a.nbatch);
  if (a.N == 1) HODLR_LAUNCH(f64_thin_update_kernel<1>, grid, bt, 0, s, a, nrt);
  else if (a.N == 2) HODLR_LAUNCH(f64_thin_update_kernel<2>, grid, bt, 0, s, a, nrt);
  else if (a.N <= 4) HODLR_LAUNCH(f64_thin_update_kernel<4>, grid, bt, 0, s, a, nrt);
  else HODLR_LAUNCH(f64_thin_update_kernel<8>, grid, bt, 0, s, a, nrt);
  return cudaGetLastError();
}

cudaError_t launch_f64_thin_outer(const UpdateArgs &a, cudaStream_t s) {
  const int bt = std::min(256, (a.M + 31) / 32 * 32), nrt = ceil_div(a.M, bt), nct = ceil_div(a.N, kOutCols);
  const unsigned grid = (unsigned)((long long)nrt * nct * a.nbatch);
  if (a.K == 1) HODLR_LAUNCH(f64_thin_outer_kernel<1>, grid, bt, 0, s, a, nrt, nct);
  else if (a.K == 2) HODLR_LAUNCH(f64_thin_outer_kernel<2>, grid, bt, 0, s, a, nrt, nct);
  else HODLR_LAUNCH(f64_thin_outer_kernel<4>, grid, bt, 0, s, a, nrt, nct);
  return cudaGetLastError();
}

template <int NC>
static cudaError_t thin_reduce_nc(const double *A, long long lda, const double *X, long long ldx, long long nrows,
                                  int nbatch, int r, int C, int chunk_rows, int nchunks, double *dst, const int *skip,
                                  cudaStream_t s) {
  const unsigned grid = (unsigned)((long long)nbatch * nchunks);
#define HODLR_THIN_RED(RQ, W)                                                                                       \
  HODLR_LAUNCH((f64_thin_reduce_kernel<RQ, NC, W>), grid, 32 * W, 0, s, A, lda, X, ldx, nrows, r, C, chunk_rows,    \
               nchunks, dst, skip)
  if (r <= 8) HODLR_THIN_RED(1, 8);
  else if (r <= 16) HODLR_THIN_RED(2, 8);
  else if (r <= 32) HODLR_THIN_RED(4, 8);
  else HODLR_THIN_RED(4, 16);
#undef HODLR_THIN_RED
  return cudaGetLastError();
}

cudaError_t launch_f64_thin_reduce(const double *A, long long lda, const double *X, long long ldx, long long nrows,
                                   int nbatch, int r, int C, int chunk_rows, int nchunks, double *dst, const int *skip,
                                   cudaStream_t s) {
  if (C == 1) return thin_reduce_nc<1>(A, lda, X, ldx, nrows, nbatch, r, C, chunk_rows, nchunks, dst, skip, s);
  if (C == 2) return thin_reduce_nc<2>(A, lda, X, ldx, nrows, nbatch, r, C, chunk_rows, nchunks, dst, skip, s);
  if (C <= 4) return thin_reduce_nc<4>(A, lda, X, ldx, nrows, nbatch, r, C, chunk_rows, nchunks, dst, skip, s);
  return thin_reduce_nc<8>(A, lda, X, ldx, nrows, nbatch, r, C, chunk_rows, nchunks, dst, skip, s);
}

template <int NC>
static cudaError_t thin_leaf_nc(const double *Dinv, int m, int nleaf, double *X, long long ldx, int C, bool trans,
                                const int *skip, cudaStream_t s) {
  const size_t bytes = sizeof(double) * ((size_t)m * NC + std::max<size_t>((size_t)256 * NC, trans ? 32 * (m + 1) : 0));
  cudaError_t e;
  if (trans) {
    auto k = f64_thin_leaf_kernel<NC, true>;
    if ((e = allow_dyn_smem(k, bytes)) != cudaSuccess) return e;
    HODLR_LAUNCH(k, nleaf, 256, bytes, s, Dinv, m, X, ldx, C, skip);
  } else {
    auto k = f64_thin_leaf_kernel<NC, false>;
    if ((e = allow_dyn_smem(k, bytes)) != cudaSuccess) return e;
    HODLR_LAUNCH(k, nleaf, 256, bytes, s, Dinv, m, X, ldx, C, skip);
  }
  return cudaGetLastError();
}

cudaError_t launch_f64_thin_leaf(const double *Dinv, int m, int nleaf, double *X, long long ldx, int C, bool trans,
                                 const int *skip, cudaStream_t s) {
  if (C == 1) return thin_leaf_nc<1>(Dinv, m, nleaf, X, ldx, C, trans, skip, s);
  if (C == 2) return thin_leaf_nc<2>(Dinv, m, nleaf, X, ldx, C, trans, skip, s);
  if (C <= 4) return thin_leaf_nc<4>(Dinv, m, nleaf, X, ldx, C, trans, skip, s);
  return thin_leaf_nc<8>(Dinv, m, nleaf, X, ldx, C, trans, skip, s);
}

template <int NC> static cudaError_t thin_cap_nc(const CapApplyArgs &a, cudaStream_t s) {
  const int n2 = 2 * a.r;
  if (n2 <= 32) HODLR_LAUNCH((f64_thin_cap_kernel<32, NC>), a.nnode, 256, 0, s, a);
  else if (n2 <= 64) HODLR_LAUNCH((f64_thin_cap_kernel<64, NC>), a.nnode, 256, 0, s, a);
  else HODLR_LAUNCH((f64_thin_cap_kernel<128, NC>), a.nnode, 256, 0, s, a);
  return cudaGetLastError();
}

cudaError_t launch_f64_thin_cap(const CapApplyArgs &a, cudaStream_t s) {
  if (a.C == 1) return thin_cap_nc<1>(a, s);
  if (a.C == 2) return thin_cap_nc<2>(a, s);
  if (a.C <= 4) return thin_cap_nc<4>(a, s);
  return thin_cap_nc<8>(a, s);
}

}  // namespace hodlr
