// The inputs of a handle from device memory: one pass over each input writes
// the handle's FP64 copy and, in the mixed mode with the tensor-core residual,
// everything derived from it -- the digit slices and exponents of ozaki.cuh,
// and V in FP32 -- while the values are in registers.
//
// What bounds it: HBM.  At N = 2^20, leaf 128, 13 levels, rank 32 the copies
// alone took 7.3 ms by cudaMemcpy2DAsync (2.4 TB/s) and take 2.6 here; with the
// separate digit and conversion kernels, which read the copy again, a mixed
// handle's inputs took 17.1 ms and take 6.8 (32 GB in all).
#include <algorithm>

#include "kernels.cuh"
#include "ozaki.cuh"

namespace hodlr {

// dst = src, rows x cols, column-major; 16-byte accesses when VEC (bases and
// leading dimensions allow it).
template <bool VEC>
__global__ void __launch_bounds__(256) copy2d_kernel(const double *__restrict__ src, long long lds,
                                                     double *__restrict__ dst, long long ldd, long long rows, int cols) {
  constexpr int W = VEC ? 2 : 1, UN = 4;  // values a thread and step, steps in flight
  for (int j = blockIdx.y; j < cols; j += gridDim.y) {
    const double *s = src + (long long)j * lds;
    double *d = dst + (long long)j * ldd;
    for (long long i0 = ((long long)blockIdx.x * 256 * UN + threadIdx.x) * W; i0 < rows;
         i0 += (long long)gridDim.x * 256 * UN * W) {
      double2 v[UN];
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        const long long i = i0 + (long long)u * 256 * W;
        if (VEC && i + 1 < rows)
          v[u] = *reinterpret_cast<const double2 *>(s + i);
        else if (i < rows)
          v[u].x = s[i];
      }
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        const long long i = i0 + (long long)u * 256 * W;
        if (VEC && i + 1 < rows)
          *reinterpret_cast<double2 *>(d + i) = v[u];
        else if (i < rows)
          d[i] = v[u].x;
      }
    }
  }
}

cudaError_t launch_copy2d(const double *src, long long lds, double *dst, long long ldd, long long rows, int cols,
                          cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  if (lds == rows && ldd == rows) {  // one run of values
    rows *= cols;
    cols = 1;
  }
  const bool vec = !(((uintptr_t)src | (uintptr_t)dst) & 15) && (cols == 1 || !((lds | ldd) & 1));
  const long long per = vec ? 2048 : 1024;
  const int gy = std::min(cols, 65535);
  const long long gx = std::max<long long>(1, std::min<long long>((rows + per - 1) / per, (16LL * kNumSMs + gy - 1) / gy));
  const dim3 grid((unsigned)gx, (unsigned)gy);
  if (vec)
    HODLR_LAUNCH(copy2d_kernel<true>, grid, 256, 0, s, src, lds, dst, ldd, rows, cols);
  else
    HODLR_LAUNCH(copy2d_kernel<false>, grid, 256, 0, s, src, lds, dst, ldd, rows, cols);
  return cudaGetLastError();
}

// Rows of `cols` values (U of a level: cols = r; the leaf blocks: cols = m),
// row i's value q at src[(i / rpb) bstride + i % rpb + q ld]: the copy to
// dst[(i / rpb) dbstride + i % rpb + q ldd], the row's exponent, and its digits
// at out + i cols + q, slice s at + s sstride.  A CTA takes 64 rows through
// shared memory, so that both the loads (along the rows of a column) and the
// digit stores (along a row) are contiguous.
constexpr int kSetRows = 64;
__global__ void __launch_bounds__(256) set_rows_kernel(const double *__restrict__ src, long long rpb, long long bstride,
                                                       long long ld, double *__restrict__ dst, long long dbstride,
                                                       long long ldd, long long rows, int cols, __nv_bfloat16 *out,
                                                       long long sstride, int *exps) {
  extern __shared__ double tile[];  // [cols][kSetRows + 1]
  __shared__ unsigned long long smax[kSetRows];
  constexpr int LD = kSetRows + 1;
  const long long i0 = (long long)blockIdx.x * kSetRows;
  const int nr = (int)min((long long)kSetRows, rows - i0), tid = threadIdx.x, r = tid & (kSetRows - 1);
  if (tid < kSetRows) smax[tid] = 0;
  __syncthreads();
  if (r < nr) {
    const long long i = i0 + r, b = i / rpb, ii = i - b * rpb;
    const double *s = src + b * bstride + ii;
    double *d = dst + b * dbstride + ii;
    unsigned long long mb = 0;
#pragma unroll 8
    for (int q = tid / kSetRows; q < cols; q += 256 / kSetRows) {
      const double v = s[(long long)q * ld];
      d[(long long)q * ldd] = v;
      tile[q * LD + r] = v;
      mb = max(mb, abs_bits(v));
    }
    atomicMax(&smax[r], mb);
  }
  __syncthreads();
  const int nchunk = cols / 8;
  for (int t = tid; t < nr * nchunk; t += 256) {
    const int row = t / nchunk, c = t - row * nchunk, E = oz_exponent_bits(smax[row]);
    if (c == 0) exps[i0 + row] = E;
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = tile[(8 * c + u) * LD + row];
    uint4 d[kOzSlices];
    oz_digits8(v, E, d);
    __nv_bfloat16 *o = out + (i0 + row) * cols + 8 * c;
#pragma unroll
    for (int sl = 0; sl < kOzSlices; ++sl) *reinterpret_cast<uint4 *>(o + sl * sstride) = d[sl];
  }
}

cudaError_t launch_set_rows(const double *src, long long rpb, long long bstride, long long ld, double *dst,
                            long long dbstride, long long ldd, long long rows, int cols, __nv_bfloat16 *out,
                            long long sstride, int *exps, cudaStream_t s) {
  if (cols % 8 || (sstride % 8)) return cudaErrorNotSupported;
  const size_t bytes = sizeof(double) * cols * (kSetRows + 1);
  cudaError_t e = allow_dyn_smem(set_rows_kernel, bytes);
  if (e != cudaSuccess) return e;
  HODLR_LAUNCH(set_rows_kernel, ceil_div(rows, kSetRows), 256, bytes, s, src, rpb, bstride, ld, dst, dbstride, ldd, rows,
               cols, out, sstride, exps);
  return cudaGetLastError();
}

// V of a level: the copy, V in FP32, and the digits scaled per 64-row chunk of
// each column (column-major, chunk ch and column j's exponent at ch c + j).
// Eight lanes a chunk, eight rows each.
__global__ void __launch_bounds__(256) set_cols_kernel(const double *__restrict__ src, long long lds,
                                                       double *__restrict__ dst, float *__restrict__ dst32,
                                                       long long ldd, long long nchunk, int c, __nv_bfloat16 *out,
                                                       long long sstride, int *exps) {
  static_assert(kOzChunk == 64, "8 lanes x 8 rows per exponent group");
  const long long g = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int lane = threadIdx.x & 31, sub = lane & 7;
  if (g >= nchunk * c) return;  // whole 8-lane groups leave together
  const unsigned gmask = 0xffu << (lane & 24);
  const long long ch = g % nchunk;  // neighbouring groups: one column
  const int j = (int)(g / nchunk);
  const long long i0 = ch * kOzChunk + 8 * sub;
  double v[8];
  const double2 *xp = reinterpret_cast<const double2 *>(src + i0 + j * lds);
  double2 *op = reinterpret_cast<double2 *>(dst + i0 + j * ldd);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const double2 t = xp[u];
    v[2 * u] = t.x;
    v[2 * u + 1] = t.y;
    op[u] = t;
  }
  float4 *fp = reinterpret_cast<float4 *>(dst32 + i0 + j * ldd);
#pragma unroll
  for (int u = 0; u < 2; ++u)
    fp[u] = make_float4(f64_to_f32_rn(v[4 * u]), f64_to_f32_rn(v[4 * u + 1]), f64_to_f32_rn(v[4 * u + 2]),
                        f64_to_f32_rn(v[4 * u + 3]));
  unsigned long long mb = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) mb = max(mb, abs_bits(v[u]));
#pragma unroll
  for (int o = 4; o; o >>= 1) mb = max(mb, __shfl_xor_sync(gmask, mb, o));
  const int E = oz_exponent_bits(mb);
  if (sub == 0) exps[ch * c + j] = E;
  uint4 d[kOzSlices];
  oz_digits8(v, E, d);
  __nv_bfloat16 *o = out + j * ldd + i0;
#pragma unroll
  for (int sl = 0; sl < kOzSlices; ++sl) *reinterpret_cast<uint4 *>(o + sl * sstride) = d[sl];
}

cudaError_t launch_set_cols(const double *src, long long lds, double *dst, float *dst32, long long ldd, long long n,
                            int c, __nv_bfloat16 *out, long long sstride, int *exps, cudaStream_t s) {
  if (n % kOzChunk || (((uintptr_t)src | (uintptr_t)dst | (uintptr_t)dst32 | (uintptr_t)out) & 15) || lds % 2 ||
      ldd % 8 || sstride % 8)
    return cudaErrorNotSupported;
  HODLR_LAUNCH(set_cols_kernel, ceil_div(n / kOzChunk * c * 8, 256), 256, 0, s, src, lds, dst, dst32, ldd, n / kOzChunk, c,
               out, sstride, exps);
  return cudaGetLastError();
}

}  // namespace hodlr
