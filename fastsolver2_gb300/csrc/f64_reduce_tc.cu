// K3 in FP64 on the tcgen05 tensor cores: Out_b = V_b^T X_b (r x C per child
// block, the block's rows summed) with exact digit products (f64_tc.cuh).
//
// The columns of X are the product's rows (128 a tile) and the ranks of V its
// columns (32 a tile), so that the long row dimension of both operands, which
// is contiguous in memory, is the inner one.  It is taken in groups of 64
// rows: each X column and each V column has one scale a group, the group's
// products run as two chunks of 32, and the group's exact sums are rounded to
// FP64 and added to FP64 sums in registers.  Rows are balanced (f64_tc.cuh) by
// the largest entry of V's row.
//
// What bounds it: X is read once, 64 KB a group of 128 columns (2800 clocks of
// an SM's share of HBM), the products take 2900 clocks of the tensor pipe; but
// cutting a value into digits takes some 40 instructions, most of them on the
// integer pipe, which issues at half rate, and turning the sums into FP64 some
// 40 an output: 12400 clocks a group measured, the integer pipe two thirds busy.
// The outputs are rounded on the FP64 pipe (dig_double), which has little else to
// do here; with the integer packing of dig_value, 60 instructions an output, and
// the balance held in registers a group took 15000 clocks.  64
// rows a group because the output side is paid once a group (at 32 rows it
// would cost as much as the digits), and because 128 would take both of the
// 57 KB plane buffers that let one half's products overlap the other half's
// digits.  X's values stay in registers from their load to their digits, and a
// half's registers are loaded for the next group as soon as they are cut (a
// first version that loaded the values twice, with eight warps, took 40.3 ms, this
// order 37.0 at first and now 31: the reductions of one factor + solve at N = 2^20,
// leaf 128, rank 32, 64 right-hand sides.  The FP64 FMA kernel took 229.)
#include <algorithm>

#include "f64_tc.cuh"
#include "kernels.cuh"

namespace hodlr {

namespace {

constexpr int kXW = 16, kVW = 4, kEW = 8;  // warps cutting X, cutting V, epilogue
constexpr int kMmaWarp = kXW + kVW + kEW, kThreads = 32 * (kMmaWarp + 1);
constexpr int kGroup = 64;  // rows a group
constexpr long long kWait = 2000000000LL;  // about one second of SM clocks

__device__ WaitFault g_wait_fault = {-1, -1, 0};

struct RedArgs {
  const double *V, *X;
  long long ldv, ldx, nrows;
  int r, C, chunk_rows, nchunks, nct, nrt;
  long long units;  // blocks x chunks x column tiles x rank tiles
  double *out;      // [block][chunk] r x C
  const int *skip;
  DevStatus *st;
};

struct Shared {
  uint64_t x_full[2], x_empty[2], v_full[2], v_empty[2], bal_full[2], acc_full[2], acc_free[2], drain;
  int xs[4][128], vs[4][kDigN];  // the scales of the last groups
  alignas(16) unsigned rowmax[4][kGroup];    // largest |V| of each row (high words) of the last groups
  long long budget;  // of the wait the hook lets run out, in SM clocks
  int skip;          // test hook: the stage whose digits are never announced (-1: none)
  unsigned tmem;
  int marked;    // a result is a NaN
  RedArgs args;  // for sum_marked (the address of a kernel's parameter costs registers)
  int abort;
};
constexpr size_t kSmem = (size_t)2 * kDigABytes + (size_t)4 * kDigBBytes + sizeof(Shared) + 1024;

struct Unit {
  long long row0, blk;  // first row; index of the r x C result
  int rows, c0, q0, groups;
};
__device__ __forceinline__ Unit unit_of(const RedArgs &a, long long u) {
  Unit w;
  w.q0 = (int)(u % a.nrt) * kDigN;
  u /= a.nrt;
  w.c0 = (int)(u % a.nct) * 128;
  u /= a.nct;
  w.blk = u;
  const int chunk = (int)(u % a.nchunks);
  const long long b = u / a.nchunks, r0 = (long long)chunk * a.chunk_rows;
  w.row0 = b * a.nrows + r0;
  w.rows = (int)min((long long)a.chunk_rows, a.nrows - r0);
  w.groups = (w.rows + kGroup - 1) / kGroup;
  return w;
}

// The results of a CTA's units that are NaN -- an infinity or NaN among their values
// -- again by FMAs: all threads, after the units.
__device__ __noinline__ void sum_marked(const RedArgs &a) {
  for (long long u = blockIdx.x; u < a.units; u += gridDim.x) {
    const Unit w = unit_of(a, u);
    const int nc = min(128, a.C - w.c0), nq = min(kDigN, a.r - w.q0);
    double *out = a.out + w.blk * a.r * a.C + (long long)w.c0 * a.r + w.q0;
    const double *V = a.V + w.row0 + (long long)w.q0 * a.ldv, *X = a.X + w.row0 + (long long)w.c0 * a.ldx;
    for (int e = threadIdx.x; e < nc * nq; e += kThreads) {
      const int q = e % nq, c = e / nq;
      double *o = out + q + (long long)c * a.r;
      if (!isnan(*o)) continue;
      double s = 0.0;
      for (int i = 0; i < w.rows; ++i) s = fma(V[i + q * a.ldv], X[i + c * a.ldx], s);
      *o = s;
    }
  }
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 1) f64_reduce_tc_kernel(RedArgs a) {
  if (a.skip && *a.skip) return;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *px =
      reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *pv = px + 2 * kDigABytes;
  Shared *sh = reinterpret_cast<Shared *>(pv + 4 * kDigBBytes);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int q = 0; q < 2; ++q) {
      mbar_init(&sh->x_full[q], 32 * kXW);
      mbar_init(&sh->x_empty[q], 1);
      mbar_init(&sh->v_full[q], 32 * kVW);
      mbar_init(&sh->v_empty[q], 1);
      mbar_init(&sh->bal_full[q], 32 * kVW);
      mbar_init(&sh->acc_full[q], 2);  // the products' completion, and a plain arrival that publishes the scales
      mbar_init(&sh->acc_free[q], 32 * kEW);
    }
    mbar_init(&sh->drain, 1);
    const WaitFault wf = g_wait_fault;
    const bool hit = wf.cta == (int)blockIdx.x;
    sh->skip = hit ? wf.stage : -1;
    sh->budget = hit && wf.budget > 0 ? wf.budget : kWait;
    sh->abort = sh->marked = 0;
    sh->args = a;
    mbar_fence_init();
  }
  for (int e = tid; e < 4 * kGroup; e += kThreads) sh->rowmax[0][e] = 0;
  if (warp == kMmaWarp) {
    tc_alloc(&sh->tmem, 2 * kDigAccCols);
    tc_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = sh->tmem;
  auto wait = [&](uint64_t *bar, unsigned parity) { return mbar_wait_or_abort(bar, parity, &sh->abort, kWait); };
  auto wwait = [&](uint64_t *bar, unsigned parity) { return __all_sync(0xffffffffu, wait(bar, parity)); };
  // lanes of a slicer warp: column lane / 8 of four, rows 4 (lane % 8) .. + 3 of each half of the group
  const int lc = lane >> 3, lr = 4 * (lane & 7);
  int g = 0;  // groups this CTA has passed
  // the balance of four rows of a half of group g (read again for the digits: eight
  // registers less to hold)
  auto balance = [&](int g, int h, int *bal) {
    const uint4 m = *reinterpret_cast<const uint4 *>(&sh->rowmax[g & 3][32 * h + lr]);
    bal[0] = (int)(m.x >> 20);
    bal[1] = (int)(m.y >> 20);
    bal[2] = (int)(m.z >> 20);
    bal[3] = (int)(m.w >> 20);
  };
  bool ok = true;

  if (warp < kXW) {
    // ------------------------------------------------------------ X digits
    // two columns, 64 apart, a lane; a half's values are loaded for the next
    // group as soon as its digits are out
    double x[2][8];
    auto load = [&](const Unit &w, int gi, int h) {
      const int left = w.rows - gi * kGroup - lr - 32 * h;  // rows from the lane's first on
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int c = w.c0 + 4 * warp + lc + 64 * p;
        const double *Xc = a.X + w.row0 + (long long)gi * kGroup + lr + 32 * h + (long long)c * a.ldx;
#pragma unroll
        for (int e = 0; e < 4; ++e) x[p][4 * h + e] = c < a.C && e < left ? Xc[e] : 0.0;
      }
    };
    long long u = blockIdx.x;
    Unit w = unit_of(a, u);
    int gi = 0;
    load(w, 0, 0);
    load(w, 0, 1);
    while (u < a.units) {
      int key[2] = {kDigZero, kDigZero};
      unsigned mxs[2] = {0, 0};
      if (!wwait(&sh->bal_full[g & 1], (unsigned)((g >> 1) & 1))) break;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        int bal[4];
        balance(g, h, bal);
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const unsigned a = dig_ahi(x[p][4 * h + e]);
            dig_key(key[p], a, bal[e]);
            mxs[p] = max(mxs[p], a);
          }
      }
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        unsigned mx = mxs[p];
#pragma unroll
        for (int s = 1; s < 8; s <<= 1) {
          key[p] = max(key[p], __shfl_xor_sync(0xffffffffu, key[p], s));
          mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, s));
        }
        if ((lane & 7) == 0) sh->xs[g & 3][4 * warp + lc + 64 * p] = dig_scale(key[p], mx, kDigZeroB);
      }
      if (++gi == w.groups) {  // the group to load next
        gi = 0;
        u += gridDim.x;
        if (u < a.units) w = unit_of(a, u);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (g > 0 && !wwait(&sh->x_empty[h], (unsigned)((g - 1) & 1))) ok = false;
        if (!ok) break;
        int bal[4];
        balance(g, h, bal);
#pragma unroll
        for (int p = 0; p < 2; ++p)
          dig_put4(px + h * kDigABytes, kDigAPlane, swz64(4 * warp + lc + 64 * p, lr >> 3) + 2 * (lr & 7), x[p] + 4 * h,
                   [&](int e) { return bal[e]; }, key[p]);
        fence_proxy_async_smem();
        mbar_arrive(&sh->x_full[h]);
        if (u < a.units) load(w, gi, h);
      }
      if (!ok) break;
      ++g;
    }
  } else if (warp < kXW + kVW) {
    // ------------------------------------------------------------ V digits
    const int vw = warp - kXW;
    for (long long u = blockIdx.x; ok && u < a.units; u += gridDim.x) {
      const Unit w = unit_of(a, u);
      for (int gi = 0; gi < w.groups; ++gi, ++g) {
        const int left = w.rows - gi * kGroup, slot = g & 1;
        const double *Vg = a.V + w.row0 + (long long)gi * kGroup + lr + (long long)(w.q0 + 4 * vw + lc) * a.ldv;
        double x[2][8];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const bool in = w.q0 + 4 * vw + lc + 16 * p < a.r;
          const double *Vc = Vg + (long long)(16 * p) * a.ldv;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int i = 32 * (e >> 2) + (e & 3);
            x[p][e] = in && lr + i < left ? Vc[i] : 0.0;
          }
        }
        // group g - 2 is done with its planes, scales and row maxima
        if (g >= 2 && !wwait(&sh->v_empty[slot], (unsigned)(((g >> 1) - 1) & 1))) {
          ok = false;
          break;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          unsigned m = max(dig_finite(dig_ahi(x[0][e])), dig_finite(dig_ahi(x[1][e])));
          m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
          m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
          if (lc == 0) atomicMax(&sh->rowmax[g & 3][32 * (e >> 2) + lr + (e & 3)], m);
        }
        if (vw == 0) {  // the slot of group g + 2, last read for group g - 2
          sh->rowmax[(g + 2) & 3][2 * lane] = 0;
          sh->rowmax[(g + 2) & 3][2 * lane + 1] = 0;
        }
        mbar_arrive(&sh->bal_full[slot]);
        if (!wwait(&sh->bal_full[g & 1], (unsigned)((g >> 1) & 1))) {
          ok = false;
          break;
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          int key = kDigZero;
          unsigned mx = 0;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            int bal[4];
            balance(g, h, bal);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const unsigned b = dig_ahi(x[p][4 * h + e]);
              dig_key(key, b, -bal[e]);
              mx = max(mx, b);
            }
          }
#pragma unroll
          for (int s = 1; s < 8; s <<= 1) {
            key = max(key, __shfl_xor_sync(0xffffffffu, key, s));
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, s));
          }
          const int col = 4 * vw + lc + 16 * p;
          if ((lane & 7) == 0) sh->vs[g & 3][col] = dig_scale(key, mx, kDigZeroA);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            int bal[4];
            balance(g, h, bal);
            dig_put4(pv + (2 * slot + h) * kDigBBytes, kDigBPlane, swz64(col, lr >> 3) + 2 * (lr & 7), x[p] + 4 * h,
                     [&](int e) { return -bal[e]; }, key);
          }
        }
        fence_proxy_async_smem();
        if (g != sh->skip) mbar_arrive(&sh->v_full[slot]);
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ products
    if (lane == 0) {
      for (long long u = blockIdx.x; ok && u < a.units; u += gridDim.x) {
        const Unit w = unit_of(a, u);
        for (int gi = 0; ok && gi < w.groups; ++gi, ++g) {
          const int slot = g & 1;
          if (!mbar_wait_or_abort(&sh->v_full[slot], (unsigned)((g >> 1) & 1), &sh->abort, &sh->budget) ||
              (g >= 2 && !wait(&sh->acc_free[slot], (unsigned)(((g >> 1) - 1) & 1)))) {
            ok = false;
            break;
          }
          for (int h = 0; h < 2; ++h) {
            if (!wait(&sh->x_full[h], (unsigned)(g & 1))) {
              ok = false;
              break;
            }
            tc_fence_after();
            dig_mma_chunk(tmem + (unsigned)slot * kDigAccCols, smem_u32(px + h * kDigABytes),
                          smem_u32(pv + (2 * slot + h) * kDigBBytes), 2, h == 0);
            tc_commit(&sh->x_empty[h]);
          }
          if (!ok) break;
          tc_commit(&sh->acc_full[slot]);
          mbar_arrive(&sh->acc_full[slot]);
          tc_commit(&sh->v_empty[slot]);
        }
      }
      tc_commit(&sh->drain);  // completes once every product issued above has
      const long long w0 = clock64();
      while (!mbar_try_wait(&sh->drain, 0) && clock64() - w0 < kWait) {
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3, h = (warp - kXW - kVW) >> 2, row = 32 * q + lane;  // a column of X, 16 ranks
    for (long long u = blockIdx.x; ok && u < a.units; u += gridDim.x) {
      const Unit w = unit_of(a, u);
      double acc[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) acc[c] = 0.0;
      for (int gi = 0; gi < w.groups; ++gi, ++g) {
        const int slot = g & 1;
        if (!wwait(&sh->acc_full[slot], (unsigned)((g >> 1) & 1))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const int ex = sh->xs[g & 3][row];
        const unsigned tl = tmem + ((unsigned)(32 * q) << 16) + (unsigned)slot * kDigAccCols + 16 * h;
#pragma unroll
        for (int c2 = 0; c2 < 16; c2 += 2) {
          unsigned v[kDiag][2];
#pragma unroll
          for (int d = 0; d < kDiag; ++d) tc_ld2(tl + (unsigned)(d * kDigN + c2), v[d]);
          tc_wait_ld(v);
          const int *ev = sh->vs[g & 3] + 16 * h + c2;
          bool odd = false;
          double y[2], f[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            y[c] = dig_double(dig_combine<64>(v, c));
            f[c] = dig_power(ex + ev[c], odd);
          }
          if (odd)
            for (int c = 0; c < 2; ++c) {
              y[c] = dig_value_any(dig_combine<64>(v, c), ex + ev[c]);
              f[c] = 1.0;
            }
          acc[c2] = fma(f[0], y[0], acc[c2]);
          acc[c2 + 1] = fma(f[1], y[1], acc[c2 + 1]);
        }
        tc_fence_before();
        mbar_arrive(&sh->acc_free[slot]);
      }
      if (ok && w.c0 + row < a.C) {
        double *o = a.out + w.blk * a.r * a.C + (long long)(w.c0 + row) * a.r + w.q0 + 16 * h;
#pragma unroll
        for (int c = 0; c < 16; ++c)
          if (w.q0 + 16 * h + c < a.r) {
            o[c] = acc[c];
            if (isnan(acc[c])) sh->marked = 1;
          }
      }
    }
  }
  __syncthreads();
  if (tid == 0 && sh->abort) report_error(a.st, HODLR_ERR_TIMEOUT, blockIdx.x);
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tc_dealloc(tmem, 2 * kDigAccCols);
  }
  if (sh->marked && !sh->abort) sum_marked(sh->args);
}

// Row chunks per block: of the counts that fill one, two, .. `per_sm` waves of
// units over the SMs, the one whose waves take the fewest groups; at most
// `most` (an FP64 partial sum a chunk, added in a fixed order by the second
// pass).
void f64_reduce_tc_plan(long long nrows, int nbatch, int r, int C, int per_sm, int most, int &nchunks,
                        int &chunk_rows) {
  const long long base = (long long)nbatch * ceil_div(C, 128) * ceil_div(r, kDigN);
  long long best = -1;
  for (int w = 0; w <= per_sm; ++w) {
    const long long n = std::max<long long>(1, std::min<long long>(most, (long long)w * kNumSMs / base));
    const long long groups = ((nrows + n - 1) / n + kGroup - 1) / kGroup, rows = groups * kGroup;
    const long long m = (nrows + rows - 1) / rows;
    // the groups of the longest SM, with a unit's start and the second pass worth about one each
    const long long cost = ((base * m + kNumSMs - 1) / kNumSMs) * (groups + 1) + (m > 1 ? 1 : 0);
    if (best >= 0 && cost >= best) continue;
    best = cost;
    nchunks = (int)m;
    chunk_rows = (int)std::min<long long>(rows, nrows);
  }
}

cudaError_t f64_reduce_tc_set_wait_fault(const WaitFault &wf) {
  return cudaMemcpyToSymbol(g_wait_fault, &wf, sizeof wf);
}

bool f64_reduce_tc_try(const double *V, long long ldv, const double *X, long long ldx, long long nrows, int nbatch,
                       int r, int C, int chunk_rows, int nchunks, double *dst, const int *skip, DevStatus *st,
                       cudaStream_t s, cudaError_t &err) {
  RedArgs a;
  a.V = V;
  a.X = X;
  a.ldv = ldv;
  a.ldx = ldx;
  a.nrows = nrows;
  a.r = r;
  a.C = C;
  a.chunk_rows = chunk_rows;
  a.nchunks = nchunks;
  a.nct = ceil_div(C, 128);
  a.nrt = ceil_div(r, kDigN);
  a.units = (long long)nbatch * nchunks * a.nct * a.nrt;
  a.out = dst;
  a.skip = skip;
  a.st = st;
  note_waiting_launch();
  err = allow_dyn_smem(f64_reduce_tc_kernel, kSmem);
  if (err != cudaSuccess) return true;
  HODLR_LAUNCH(f64_reduce_tc_kernel, (unsigned)std::min<long long>(a.units, kNumSMs), kThreads, kSmem, s, a);
  err = cudaGetLastError();
  return true;
}

}  // namespace hodlr
