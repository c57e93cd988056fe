// K5 in FP64 on the tcgen05 tensor cores: C_b += alpha A_b diag(scale) op(B_b)
// with exact digit products (f64_tc.cuh), inner dimension up to 64.
//
// What bounds it: C is read and written once (64 KB per 128 x 32 tile, 2800
// clocks of an SM's share of HBM); the digit products take 1600 clocks of the
// tensor pipe and the one FP64 instruction left per value, the fused
// multiply-add into C, 1950, since GB300's FP64 pipe takes half a lane per
// clock and sub-partition.  The roles overlap: eight warps cut the A tile of
// 128 rows (once for all its column tiles) and the B tiles of 32 columns into
// digit planes, one thread issues the products into one of two accumulator
// sets (8 x 32 tensor-memory columns each), and sixteen epilogue warps turn
// the other set into FP64, add it to the C values they loaded a tile earlier
// and store.  Every CTA walks one contiguous range of tiles, so the SMs end
// together and the A tile is cut again only at a new row tile.  Everything is
// loaded with plain loads: any size, alignment and leading dimension.
//
// Measured (2^19 rows, inner 32): 5600 clocks a tile at 384 columns (3.6 TB/s
// of C and A), 6000 at 192, 8200 at 64 and 12300 at 32, where cutting the A
// tile is not hidden; the issue slots of the epilogue (some 60 instructions a
// value) are what is left.  At N = 2^20, leaf 128, rank 32, 64 right-hand
// sides the updates of one factor + solve take 18.6 ms; the FP64 FMA kernel
// (update_nn_kernel) took 196.
#include <algorithm>

#include "f64_tc.cuh"
#include "kernels.cuh"

namespace hodlr {

namespace {

constexpr int kSlicers = 256, kEpi = 512, kThreads = kSlicers + kEpi + 32;
constexpr int kEpiCols = kDigN * 128 / kEpi;  // columns of an epilogue thread
constexpr int kMmaWarp = (kSlicers + kEpi) / 32;
constexpr long long kWait = 2000000000LL;  // about one second of SM clocks

__device__ WaitFault g_wait_fault = {-1, -1, 0};

struct Shared {
  uint64_t a_full[2], a_empty[2], b_full[2], b_empty[2], acc_full[2], acc_free[2], slicers, drain;
  int ea[4][128], eb[8][kDigN];  // the scales of the last row tiles and tiles, read by the epilogue
  unsigned colw[2][4][64];       // largest |A(., k)| of each 32 rows of the last row tiles (high words)
  int key2[2][2][128];           // each half's key and largest of a row, of the last row tiles
  unsigned mx2[2][2][128];
  long long budget;  // of the wait the hook lets run out, in SM clocks
  int skip;          // test hook: the stage whose digits are never announced (-1: none)
  unsigned tmem;
  int marked;       // a group with an infinity or a NaN was met
  UpdateArgs args;  // for add_marked (the address of a kernel's parameter costs registers)
  int abort;
};

// KC: 32-value chunks of the inner dimension (1: two A buffers; 2: one).
template <int KC> struct Cfg {
  static constexpr size_t kSmem = (size_t)2 * kDigABytes + (size_t)2 * KC * kDigBBytes + sizeof(Shared) + 1024;
};

// A CTA's tiles in order, column tiles fastest.
struct Walk {
  int nrt, nct;
  int t, ct, rt, b, i0;  // tile; its column tile, row tile (counted over all blocks), block, first row in it
  __device__ __forceinline__ Walk(int nrt_, int nct_, int t0) : nrt(nrt_), nct(nct_), t(t0) {
    rt = t0 / nct;
    ct = t0 - rt * nct;
    b = rt / nrt;
    i0 = (rt - b * nrt) * 128;
  }
  __device__ __forceinline__ void next() {
    ++t;
    if (++ct < nct) return;
    ct = 0;
    ++rt;
    i0 += 128;
    if (i0 < nrt * 128) return;
    i0 = 0;
    ++b;
  }
};

// The products of marked rows of A and columns of B, left out of a CTA's tiles
// [t0, t1), added by FMAs: all threads, after the tiles.
__device__ __noinline__ void add_marked(const UpdateArgs &a, int nrt, int nct, int t0, int t1, unsigned char *smem) {
  double *sb = reinterpret_cast<double *>(smem);  // the tile's columns of op(B): [32][64]
  bool *row = reinterpret_cast<bool *>(sb + kDigN * 64), *column = row + 128;
  for (Walk w(nrt, nct, t0); w.t < t1; w.next()) {
    const int j0 = w.ct * kDigN, nr = min(128, a.M - w.i0), nc = min(kDigN, a.N - j0);
    const double *A = static_cast<const double *>(a.A) + (long long)w.b * a.a_bstride + w.i0;
    const double *B = a.B + (long long)(w.b >> 1) * a.b_s1 + (long long)((w.b & 1) ^ a.b_flip) * a.b_s2;
    double *C = static_cast<double *>(a.C) + (long long)w.b * a.c_bstride + w.i0 + (long long)j0 * a.ldc;
    __syncthreads();
    for (int e = threadIdx.x; e < nc * a.K; e += kThreads) {
      const int j = j0 + e / a.K, q = e % a.K;
      double v = a.b_trans ? B[j + (long long)q * a.ldb] : B[q + (long long)j * a.ldb];
      if (a.scale) v *= a.scale_cols ? a.scale[j] : a.scale[q];
      sb[e / a.K * 64 + q] = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nr + nc; e += kThreads) {
      if (e < nr)
        row[e] = dig_marked(A + e, a.lda, a.K);
      else
        column[e - nr] = dig_marked(sb + (e - nr) * 64, 1, a.K);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nr * nc; e += kThreads) {
      const int i = e % nr, j = e / nr;
      if (!row[i] && !column[j]) continue;
      double s = 0.0;
      for (int q = 0; q < a.K; ++q) s = fma(A[i + (long long)q * a.lda], sb[j * 64 + q], s);
      double *c = C + i + (long long)j * a.ldc;
      *c = fma(a.alpha, s, *c);
    }
  }
}

}  // namespace

template <int KC>
__global__ void __launch_bounds__(kThreads, 1)
f64_update_tc_kernel(UpdateArgs a, int nrt, int nct, int ntiles, DevStatus *st) {
  if (a.skip && *a.skip) return;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *pa =
      reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *pb = pa + 2 * kDigABytes;
  Shared *sh = reinterpret_cast<Shared *>(pb + 2 * KC * kDigBBytes);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int q = 0; q < 2; ++q) {
      mbar_init(&sh->a_full[q], kSlicers);
      mbar_init(&sh->a_empty[q], 1);
      mbar_init(&sh->b_full[q], kSlicers / 2);
      mbar_init(&sh->b_empty[q], 1);
      mbar_init(&sh->acc_full[q], 2);  // the products' completion, and a plain arrival that publishes the scales
      mbar_init(&sh->acc_free[q], kEpi);
    }
    mbar_init(&sh->slicers, kSlicers);
    mbar_init(&sh->drain, 1);
    const WaitFault wf = g_wait_fault;
    const bool hit = wf.cta == (int)blockIdx.x;
    sh->skip = hit ? wf.stage : -1;
    sh->budget = hit && wf.budget > 0 ? wf.budget : kWait;
    sh->abort = sh->marked = 0;
    sh->args = a;
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    tc_alloc(&sh->tmem, 2 * kDigAccCols);
    tc_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = sh->tmem;
  auto wait = [&](uint64_t *bar, unsigned parity) { return mbar_wait_or_abort(bar, parity, &sh->abort, kWait); };
  const int ksteps = (a.K + 15) / 16;
  const int t0 = (int)((long long)ntiles * blockIdx.x / gridDim.x);
  const int t1 = (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x);
  const int r0 = t0 / nct;  // first row tile
  auto abuf = [&](int rt) { return KC == 1 ? (rt - r0) & 1 : 0; };
  auto ause = [&](int rt) { return KC == 1 ? (rt - r0) >> 1 : rt - r0; };  // earlier fills of that buffer

  if (warp < kSlicers / 32) {
    // ------------------------------------------------------------- slicers
    // A: two threads a row, 16 values of each chunk.  B: the two halves of the
    // slicers take the tiles in turn, so that a tile's loads are in flight for
    // two tiles.
    constexpr int LPC = 4 * KC, HT = kSlicers / 2, BP = kDigN * LPC / HT;  // lanes a column of B, passes over its tile
    const int half = tid / HT, ht = tid % HT;
    const int o = ht % LPC;  // this lane's 8 K values of its columns
    double xb[BP][8];
    auto load_b = [&](const Walk &w) {
      const int j0 = w.ct * kDigN;
      const double *Bb = a.B + (long long)(w.b >> 1) * a.b_s1 + (long long)((w.b & 1) ^ a.b_flip) * a.b_s2;
#pragma unroll
      for (int p = 0; p < BP; ++p) {
        const int j = j0 + ht / LPC + p * (HT / LPC);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int q = 8 * o + e;
          double v = 0.0;
          if (q < a.K && j < a.N) {
            v = a.b_trans ? Bb[j + (long long)q * a.ldb] : Bb[q + (long long)j * a.ldb];
            if (a.scale) v *= a.scale_cols ? a.scale[j] : a.scale[q];
          }
          xb[p][e] = v;
        }
      }
    };
    auto wwait = [&](uint64_t *bar, unsigned parity) {  // with a warp-uniform outcome
      return __all_sync(0xffffffffu, wait(bar, parity));
    };
    // value k of the thread's row of a row tile: a_ptr(w)[k * lda], if a_in(w)
    auto a_ptr = [&](const Walk &w) { return static_cast<const double *>(a.A) + (long long)w.b * a.a_bstride + w.i0 + ht; };
    auto a_in = [&](const Walk &w) { return w.i0 + ht < a.M; };
    Walk w(nrt, nct, t0), wb = w;  // this tile; the half's next tile to load
    if (half == 1) wb.next();
    if (wb.t < t1) load_b(wb);
    // all slicers together; false when a role has given up
    int syncs = 0;
    auto sync = [&]() {
      mbar_arrive(&sh->slicers);
      return wwait(&sh->slicers, (unsigned)(syncs++ & 1));
    };
    int bal[KC];  // lane k: the balance of inner index 32 c + k
    for (; w.t < t1; w.next()) {
      const int ti = w.t - t0, rt = w.rt;
      if (w.t == t0 || w.ct == 0) {
        const int ab = abuf(rt), par = (rt - r0) & 1;
        const double *Ar = a_ptr(w);
        const bool in = a_in(w);
        unsigned xe[16] = {};  // the values' exponents, chunk c's from bit 16 c on
#pragma unroll
        for (int c = 0; c < KC; ++c)
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            const int k = 32 * c + 16 * half + q;
            if (in && k < a.K) xe[q] |= dig_ahi(Ar[(long long)k * a.lda]) >> 20 << (16 * c);
          }
        auto exponent = [&](int c, int q) { return KC == 1 ? xe[q] : xe[q] >> (16 * c) & 0xffffu; };
        // The balance: the largest |A(., k)| of this row tile, no other's: any power of
        // two keeps the products exact, but both operands are cut relative to the
        // largest balanced value, and one that does not fit the tile's columns shifts
        // their digits out.  It costs the slicers a second meeting a row tile: nothing
        // at inner dimensions up to 32, 3 to 8 % above (2^19 rows, inner 64, 64 columns
        // 462 us, 448 with the maxima of the row tile before; 192 columns 870, 844).
        // Exponents, not high words, are held across it: two chunks of the latter spill.
#pragma unroll
        for (int c = 0; c < KC; ++c)
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            const unsigned e = exponent(c, q), m = __reduce_max_sync(0xffffffffu, e == 0x7ffu ? 0u : e);
            if (lane == q) sh->colw[par][warp & 3][32 * c + 16 * half + q] = m;
          }
        if (!sync()) break;
#pragma unroll
        for (int c = 0; c < KC; ++c) {
          const unsigned(*cw)[64] = sh->colw[par];
          const int k = 32 * c + lane;
          bal[c] = (int)max(max(cw[0][k], cw[1][k]), max(cw[2][k], cw[3][k]));
        }
        int key = kDigZero;
        unsigned mx = 0;
#pragma unroll
        for (int c = 0; c < KC; ++c)
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            const unsigned e = exponent(c, q);
            const int b = __shfl_sync(0xffffffffu, bal[c], 16 * half + q);
            if (e) key = max(key, (int)e - b);
            mx = max(mx, e);
          }
        mx <<= 20;
        sh->key2[par][half][ht] = key;
        sh->mx2[par][half][ht] = mx;
        if (!sync()) break;
        key = max(key, sh->key2[par][half ^ 1][ht]);
        mx = max(mx, sh->mx2[par][half ^ 1][ht]);
        if (ause(rt) > 0 && !wwait(&sh->a_empty[ab], (unsigned)((ause(rt) - 1) & 1))) break;
        // Only now: the products of row tile rt - 2 (KC 2: rt - 1) are complete, so they
        // were issued, two tiles after those of rt - 4 at least, once the epilogue had
        // freed that set -- and read the scales this slot held.
        if (half == 0) sh->ea[rt & 3][ht] = dig_scale(key, mx, kDigZeroA);
        if (mx >= 0x7ff00000u) sh->marked = 1;
#pragma unroll
        for (int c = 0; c < KC; ++c)
#pragma unroll
          for (int g = 0; g < 2; ++g) {  // the values once more, from the L1 cache
            const int k0 = 16 * half + 8 * g;
            double x[8];
            int bx[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
              x[e] = in && 32 * c + k0 + e < a.K ? Ar[(long long)(32 * c + k0 + e) * a.lda] : 0.0;
#pragma unroll
            for (int e = 0; e < 8; ++e) bx[e] = -__shfl_sync(0xffffffffu, bal[c], k0 + e);
            if (32 * c + k0 < 16 * ksteps)
              dig_put8(pa + (ab + c) * kDigABytes, kDigAPlane, swz64(ht, 2 * half + g), x,
                       [&](int e) { return bx[e]; }, key);
          }
        fence_proxy_async_smem();
        mbar_arrive(&sh->a_full[ab]);
        if (w.i0 + 128 < a.M && (lane & 15) == 0) {  // the next row tile's values into L2
#pragma unroll
          for (int k = 0; k < 16 * KC; ++k) {
            const int kk = (k >> 4) * 32 + 16 * half + (k & 15);
            if (kk < a.K) asm volatile("prefetch.global.L2 [%0];" ::"l"(Ar + 128 + (long long)kk * a.lda));
          }
        }
      }
      const int slot = ti & 1;
      if (half != slot) continue;
      if (ti >= 2 && !wwait(&sh->b_empty[slot], (unsigned)(((ti >> 1) - 1) & 1))) break;
#pragma unroll
      for (int p = 0; p < BP; ++p) {
        const int col = ht / LPC + p * (HT / LPC);
        int key = kDigZero, bx[8];
        unsigned mx = 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          bx[e] = __shfl_sync(0xffffffffu, bal[0], (8 * o + e) & 31);
          if (KC == 2) {
            const int b1 = __shfl_sync(0xffffffffu, bal[KC - 1], (8 * o + e) & 31);
            if (o >= 4) bx[e] = b1;
          }
          dig_key(key, dig_ahi(xb[p][e]), bx[e]);
          mx = max(mx, dig_ahi(xb[p][e]));
        }
#pragma unroll
        for (int x = 1; x < LPC; x <<= 1) {
          key = max(key, __shfl_xor_sync(0xffffffffu, key, x));
          mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, x));
        }
        if (o == 0) sh->eb[ti & 7][col] = dig_scale(key, mx, kDigZeroB);
        if (mx >= 0x7ff00000u) sh->marked = 1;
        if (8 * o < 16 * ksteps)
          dig_put8(pb + (slot * KC + o / 4) * kDigBBytes, kDigBPlane, swz64(col, o & 3), xb[p],
                   [&](int e) { return bx[e]; }, key);
      }
      fence_proxy_async_smem();
      if (ti != sh->skip) mbar_arrive(&sh->b_full[slot]);
      wb.next();
      wb.next();
      if (wb.t < t1) load_b(wb);
    }
  } else if (warp == kMmaWarp) {
    // ----------------------------------------------------------- products
    if (lane == 0) {
      for (Walk w(nrt, nct, t0); w.t < t1; w.next()) {
        const int ti = w.t - t0, rt = w.rt, ab = abuf(rt), slot = ti & 1;
        if ((w.t == t0 || w.ct == 0) && !wait(&sh->a_full[ab], (unsigned)(ause(rt) & 1))) break;
        if (!mbar_wait_or_abort(&sh->b_full[slot], (unsigned)((ti >> 1) & 1), &sh->abort, &sh->budget) ||
            (ti >= 2 && !wait(&sh->acc_free[slot], (unsigned)(((ti >> 1) - 1) & 1))))
          break;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < KC; ++c)
          dig_mma_chunk(tmem + (unsigned)slot * kDigAccCols, smem_u32(pa + (ab + c) * kDigABytes),
                        smem_u32(pb + (slot * KC + c) * kDigBBytes), min(2, ksteps - 2 * c), c == 0);
        tc_commit(&sh->acc_full[slot]);
        mbar_arrive(&sh->acc_full[slot]);
        tc_commit(&sh->b_empty[slot]);
        if (w.ct + 1 == nct) tc_commit(&sh->a_empty[ab]);
      }
      tc_commit(&sh->drain);  // completes once every product issued above has
      const long long w0 = clock64();
      while (!mbar_try_wait(&sh->drain, 0) && clock64() - w0 < kWait) {
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3, h = (warp - kSlicers / 32) >> 2, row = 32 * q + lane;
    // C values of the thread's row and columns of a tile; those of two
    // columns are loaded again, for the next tile, as soon as they are used
    double cv[kEpiCols];
    auto c_ptr = [&](const Walk &w, int &jn) -> double * {  // jn: valid columns from the pointer on
      const int i = w.i0 + row, j0 = w.ct * kDigN + kEpiCols * h;
      jn = i < a.M ? a.N - j0 : 0;
      return static_cast<double *>(a.C) + (long long)w.b * a.c_bstride + i + (long long)j0 * a.ldc;
    };
    int jn = 0, jn1 = 0;
    Walk w(nrt, nct, t0);
    double *Cr = c_ptr(w, jn), *Cn = Cr;
    if (t0 >= t1) jn = 0;
#pragma unroll
    for (int c = 0; c < kEpiCols; ++c) cv[c] = c < jn && !a.overwrite ? Cr[(long long)c * a.ldc] : 0.0;
    while (w.t < t1) {
      const int ti = w.t - t0, slot = ti & 1, rt = w.rt;
      w.next();
      jn1 = 0;
      if (w.t < t1) Cn = c_ptr(w, jn1);
      if (!__all_sync(0xffffffffu, wait(&sh->acc_full[slot], (unsigned)((ti >> 1) & 1)))) break;
      tc_fence_after();
      const int ea = sh->ea[rt & 3][row];
      const unsigned tl = tmem + ((unsigned)(32 * q) << 16) + (unsigned)slot * kDigAccCols + kEpiCols * h;
#pragma unroll
      for (int c2 = 0; c2 < kEpiCols; c2 += 2) {
        unsigned v[kDiag][2];
#pragma unroll
        for (int d = 0; d < kDiag; ++d) tc_ld2(tl + (unsigned)(d * kDigN + c2), v[d]);
        tc_wait_ld(v);
        if (c2 == kEpiCols - 2) {
          tc_fence_before();
          mbar_arrive(&sh->acc_free[slot]);
        }
        const int *eb = sh->eb[ti & 7] + kEpiCols * h + c2;
        bool odd = false;
        double x[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) x[c] = dig_value(dig_combine<32 * KC>(v, c), ea + eb[c], odd);
        if (odd)
          for (int c = 0; c < 2; ++c) x[c] = dig_value_any<false>(dig_combine<32 * KC>(v, c), ea + eb[c]);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int cc = c2 + c;
          if (cc < jn) Cr[(long long)cc * a.ldc] = fma(a.alpha, x[c], cv[cc]);
          cv[cc] = cc < jn1 && !a.overwrite ? Cn[(long long)cc * a.ldc] : 0.0;
        }
      }
      Cr = Cn;
      jn = jn1;
    }
  }
  __syncthreads();
  if (tid == 0 && sh->abort) report_error(st, HODLR_ERR_TIMEOUT, blockIdx.x);
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tc_dealloc(tmem, 2 * kDigAccCols);
  }
  if (sh->marked && !sh->abort) add_marked(sh->args, nrt, nct, t0, t1, pa);
}

template <int KC>
static cudaError_t launch_kc(const UpdateArgs &a, DevStatus *st, cudaStream_t s) {
  auto k = f64_update_tc_kernel<KC>;
  cudaError_t e = allow_dyn_smem(k, Cfg<KC>::kSmem);
  if (e != cudaSuccess) return e;
  const int nrt = ceil_div(a.M, 128), nct = ceil_div(a.N, kDigN);
  const int ntiles = nrt * nct * a.nbatch;
  note_waiting_launch();
  HODLR_LAUNCH(k, (unsigned)std::min(ntiles, kNumSMs), kThreads, Cfg<KC>::kSmem, s, a, nrt, nct, ntiles, st);
  return cudaGetLastError();
}

cudaError_t f64_update_tc_set_wait_fault(const WaitFault &wf) {
  return cudaMemcpyToSymbol(g_wait_fault, &wf, sizeof wf);
}

bool f64_update_tc_try(const UpdateArgs &a, DevStatus *st, cudaStream_t s, cudaError_t &err) {
  if (a.a_trans || a.K < 1 || a.K > 64) return false;
  if ((long long)ceil_div(a.M, 128) * ceil_div(a.N, kDigN) * a.nbatch > (1 << 30)) return false;  // 32-bit tile counts
  err = a.K <= 32 ? launch_kc<1>(a, st, s) : launch_kc<2>(a, st, s);
  return true;
}

}  // namespace hodlr
