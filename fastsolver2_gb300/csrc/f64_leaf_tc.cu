// K2 in FP64 on the tcgen05 tensor cores: Y_i = Dinv_i X_i on the rows of every
// leaf i (leaf sizes 64, 128 and 256) with exact digit products (f64_tc.cuh).
//
// The inverses are cut into digits once, after the factorisation made them
// (leaf_image_kernel: 14 bytes a value, in the shared-memory layout the
// products read, so that a chunk of 32 columns of an inverse is one bulk copy
// of 56 KB); the columns of X are cut as they are used.  A unit of work is a
// leaf and two accumulator sets of 128 rows x 32 columns: 64 columns of X for
// leaves up to 128 rows, 32 columns and both row tiles for 256, so that a chunk
// of X's digits is used twice, or a chunk of the inverse's.  The exactness of
// the accumulators ends at 128 terms: leaves of 256 rows run as two halves of
// the inner dimension, added in FP64.
//
// What bounds it: the products, 2 x 4 chunks x 16 instructions of about 100
// clocks a unit at leaf 128 (12800 clocks; HBM's share of a unit is 5600);
// the digits of X (40 instructions a value) and the packing of the results (60)
// run beside them on other warps.  Measured at N = 2^20, leaf 128, rank 32, 64
// right-hand sides: the 416 columns of the factorisation and the solve's 64
// together 4.2 ms, the images 0.6; the FP64 FMA kernel took 110.
#include <algorithm>

#include "f64_tc.cuh"
#include "kernels.cuh"

namespace hodlr {

namespace {

constexpr int kSW = 8, kEW = 16;  // warps cutting X, epilogue
constexpr int kMmaWarp = kSW + kEW, kProdWarp = kMmaWarp + 1, kThreads = 32 * (kProdWarp + 1);
constexpr int kAStages = 2, kBStages = 3;
constexpr int kEpiCols = kDigN * 4 / kEW;  // columns of a set an epilogue thread turns
constexpr long long kWait = 2000000000LL;  // about one second of SM clocks

__device__ WaitFault g_wait_fault = {-1, -1, 0};

struct Shared {
  uint64_t a_full[kAStages], a_empty[kAStages], b_full[kBStages], b_empty[kBStages], acc_full[2], acc_free[2], drain;
  int eb[4][2 * kDigN];  // the column scales of the last groups
  long long budget;  // of the wait the hook lets run out, in SM clocks
  int skip;          // test hook: the stage whose digits are never announced (-1: none)
  unsigned tmem;
  int abort;
};

// MT: row tiles of a leaf (2 for 256 rows); column tiles a unit.
template <int MT> struct Cfg {
  static constexpr int kNT = 3 - MT;
  static constexpr int kBStage = kNT * kDigBBytes;
  static constexpr size_t kSmem = (size_t)kAStages * kDigABytes + (size_t)kBStages * kBStage + sizeof(Shared) + 1024;
};

struct LeafArgs {
  const unsigned char *img;  // [leaf][half][chunk][row tile] planes
  const int *rows;           // [leaf][half][row tile][128] row scales
  const int *bal;            // [leaf][m] balances
  const double *X;
  double *Y;
  long long ldx, ldy;
  int m, ncols, nct;  // column groups of a leaf (kNT tiles each)
  long long units;
  const int *skip;
  DevStatus *st;
};

__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

}  // namespace

// ------------------------------------------------------------- the images
// One CTA a leaf: the balance of every inner index (its column's largest), the
// row scales of each half, and the digit planes chunk by chunk through shared
// memory.  A stream over the inverses: 8 bytes read and 14 written a value.
__global__ void __launch_bounds__(256) leaf_image_kernel(const double *__restrict__ Dinv, int m, unsigned char *img,
                                                         int *rows, int *bal) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *planes =
      reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ int sbal[256], skey[2][128];
  __shared__ unsigned smx[2][128];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long leaf = blockIdx.x;
  const double *A = Dinv + leaf * m * m;
  for (int k = warp; k < m; k += 8) {
    unsigned mx = 0;
    for (int i = lane; i < m; i += 32) mx = max(mx, dig_finite(dig_ahi(A[i + (long long)k * m])));
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) {
      sbal[k] = (int)(mx >> 20);
      bal[leaf * m + k] = sbal[k];
    }
  }
  __syncthreads();
  const int mt = m > 128 ? m / 128 : 1, kh = mt, kc = min(m, 128) / kDigK;  // row tiles, halves, chunks a half
  const int row = tid & 127, part = tid >> 7;
  for (int h = 0; h < kh; ++h)
    for (int t = 0; t < mt; ++t) {
      const bool in = row < m;
      const double *Ar = A + t * 128 + row;
      int key = kDigZero;
      unsigned mx = 0;
      if (in)
        for (int k = part; k < kDigK * kc; k += 2) {
          const int kk = 128 * h + k;
          const unsigned w = dig_ahi(Ar[(long long)kk * m]);
          dig_key(key, w, -sbal[kk]);
          mx = max(mx, w);
        }
      skey[part][row] = key;
      smx[part][row] = mx;
      __syncthreads();
      key = max(skey[0][row], skey[1][row]);
      mx = max(smx[0][row], smx[1][row]);
      if (part == 0) rows[((leaf * kh + h) * mt + t) * 128 + row] = dig_scale(key, mx, kDigZeroA);
      for (int c = 0; c < kc; ++c) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const int k0 = 16 * part + 8 * g, kk = 128 * h + kDigK * c + k0;
          double x[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = in ? Ar[(long long)(kk + e) * m] : 0.0;
          dig_put8(planes, kDigAPlane, swz64(row, k0 >> 3), x, [&](int e) { return -sbal[kk + e]; }, key);
        }
        __syncthreads();
        uint4 *dst = reinterpret_cast<uint4 *>(img + (((leaf * kh + h) * kc + c) * mt + t) * kDigABytes);
        for (int e = tid; e < kDigABytes / 16; e += 256) dst[e] = reinterpret_cast<const uint4 *>(planes)[e];
        __syncthreads();
      }
    }
}

template <int MT>
__global__ void __launch_bounds__(kThreads, 1) f64_leaf_tc_kernel(LeafArgs a) {
  if (a.skip && *a.skip) return;
  constexpr int NT = Cfg<MT>::kNT, KH = MT;  // halves of the inner dimension
  extern __shared__ unsigned char smem_raw[];
  unsigned char *pa =
      reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *pb = pa + kAStages * kDigABytes;
  Shared *sh = reinterpret_cast<Shared *>(pb + kBStages * Cfg<MT>::kBStage);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int q = 0; q < kAStages; ++q) {
      mbar_init(&sh->a_full[q], 1);
      mbar_init(&sh->a_empty[q], 1);
    }
    for (int q = 0; q < kBStages; ++q) {
      mbar_init(&sh->b_full[q], 32 * kSW);
      mbar_init(&sh->b_empty[q], 1);
    }
    for (int q = 0; q < 2; ++q) {
      mbar_init(&sh->acc_full[q], 2);  // the products' completion, and a plain arrival that publishes the scales
      mbar_init(&sh->acc_free[q], 32 * kEW);
    }
    mbar_init(&sh->drain, 1);
    const WaitFault wf = g_wait_fault;
    const bool hit = wf.cta == (int)blockIdx.x;
    sh->skip = hit ? wf.stage : -1;
    sh->budget = hit && wf.budget > 0 ? wf.budget : kWait;
    sh->abort = 0;
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
  auto wwait = [&](uint64_t *bar, unsigned parity) { return __all_sync(0xffffffffu, wait(bar, parity)); };
  const int kc = min(a.m, 128) / kDigK;  // chunks of a half
  const long long u0 = a.units * blockIdx.x / gridDim.x, u1 = a.units * (blockIdx.x + 1) / gridDim.x;
  long long leaf = u0 / a.nct;
  int cg = (int)(u0 - leaf * a.nct);  // the unit: leaf, column group
  auto next = [&]() {
    if (++cg == a.nct) {
      cg = 0;
      ++leaf;
    }
  };
  int stage = 0;  // A stages issued (the producer)
  bool ok = true;

  if (warp < kSW) {
    // ------------------------------------------------------------ X digits
    // lane: column lane / 8 of its warp's four in each column tile, rows
    // 4 (lane % 8) .. + 3 of each chunk
    const int col = 4 * warp + (lane >> 3), lr = 4 * (lane & 7);
    int grp = 0, bs = 0;  // groups (unit, half) and B stages passed
    for (long long u = u0; ok && u < u1; ++u, next()) {
      const int c0 = cg * NT * kDigN;
      for (int h = 0; ok && h < KH; ++h, ++grp) {
        const double *Xg = a.X + leaf * a.m + 128 * h + lr + (long long)(c0 + col) * a.ldx;
        const int *bg = a.bal + leaf * a.m + 128 * h + lr;
        int key[NT];
        unsigned mx[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          key[t] = kDigZero;
          mx[t] = 0;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c >= kc) continue;
          unsigned xh[NT][4];
          const int4 b = *reinterpret_cast<const int4 *>(bg + kDigK * c);
          const int bal[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              xh[t][e] = c0 + kDigN * t + col < a.ncols ? dig_ahi(Xg[kDigK * c + e + (long long)(kDigN * t) * a.ldx]) : 0u;
#pragma unroll
          for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              dig_key(key[t], xh[t][e], bal[e]);
              mx[t] = max(mx[t], xh[t][e]);
            }
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
#pragma unroll
          for (int s = 1; s < 8; s <<= 1) {
            key[t] = max(key[t], __shfl_xor_sync(0xffffffffu, key[t], s));
            mx[t] = max(mx[t], __shfl_xor_sync(0xffffffffu, mx[t], s));
          }
          if ((lane & 7) == 0) sh->eb[grp & 3][kDigN * t + col] = dig_scale(key[t], mx[t], kDigZeroB);
        }
        double x[NT][4];
        auto load = [&](int c) {  // the values, from the L2
#pragma unroll
          for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              x[t][e] = c0 + kDigN * t + col < a.ncols ? Xg[kDigK * c + e + (long long)(kDigN * t) * a.ldx] : 0.0;
        };
        load(0);
        for (int c = 0; c < kc; ++c, ++bs) {
          const int slot = bs % kBStages;
          if (bs >= kBStages && !wwait(&sh->b_empty[slot], (unsigned)((bs / kBStages - 1) & 1))) {
            ok = false;
            break;
          }
          const int4 b = *reinterpret_cast<const int4 *>(bg + kDigK * c);
#pragma unroll
          for (int t = 0; t < NT; ++t)
            dig_put4(pb + slot * Cfg<MT>::kBStage + t * kDigBBytes, kDigBPlane, swz64(col, lr >> 3) + 2 * (lr & 7), x[t],
                     [&](int e) { return e == 0 ? b.x : e == 1 ? b.y : e == 2 ? b.z : b.w; }, key[t]);
          fence_proxy_async_smem();
          if (bs != sh->skip) mbar_arrive(&sh->b_full[slot]);
          if (c + 1 < kc) load(c + 1);
        }
      }
    }
  } else if (warp == kProdWarp) {
    // ------------------------------------------- the inverses' digits, in order
    if (lane == 0)
      for (long long u = u0; ok && u < u1; ++u, next()) {
        const unsigned char *src = a.img + leaf * (KH * kc * MT) * (long long)kDigABytes;
        for (int i = 0; i < KH * kc * MT; ++i, ++stage) {
          const int slot = stage % kAStages;
          if (stage >= kAStages && !wait(&sh->a_empty[slot], (unsigned)((stage / kAStages - 1) & 1))) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&sh->a_full[slot], kDigABytes);
          bulk_load(pa + slot * kDigABytes, src + (long long)i * kDigABytes, kDigABytes, &sh->a_full[slot]);
        }
      }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ products
    if (lane == 0) {
      int as = 0, bs = 0, grp = 0;
      for (long long u = u0; ok && u < u1; ++u, next()) {
        const bool two = NT == 1 || (cg * NT + 1) * kDigN < a.ncols;  // the second set has columns
        for (int h = 0; ok && h < KH; ++h, ++grp)
          for (int c = 0; ok && c < kc; ++c, ++bs) {
            const int bslot = bs % kBStages;
            if (!mbar_wait_or_abort(&sh->b_full[bslot], (unsigned)((bs / kBStages) & 1), &sh->abort, &sh->budget)) ok = false;
            for (int t = 0; ok && t < MT; ++t, ++as) {
              const int aslot = as % kAStages;
              if (!wait(&sh->a_full[aslot], (unsigned)((as / kAStages) & 1))) {
                ok = false;
                break;
              }
              for (int n = 0; n < NT; ++n) {
                const int set = MT == 2 ? t : n;
                if (c == 0 && grp > 0 && !wait(&sh->acc_free[set], (unsigned)((grp - 1) & 1))) {
                  ok = false;
                  break;
                }
                tc_fence_after();
                if (set == 0 || two)
                  dig_mma_chunk(tmem + (unsigned)set * kDigAccCols, smem_u32(pa + aslot * kDigABytes),
                                smem_u32(pb + bslot * Cfg<MT>::kBStage + n * kDigBBytes), 2, c == 0);
                if (c == kc - 1) {
                  tc_commit(&sh->acc_full[set]);
                  mbar_arrive(&sh->acc_full[set]);
                }
              }
              if (ok) tc_commit(&sh->a_empty[aslot]);
            }
            if (ok) tc_commit(&sh->b_empty[bslot]);
          }
      }
      tc_commit(&sh->drain);  // completes once every product issued above has
      const long long w0 = clock64();
      while (!mbar_try_wait(&sh->drain, 0) && clock64() - w0 < kWait) {
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3, h4 = (warp - kSW) >> 2, row = 32 * q + lane;
    const bool idle = 32 * q >= a.m;  // rows past a leaf of 64
    int grp = 0;
    for (long long u = u0; ok && u < u1; ++u, next()) {
      double y[KH == 2 ? 2 : 1][kEpiCols];
      for (int h = 0; ok && h < KH; ++h, ++grp)
#pragma unroll
        for (int set = 0; set < 2; ++set) {
          const int mt = MT == 2 ? set : 0, c0 = (cg * NT + (MT == 2 ? 0 : set)) * kDigN + kEpiCols * h4;
          const int er = idle ? 0 : a.rows[((leaf * KH + h) * MT + mt) * 128 + row];
          if (!wwait(&sh->acc_full[set], (unsigned)(grp & 1))) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (!idle && c0 < a.ncols) {  // warp-uniform
            const unsigned tl = tmem + ((unsigned)(32 * q) << 16) + (unsigned)set * kDigAccCols + kEpiCols * h4;
            const int *eb = sh->eb[grp & 3] + (MT == 2 ? 0 : kDigN * set) + kEpiCols * h4;
            double *Yr = a.Y + leaf * a.m + 128 * mt + row + (long long)c0 * a.ldy;
#pragma unroll
            for (int c2 = 0; c2 < kEpiCols; c2 += 2) {
              unsigned v[kDiag][2];
#pragma unroll
              for (int d = 0; d < kDiag; ++d) tc_ld2(tl + (unsigned)(d * kDigN + c2), v[d]);
              tc_wait_ld(v);
              bool odd = false;
              double x[2];
#pragma unroll
              for (int c = 0; c < 2; ++c) x[c] = dig_value(dig_combine<128>(v, c), er + eb[c2 + c], odd);
              if (odd)
                for (int c = 0; c < 2; ++c) x[c] = dig_value_any(dig_combine<128>(v, c), er + eb[c2 + c]);
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                if (KH == 2 && h == 0) {
                  y[set % (KH == 2 ? 2 : 1)][c2 + c] = x[c];
                } else {
                  if (KH == 2) x[c] += y[set % (KH == 2 ? 2 : 1)][c2 + c];
                  if (c0 + c2 + c < a.ncols) Yr[(long long)(c2 + c) * a.ldy] = x[c];
                }
              }
            }
          }
          tc_fence_before();
          mbar_arrive(&sh->acc_free[set]);
        }
    }
  }
  __syncthreads();
  if (warp == kProdWarp && lane == 0 && sh->abort) {
    report_error(a.st, HODLR_ERR_TIMEOUT, blockIdx.x);
    // copies issued but possibly still landing: wait (bounded) for them
    for (int i = max(0, stage - kAStages); i < stage; ++i) {
      const long long w0 = clock64();
      while (!mbar_try_wait(&sh->a_full[i % kAStages], (unsigned)((i / kAStages) & 1)) && clock64() - w0 < kWait) {
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tc_dealloc(tmem, 2 * kDigAccCols);
  }
}

cudaError_t f64_leaf_tc_set_wait_fault(const WaitFault &wf) {
  return cudaMemcpyToSymbol(g_wait_fault, &wf, sizeof wf);
}

// Sizes of the digit images of nleaf inverses: bytes of planes, ints of row
// scales (the balances take nleaf * m ints).
size_t f64_leaf_image_bytes(int m, int nleaf) {
  const size_t mt = m > 128 ? m / 128 : 1;
  return (size_t)nleaf * mt * (m / kDigK) * kDigABytes;
}
size_t f64_leaf_image_rows(int m, int nleaf) {
  const size_t mt = m > 128 ? m / 128 : 1;
  return (size_t)nleaf * mt * mt * 128;
}

cudaError_t launch_f64_leaf_image(const double *Dinv, int m, int nleaf, unsigned char *img, int *rows, int *bal,
                                  cudaStream_t s) {
  if (nleaf <= 0) return cudaSuccess;
  const size_t bytes = kDigABytes + 1024;
  cudaError_t e = allow_dyn_smem(leaf_image_kernel, bytes);
  if (e != cudaSuccess) return e;
  HODLR_LAUNCH(leaf_image_kernel, nleaf, 256, bytes, s, Dinv, m, img, rows, bal);
  return cudaGetLastError();
}

template <int MT>
static cudaError_t launch_mt(LeafArgs a, int nleaf, cudaStream_t s) {
  auto k = f64_leaf_tc_kernel<MT>;
  cudaError_t e = allow_dyn_smem(k, Cfg<MT>::kSmem);
  if (e != cudaSuccess) return e;
  a.nct = ceil_div(a.ncols, Cfg<MT>::kNT * kDigN);
  a.units = (long long)nleaf * a.nct;
  HODLR_LAUNCH(k, (unsigned)std::min<long long>(a.units, kNumSMs), kThreads, Cfg<MT>::kSmem, s, a);
  return cudaGetLastError();
}

// Y_i = Dinv_i X_i, Y may be X (a unit's columns are read before they are written).
cudaError_t launch_f64_leaf_tc(const unsigned char *img, const int *rows, const int *bal, int m, int nleaf,
                               const double *X, long long ldx, double *Y, long long ldy, int ncols, const int *skip,
                               DevStatus *st, cudaStream_t s) {
  if (ncols <= 0 || nleaf <= 0) return cudaSuccess;
  LeafArgs a{img, rows, bal, X, Y, ldx, ldy, m, ncols, 0, 0, skip, st};
  return m <= 128 ? launch_mt<1>(a, nleaf, s) : launch_mt<2>(a, nleaf, s);
}

}  // namespace hodlr
