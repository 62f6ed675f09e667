// Panel GEMM, FP64 on the tensor pipe and FP32 on packed multiply-adds: the L.psi and .R
// contractions of HVecQt (source/mpo_dmrg_kernelQt.py:301, 306-316).
//
// Both operands are K-major with 16-byte aligned rows: the L panels of one contracted
// sector [M x Kp] against the wavefunction's panel of that sector [sum_j N_j x Kp] (all psi
// blocks of the sector side by side, so that narrow blocks share a tile), and the T3 panels
// [M x Kp] against the transposed R panels [D_r' x Kp].
//
// The FP64 tensor pipe runs at the DFMA rate (37 TFLOP/s), but one m8n8k4 product does 256
// multiply-adds from one register per operand, so neither shared memory nor issue slots
// bound the loop as they do with DFMA.  Tile: 128 rows x up to 64 columns, eight warps of
// 16 rows; a warp's column count is compiled for every multiple of 8 (small sectors end a
// tile early).  Operands come through a three-stage cp.async ring of 16-deep K slices; row pitch
// 20 elements: the eight rows x four k of a fragment touch every bank once.  A persistent grid, two CTAs per
// SM, walks the (tile, operator) list; the ring runs on from one tile into the next, so the
// short panels of L.psi (a few K slices each) do not wait for their first operands.
//
// Measured at the mid-chain dot of K=24, D=500 (160 GFLOP each; DFMA kernel before): L.psi
// 16.8 -> 7.5 ms (21.3 TFLOP/s, 58 % of the pipe), .R 14.5 -> 5.8 ms (27.6, 75 %).  L.psi is
// held back by its T1 stores and by K extents that end inside a 16-deep slice, .R by the
// last wave of tiles and the ring's barriers.
//
// FP32 keeps the ring and its bytes with 256 x 32 tiles (a sector's D_r' is rarely above 32 up to
// K=16, D=173): a thread holds 8 x 4 results as pairs over even and odd k, so that a 16-byte
// read of a K-major row is two packed operands without a move.  K=16, D=173 (6.5 GFLOP): L.psi and
// .R together 992 us on the grouped kernel with row-major operands, now 190 + 171 us, bound by
// tiles of short K (L.psi) and of few columns (.R).  At K=24, D=200, whose sectors are wider, 693 + 525 us
// against 849 + 619 in FP64 under the profiler: 1.2 times faster where the pipes allow 2.
#include <cuda_runtime.h>
#include <atomic>
#include <cstdio>
#include "qc_types.h"

namespace {

constexpr int DP_BK = 16, DP_ST = 3, DP_THREADS = 256;
constexpr int DP_P = DP_BK + 4;                                  // row pitch in elements

// Tile of a type: rows x columns, elements of a 16-byte copy.
template <typename T>
struct Dp {
  static constexpr int BM = sizeof(T) == 8 ? 128 : 256, BN = sizeof(T) == 8 ? 64 : 32, V = 16 / sizeof(T);
  static constexpr int STAGE = (BM + BN) * DP_P;                 // elements of one stage
  static constexpr int SMEM = DP_ST * STAGE * (int)sizeof(T);
  static constexpr int RP = DP_THREADS * V / DP_BK;              // rows that one copy of all threads covers
};
constexpr int DP_PT = Dp<double>::BM + 4;                        // pitch of an A tile staged [k][m]
constexpr int DP_NT = 8;                                         // FP64: column groups of eight of a tile

template <typename T>
__device__ __forceinline__ void dp_cp16(unsigned dst, const T *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void dp_mma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// One K slice (k4 groups of four k) of a warp's 16 x 8 NT tile.  LONG: whole slices have code of
// their own without the tests of k4, so that the next group's operands are read ahead of the
// products.  .R (long K): 6.18 -> 5.77 ms at D = 500; L.psi, whose tiles are 1 to 7 slices, lost 3 %.
template <int NT, bool AT, bool LONG, bool FULL = false>
__device__ __forceinline__ void dp_slice(const double *as, const double *bs, int k4, double (&acc)[2][DP_NT][2]) {
  if (LONG && !FULL && k4 == DP_BK / 4) return dp_slice<NT, AT, LONG, true>(as, bs, k4, acc);
#pragma unroll
  for (int kk = 0; kk < DP_BK / 4; ++kk) {
    if (FULL || kk < k4) {
      const double a0 = as[4 * kk * (AT ? DP_PT : 1)], a1 = as[4 * kk * (AT ? DP_PT : 1) + 8 * (AT ? 1 : DP_P)];
      double b[NT];
#pragma unroll
      for (int j = 0; j < NT; ++j) b[j] = bs[8 * j * DP_P + 4 * kk];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        dp_mma(acc[0][j], a0, b[j]);
        dp_mma(acc[1][j], a1, b[j]);
      }
    }
  }
}

// The same in FP32: 32 rows x 8 NT columns of a warp, lane (i, j) = (lane / 8, lane % 8) holds rows i,
// i + 4, ... and columns j, j + 8, ...; a packed accumulator sums the even and the odd k.
template <int NT>
__device__ __forceinline__ void dp_slice(const float *as, const float *bs, int k4, unsigned long long (&acc)[8][4]) {
#pragma unroll
  for (int kk = 0; kk < DP_BK / 4; ++kk) {
    if (kk < k4) {
      ulonglong2 b[NT];
#pragma unroll
      for (int j = 0; j < NT; ++j) b[j] = *reinterpret_cast<const ulonglong2 *>(bs + 8 * j * DP_P + 4 * kk);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(as + 4 * i * DP_P + 4 * kk);
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(a.x), "l"(b[j].x));
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(a.y), "l"(b[j].y));
        }
      }
    }
  }
}

struct DpRec {
  qc_dunit u;
  qc_op o;
};
static_assert(sizeof(DpRec) == 96, "unit and operator records back to back");
constexpr int DP_RECS = 8;       // a CTA's records in flight: the loads run at most two tiles ahead
// place of tile column n in the staged B tile: an accumulator pair of lane l holds the columns
// l % 4 and l % 4 + 4 of its group of eight, so that four lanes store 32 contiguous bytes
__device__ __forceinline__ int dp_col_place(int n) { return (n & ~7) | ((n & 3) << 1) | ((n >> 2) & 1); }

constexpr int DP_ROWS = 0, DP_COLS = 1, DP_BLK = 2;      // where a tile goes (qc_dunit)

template <typename T, int MODE>
__global__ void __launch_bounds__(DP_THREADS, 2)
k_dpanel(const qc_dunit *__restrict__ units, const int2 *__restrict__ work, int nwork,
         const qc_op *__restrict__ ops, const long long *__restrict__ crow, const qc_dcol *__restrict__ cols,
         const T *__restrict__ A, const T *__restrict__ B, T *__restrict__ C) {
  constexpr bool COLS = MODE == DP_COLS, AT = MODE == DP_BLK, LONG = MODE == DP_ROWS, F64 = sizeof(T) == 8;
  constexpr int BM = Dp<T>::BM, BN = Dp<T>::BN, V = Dp<T>::V, STAGE = Dp<T>::STAGE, RP = Dp<T>::RP, EL = sizeof(T);
  extern __shared__ __align__(16) unsigned char dp_raw[];
  T *const dp_smem = reinterpret_cast<T *>(dp_raw);
  __shared__ __align__(16) DpRec recs[DP_RECS];
  __shared__ __align__(16) qc_dcol scols[COLS ? DP_RECS : 1][BN];
  __shared__ __align__(16) long long srow[MODE == DP_ROWS ? DP_RECS : 1][BM];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = (int)gridDim.x;
  const int ntile = (nwork - (int)blockIdx.x + G - 1) / G;
  // tile j of this CTA: every other pass over the grid runs backwards (the list is sorted)
  auto item = [&](int j) {
    const int i = j * G + ((j & 1) ? G - 1 - (int)blockIdx.x : (int)blockIdx.x);
    return i < nwork ? i : j * G + (int)blockIdx.x;
  };
  auto fetch = [&](int j, int2 w) {            // records of tile j into their slot
    if (tid < 6) {
      const char *src = tid < 4 ? reinterpret_cast<const char *>(units + w.x) + 16 * tid
                                : reinterpret_cast<const char *>(ops + w.y) + 16 * (tid - 4);
      const unsigned d = (unsigned)__cvta_generic_to_shared(&recs[j & (DP_RECS - 1)]) + 16u * tid;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    }
  };
  for (int j = 0; j < min(3, ntile); ++j) fetch(j, work[item(j)]);
  asm volatile("cp.async.commit_group;" ::: "memory");
  int2 nw = ntile > 3 ? work[item(3)] : make_int2(0, 0);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  const unsigned sbase = (unsigned)__cvta_generic_to_shared(dp_smem);
  // this thread copies 16 bytes (V values of k) of rows r0, r0 + RP, ... of both operands
  const int ck = V * (tid & (DP_BK / V - 1)), r0 = tid / (DP_BK / V);
  const int cm = 2 * (tid & 63), rk = tid >> 6;      // A given as [K x M]: two m of rows rk, rk + 4, ...
  int lt = 0, lk = 0, lnk, lK, lm, ln, lda, ldb;     // loads: tile, K slice, the tile's extents
  const T *Ab, *Bb;
  auto open_tile = [&]() {
    const DpRec &r = recs[lt & (DP_RECS - 1)];
    lK = r.u.K;
    lnk = max(1, (lK + DP_BK - 1) / DP_BK);
    lm = r.u.mrem;
    ln = r.u.nrem;
    lda = r.u.lda;
    ldb = r.u.ldb;
    Ab = A + r.o.a_base + r.u.a_off + (AT ? (long long)rk * lda + cm : (long long)r0 * lda + ck);
    Bb = B + r.o.b_base + r.u.b_off + (long long)r0 * ldb + ck;
    lk = 0;
    // the tile's column (row) records, read by its epilogue
    if (COLS && tid >= ln && tid < BN) scols[lt & (DP_RECS - 1)][tid].off = -1;
    if (MODE != DP_BLK && (COLS ? tid < ln : tid < lm)) {
      const void *src = COLS ? (const void *)(cols + r.u.c_off + tid) : (const void *)(crow + r.u.c_off + tid);
      const void *dst = COLS ? (const void *)&scols[lt & (DP_RECS - 1)][tid] : (const void *)&srow[lt & (DP_RECS - 1)][tid];
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                   : "memory");
    }
    if (lt + 3 < ntile) {
      fetch(lt + 3, nw);
      if (lt + 4 < ntile) nw = work[item(lt + 4)];
    }
  };
  int ls = 0;                                        // stage of the next load
  auto load = [&]() {
    if (lt < ntile) {
      const int k0 = lk * DP_BK;
      const int kb = max(0, min(V, lK - k0 - ck)) * EL;
      const unsigned s = sbase + (unsigned)(ls * STAGE + r0 * DP_P + ck) * EL;
      const unsigned sb = sbase + (unsigned)(ls * STAGE + (F64 ? dp_col_place(r0) : r0) * DP_P + ck) * EL;
      if (AT) {
        const unsigned sa = sbase + (unsigned)(ls * STAGE + rk * DP_PT + cm) * EL;
        const int mb = max(0, min(2, lm - cm)) * 8;
#pragma unroll
        for (int e = 0; e < DP_BK / 4; ++e) {
          const int v = k0 + rk + 4 * e < lK ? mb : 0;
          dp_cp16(sa + (unsigned)(4 * e * DP_PT) * EL, v ? Ab + (long long)(k0 + 4 * e) * lda : A, v);
        }
      } else {
#pragma unroll
        for (int e = 0; e < BM / RP; ++e) {
          const int v = r0 + RP * e < lm ? kb : 0;
          dp_cp16(s + (unsigned)(RP * e * DP_P) * EL, v ? Ab + (long long)(RP * e) * lda + k0 : A, v);
        }
      }
#pragma unroll
      for (int e = 0; e < (BN + RP - 1) / RP; ++e) {
        const int v = r0 + RP * e < ln ? kb : 0;
        if (BN % RP == 0 || r0 + RP * e < BN)
          dp_cp16(sb + (unsigned)((BM + RP * e) * DP_P) * EL, v ? Bb + (long long)(RP * e) * ldb + k0 : B, v);
      }
      if (++lk == lnk && ++lt < ntile) open_tile();
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    ls = ls + 1 == DP_ST ? 0 : ls + 1;
  };
  open_tile();
  for (int s = 0; s < DP_ST - 1; ++s) {
    load();
    if (lt > 0 && lk == 0) {      // a tile of one K slice: the next records have landed before they are read
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
  }

  // FP64: row lane / 4 and columns lane % 4, lane % 4 + 4 of every 8 x 8 product
  constexpr int WR = BM / 8;                       // rows of a warp
  double acc[2][DP_NT][2];
  unsigned long long facc[8][4];
  auto clear = [&]() {
    if constexpr (F64) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < DP_NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) facc[i][j] = 0ull;
    }
  };
  clear();
  const int gr = F64 ? lane >> 2 : lane >> 3, gk = F64 ? lane & 3 : lane & 7;
  int st = 0;
  for (int ct = 0; ct < ntile; ++ct) {
    const DpRec &rec = recs[ct & (DP_RECS - 1)];
    const int K = rec.u.K, nk = max(1, (K + DP_BK - 1) / DP_BK);
    const int nt = (rec.u.nrem + 7) >> 3;
    const bool live = warp * WR < rec.u.mrem;
    for (int kt = 0; kt < nk; ++kt) {
      asm volatile("cp.async.wait_group %0;" ::"n"(DP_ST - 2) : "memory");
      __syncthreads();
      load();
      if (live) {
        const int k4 = min(DP_BK / 4, (K - kt * DP_BK + 3) >> 2);
        const T *buf = dp_smem + st * STAGE;
        if constexpr (F64) {
          const double *as = buf + (AT ? gk * DP_PT + warp * WR + gr : (warp * WR + gr) * DP_P + gk);
          const double *bs = buf + (BM + gr) * DP_P + gk;
          switch (nt) {
            case 1: dp_slice<1, AT, LONG>(as, bs, k4, acc); break;
            case 2: dp_slice<2, AT, LONG>(as, bs, k4, acc); break;
            case 3: dp_slice<3, AT, LONG>(as, bs, k4, acc); break;
            case 4: dp_slice<4, AT, LONG>(as, bs, k4, acc); break;
            case 5: dp_slice<5, AT, LONG>(as, bs, k4, acc); break;
            case 6: dp_slice<6, AT, LONG>(as, bs, k4, acc); break;
            case 7: dp_slice<7, AT, LONG>(as, bs, k4, acc); break;
            default: dp_slice<8, AT, LONG>(as, bs, k4, acc); break;
          }
        } else {
          const float *as = buf + (warp * WR + gr) * DP_P, *bs = buf + (BM + gk) * DP_P;
          switch (nt) {
            case 1: dp_slice<1>(as, bs, k4, facc); break;
            case 2: dp_slice<2>(as, bs, k4, facc); break;
            case 3: dp_slice<3>(as, bs, k4, facc); break;
            default: dp_slice<4>(as, bs, k4, facc); break;
          }
        }
      }
      st = st + 1 == DP_ST ? 0 : st + 1;
    }
    T *const Cb = C + rec.o.c_base;
    const double alpha = rec.o.alpha;
    const int mrem = rec.u.mrem, nrem = rec.u.nrem;
    if constexpr (!F64) {
      const qc_dcol *cl = scols[COLS ? ct & (DP_RECS - 1) : 0];
      const long long m0 = rec.u.m0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = 8 * j + gk;
        if (n < nrem) {
          const qc_dcol c = COLS ? cl[n] : qc_dcol{};
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int m = warp * WR + 4 * i + gr;
            const float2 v = *reinterpret_cast<const float2 *>(&facc[i][j]);
            if (m < mrem && (!COLS || c.off >= 0))
              Cb[COLS ? c.off + (m0 + m) * c.ld : srow[ct & (DP_RECS - 1)][m] + rec.u.n0 + n] = float(alpha) * (v.x + v.y);
          }
        }
      }
    } else if constexpr (COLS) {
      // eight columns' records first, then their stores under predicates: with a branch for each
      // column its record's latency is paid sixteen times (D = 200: 786 -> 729 us, D = 500: 7.67 -> 7.48 ms)
      const int m = warp * WR + gr, m0 = rec.u.m0 + m;
      const bool r0 = m < mrem, r1 = m + 8 < mrem;
      const qc_dcol *cl = scols[ct & (DP_RECS - 1)] + gk;
#pragma unroll
      for (int j = 0; j < DP_NT; j += 4) {
        qc_dcol c[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) c[q] = cl[8 * j + 4 * q];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          double *dst = Cb + c[q].off + (long long)m0 * c[q].ld;
          const double v0 = alpha * acc[0][j + q / 2][q & 1], v1 = alpha * acc[1][j + q / 2][q & 1];
          if (r0 && c[q].off >= 0) dst[0] = v0;
          if (r1 && c[q].off >= 0) dst[8LL * c[q].ld] = v1;
        }
      }
    } else if constexpr (AT) {
      const int dr = rec.u.pad0, dc = rec.u.pad1, m0 = rec.u.m0, n0 = rec.u.n0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = warp * WR + 8 * i + gr;
        if (m < mrem) {
          const int q = (m0 + m) / dr, r = (m0 + m) - q * dr;
          double *dst = Cb + rec.u.c_off + (long long)q * dr * dc + (long long)n0 * dr + r;
#pragma unroll
          for (int j = 0; j < DP_NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int n = 8 * j + 4 * h + gk;
              if (n < nrem) dst[(long long)n * dr] = alpha * acc[i][j][h];
            }
        }
      }
    } else {
      const int n0 = rec.u.n0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = warp * WR + 8 * i + gr;
        if (m < mrem) {
          double *dst = Cb + srow[ct & (DP_RECS - 1)][m] + n0;
#pragma unroll
          for (int j = 0; j < DP_NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int n = 8 * j + 4 * h + gk;
              if (n < nrem) dst[n] = alpha * acc[i][j][h];
            }
        }
      }
    }
    clear();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// out[i] = x[idx[i]] (rounded to T), 0 where idx < 0
template <typename T>
__global__ void k_gather_pad(const double *__restrict__ x, const long long *__restrict__ idx, long long n,
                             T *__restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long j = idx[i];
    out[i] = j >= 0 ? T(x[j]) : T(0);
  }
}

}  // namespace

template <typename T, int MODE>
static cudaError_t launch_dpanel(const void *units, const void *work, int nwork, const void *ops,
                                 const long long *crow, const void *cols, const T *A, const T *B, T *C,
                                 cudaStream_t s) {
  // the shared-memory limit of a kernel and the SM count are properties of a device: asked once for each
  static std::atomic<int> sms[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int nsm = dev < 64 ? sms[dev].load(std::memory_order_relaxed) : 0;
  if (nsm == 0) {
    e = cudaFuncSetAttribute(k_dpanel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, Dp<T>::SMEM);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (dev < 64) sms[dev].store(nsm, std::memory_order_relaxed);
  }
  // short panels (L.psi, the renormalisation's) share a persistent grid; the long ones of .R,
  // sorted by length, are left to the hardware's scheduler, one tile per CTA (K = 24, D = 500:
  // 5.7 against 6.8 ms)
  k_dpanel<T, MODE><<<MODE != DP_ROWS && nwork > 2 * nsm ? 2 * nsm : nwork, DP_THREADS, Dp<T>::SMEM, s>>>(
      (const qc_dunit *)units, (const int2 *)work, nwork, (const qc_op *)ops, crow, (const qc_dcol *)cols, A, B, C);
  return cudaGetLastError();
}

template <typename T>
static int run_dpanel(const void *units, const void *work, long long nwork, const void *ops, const long long *crow,
                      const void *cols, const T *A, const T *B, T *C, void *stream) {
  if (nwork <= 0) return QC_OK;
  if (nwork > 0x3fffffffLL || !units || !work || !ops || (crow && cols) || (sizeof(T) == 4 && !crow && !cols) ||
      ((unsigned long long)A & 15) || ((unsigned long long)B & 15))
    return QC_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e;
  if (cols)
    e = launch_dpanel<T, DP_COLS>(units, work, (int)nwork, ops, crow, cols, A, B, C, s);
  else if (sizeof(T) == 4 || crow)
    e = launch_dpanel<T, DP_ROWS>(units, work, (int)nwork, ops, crow, cols, A, B, C, s);
  else if constexpr (sizeof(T) == 8)
    e = launch_dpanel<T, DP_BLK>(units, work, (int)nwork, ops, crow, cols, A, B, C, s);
  if (e != cudaSuccess) {
    fprintf(stderr, "[qcgpu] qc_dpanel: %s\n", cudaGetErrorString(e));
    return QC_ERR_CUDA;
  }
  return QC_OK;
}

extern "C" int qc_dpanel_f64(const void *units, const void *work, long long nwork, const void *ops,
                             const long long *crow, const void *cols, const double *A, const double *B, double *C,
                             void *stream) {
  return run_dpanel(units, work, nwork, ops, crow, cols, A, B, C, stream);
}

extern "C" int qc_dpanel_f32(const void *units, const void *work, long long nwork, const void *ops,
                             const long long *crow, const void *cols, const float *A, const float *B, float *C,
                             void *stream) {
  return run_dpanel(units, work, nwork, ops, crow, cols, A, B, C, stream);
}

template <typename T>
static int run_gather_pad(const double *x, const long long *idx, long long n, T *out, void *stream) {
  if (n <= 0) return QC_OK;
  if (!x || !idx || !out) return QC_ERR_ARG;
  long long blocks = (n + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  k_gather_pad<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(x, idx, n, out);
  return cudaGetLastError() == cudaSuccess ? QC_OK : QC_ERR_CUDA;
}

extern "C" int qc_gather_pad_f64(const double *x, const long long *idx, long long n, double *out, void *stream) {
  return run_gather_pad(x, idx, n, out, stream);
}

extern "C" int qc_gather_pad_f32(const double *x, const long long *idx, long long n, float *out, void *stream) {
  return run_gather_pad(x, idx, n, out, stream);
}
