// The two MPO-site contractions of sigma as one sparse product: T3 = T1 . (W_i W_{i+1})
// (top2 and top3 of HVecQt, source/mpo_dmrg_kernelQt.py:303-306), without the
// intermediate T2.
//
// A fiber is one (l, r) pair of bond states.  For one fiber the two contractions are a
// matrix S[k, i] from its T1 rows i = (a, n1, n2) to its T3 rows k = (c, n1', n2'), and
// every fiber of one charge difference q(l) - q(r) meets the same S.  An ab-initio MPO
// fills about a tenth of the blocks of S that symmetry allows (K = 24: 20 310 of 230 000
// elements per operator, 13 per row k, against 74 multiply-adds per element of the two
// dense block contractions), so S is kept as lists: rows k of like pattern in octets, and for
// every octet the T1 rows that any of the eight reads with their eight coefficients.
//
// One CTA takes a tile of 32, 64 or 128 fibers of one charge difference (fibers of several
// sector pairs share a tile, so small sectors fill the lanes) and walks operators: the
// tile's T1 rows are staged in shared memory (cp.async, rows contiguous over fibers), then
// every warp takes octets of S.  T3 keeps r as its fastest index, so results leave as
// contiguous rows straight from registers.  Two CTAs share an SM: one loads while the
// other multiplies.
//
// Bound: T1 read and T3 written once.  Mid-chain dot of K=24, D=500 (1.22e9 elements each: 19.5 GB
// in FP64, 3.0 ms, and half of that in FP32): two dense stages took 30.2 ms in FP64 and 15.5 ms in
// FP32, lists of four consecutive rows on scalar multiply-adds 8.1 and 4.6 ms (shared-memory pipe
// 72 % busy: a row read and a coefficient broadcast for every four rows), octets of like rows
// 6.0 and 4.05 ms (D = 200: 1.37 -> 1.00, 0.78 -> 0.71 ms), 6.07 and 4.09 (1.00, 0.72) since an octet
// ends where the T1 blocks that reach its rows change.  FP32 is still bound by the shared-memory
// pipe (75 %); copying alone takes 2.2 and 1.3 ms of it.  Twelve warps of deeper prefetch: 5.99, 4.11.
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>
#include "qc_types.h"

namespace {

constexpr int WX_WARPS = 16;
constexpr int WX_THREADS = 32 * WX_WARPS;
constexpr int WX_MAXOCT = 512;            // octets of one (delta, operator)
constexpr int WX_GRPS = 32;               // sector pairs of one tile
constexpr int WX_MAXSMEM = 224 * 1024;

__device__ __forceinline__ void cp_async_el(float *dst, const float *src, bool valid) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_el(double *dst, const double *src, bool valid) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_16(void *dst, const void *src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// Row pitch of the staged tile: FP32 lanes read consecutive fibers of one row; an FP64
// fragment reads eight fibers of four rows, which touch every bank once when the rows differ
// mod 4 (the entry lists are ordered that way) and the pitch is 4 mod 16.
template <typename T, int FT>
__host__ __device__ constexpr int wx_pitch() { return sizeof(T) == 8 ? FT + 4 : FT; }

// A warp's units of work: (octet, group of GW of the tile's fibers), octets by decreasing
// length; every other pass over the warps runs backwards, which evens out their loads.
__device__ __forceinline__ int wx_unit(int pass, int warp) {
  return pass * WX_WARPS + ((pass & 1) ? WX_WARPS - 1 - warp : warp);
}

// Offsets of a tile's fibers: T1 block (n1, n2) and T3 block (n1', n2') of every fiber (-1: absent,
// or past the tile), its T1 row stride F and its T3 row stride D_r.
template <int FT>
struct alignas(16) WxTile {
  int a[16][FT], c[16][FT];
  int F[FT], flo[FT];
};

template <typename T, int FT>
__host__ __device__ constexpr size_t wx_fixed_smem() {
  return sizeof(WxTile<FT>) + (sizeof(T) == 4 ? (size_t)WX_WARPS * 32 * 36 : 0);     // FP32: entry rings
}

template <int FT>
__device__ __forceinline__ void wx_open_tile(WxTile<FT> &w, const qc_wxitem &it, const qc_wxgrp *__restrict__ grps,
                                             int grp_e) {
  __shared__ int s_start[WX_GRPS + 1], s_slot[FT], s_f[FT];
  const int tid = threadIdx.x;
  for (int t = tid; t <= WX_GRPS; t += WX_THREADS)
    s_start[t] = (t < WX_GRPS && it.grp + t < grp_e) ? grps[it.grp + t].start : 0x7fffffff;
  __syncthreads();
  for (int t = tid; t < FT; t += WX_THREADS) {
    const int pos = s_start[0] + it.f0 + t;
    int lo = 0, hi = WX_GRPS - 1;                // largest k with start[k] <= pos
    while (lo < hi) {
      const int m = (lo + hi + 1) >> 1;
      if (s_start[m] <= pos) lo = m; else hi = m - 1;
    }
    s_slot[t] = t < it.nf ? it.grp + lo : -1;
    s_f[t] = pos - s_start[lo];
  }
  __syncthreads();
  for (int e = tid; e < 16 * FT; e += WX_THREADS) {
    const int b = e / FT, t = e - b * FT, g = s_slot[t];
    int oa = -1, oc = -1;
    if (g >= 0) {
      const qc_wxgrp *gr = grps + g;
      const int f = s_f[t], flo = gr->flo;
      oa = gr->a[b];
      if (oa >= 0) oa += f;
      oc = gr->c[b];
      if (oc >= 0) oc += (f / flo) * gr->h[b] + f % flo;
      if (b == 0) {
        w.F[t] = gr->F;
        w.flo[t] = flo;
      }
    } else if (b == 0) {
      w.F[t] = w.flo[t] = 0;
    }
    w.a[b][t] = oa;
    w.c[b][t] = oc;
  }
  __syncthreads();
}

// The tile's T1 rows and the operator's octet records on their way to shared memory.
template <typename T, int FT>
__device__ __forceinline__ void wx_stage(const WxTile<FT> &w, const int *rowt, int R, const T *Ao, T *As,
                                         const qc_wxoct *go, qc_wxoct *so, int no) {
  constexpr int P = wx_pitch<T, FT>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int F[FT / 32];
#pragma unroll
  for (int j = 0; j < FT / 32; ++j) F[j] = w.F[lane + 32 * j];
#pragma unroll 2
  for (int r = warp; r < R; r += WX_WARPS) {
    const int rec = rowt[r], a = rec & 0xffff;
    const int *ta = w.a[rec >> 16] + lane;
#pragma unroll
    for (int j = 0; j < FT / 32; ++j) {
      const int off = ta[32 * j];
      cp_async_el(As + r * P + lane + 32 * j, Ao + (off >= 0 ? off + a * F[j] : 0), off >= 0);
    }
  }
  for (int e = threadIdx.x; e < no * (int)(sizeof(qc_wxoct) / 16); e += WX_THREADS)
    cp_async_16(reinterpret_cast<char *>(so) + 16 * e, reinterpret_cast<const char *>(go) + 16 * e);
  asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ void wx_ffma2(unsigned long long &c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// FP32: lane = fiber (FT / 32 of them); an entry is one row read per fiber against eight
// broadcast coefficients, packed in pairs (fma.rn.f32x2: two multiply-adds an issue slot).
template <int FT, int GW>
__global__ void __launch_bounds__(WX_THREADS, 2)
k_wsparse_f32(const qc_wxitem *__restrict__ items, const qc_wxdelta *__restrict__ deltas,
              const qc_wxgrp *__restrict__ grps, const int *__restrict__ rows, const qc_wxdop *__restrict__ dops,
              const qc_wxoct *__restrict__ octs, const float4 *__restrict__ ent_w, const int *__restrict__ ent_r,
              const qc_op *__restrict__ ops, int maxR, int maxO, const float *__restrict__ A, float *__restrict__ C) {
  constexpr int NJ = GW / 32, NG = FT / GW;
  extern __shared__ __align__(16) unsigned char wx_smem[];
  WxTile<FT> &w = *reinterpret_cast<WxTile<FT> *>(wx_smem);
  float4 *const ring0 = reinterpret_cast<float4 *>(&w + 1);                            // [warps][2][32]
  int *const ringr0 = reinterpret_cast<int *>(ring0 + WX_WARPS * 64);                  // [warps][32]
  qc_wxoct *const so = reinterpret_cast<qc_wxoct *>(ringr0 + WX_WARPS * 32);           // [maxO]
  float *const As = reinterpret_cast<float *>(so + maxO);                              // [R + 4][FT], last rows zero
  int *const rowt = reinterpret_cast<int *>(As + (size_t)(maxR + 4) * FT);            // [maxR]

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const qc_wxitem it = items[blockIdx.x];
  const qc_wxdelta *const dl = deltas + it.delta;
  const int R = dl->R, dop_b = dl->dop_b;
  for (int r = tid; r < R; r += WX_THREADS) rowt[r] = rows[dl->row_b + r];
  for (int t = tid; t < 4 * FT; t += WX_THREADS) As[R * FT + t] = 0.f;
  wx_open_tile<FT>(w, it, grps, dl->grp_e);
  float4 *const ring = ring0 + warp * 64;
  int *const ringr = ringr0 + warp * 32;
  for (int op = it.op_b; op < it.op_e; ++op) {
    const qc_op o = ops[op];
    const qc_wxdop dop = dops[dop_b + op - it.op0];
    const int no = dop.noct;
    const qc_wxoct *const go = octs + dop.oct_b;
    wx_stage<float, FT>(w, rowt, R, A + o.a_base, As, go, so, no);
    const float4 *const ew = ent_w + 2 * dop.ent_b;
    const int *const er = ent_r + dop.ent_b;
    float *const Co = C + o.c_base;
    // the warp's first octet and its first entries, while the rows are in flight (a list's
    // length is a multiple of four: it ends in zero rows with zero coefficients)
    float4 p0, p1;
    int pr = 0;
    auto fetch = [&](int first, int cnt) {
      if (lane < cnt) {
        p0 = ew[2 * (first + lane)];
        p1 = ew[2 * (first + lane) + 1];
        pr = er[first + lane];
      }
    };
    const int nu = no * NG;
    int pass = 0, u = wx_unit(0, warp), ent = 0, cnt = 0;
    if (u < nu) {
      ent = go[u / NG].ent;
      cnt = go[u / NG].cnt;
      fetch(ent, cnt);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    while (u < nu) {
      const int q = u / NG, g0 = (u % NG) * GW + lane, n0 = cnt;
      int e0 = ent;
      u = wx_unit(++pass, warp);
      if (u < nu) {
        ent = so[u / NG].ent;
        cnt = so[u / NG].cnt;
      } else {
        cnt = 0;
      }
      unsigned long long acc[4][NJ];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[k][j] = 0ull;
      for (int left = n0;;) {
        const int n = min(32, left);
        ring[lane] = p0;
        ring[32 + lane] = p1;
        ringr[lane] = pr * FT;
        __syncwarp();
        left -= n;
        e0 += n;
        if (left > 0)
          fetch(e0, left);
        else
          fetch(ent, cnt);
        for (int e = 0; e < n; e += 4) {
          const int4 r4 = *reinterpret_cast<const int4 *>(ringr + e);
          const int rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const ulonglong2 wl = *reinterpret_cast<const ulonglong2 *>(ring + e + x);
            const ulonglong2 wh = *reinterpret_cast<const ulonglong2 *>(ring + 32 + e + x);
            const float *a = As + rr[x] + g0;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
              const float v = a[32 * j];
              unsigned long long vv;
              asm("mov.b64 %0, {%1, %1};" : "=l"(vv) : "f"(v));
              wx_ffma2(acc[0][j], wl.x, vv);
              wx_ffma2(acc[1][j], wl.y, vv);
              wx_ffma2(acc[2][j], wh.x, vv);
              wx_ffma2(acc[3][j], wh.y, vv);
            }
          }
        }
        __syncwarp();
        if (left <= 0) break;
      }
      // ---- eight rows, each of its own block; fibers of one l are contiguous
      int fl[NJ];
#pragma unroll
      for (int j = 0; j < NJ; ++j) fl[j] = w.flo[g0 + 32 * j];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int row = so[q].row[k];
        if (row < 0) break;
        const int *tc = w.c[row >> 16] + g0;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const int off = tc[32 * j];
          if (off >= 0)
            Co[off + (row & 0xffff) * fl[j]] = __uint_as_float((unsigned)(acc[k >> 1][j] >> (k & 1 ? 32 : 0)));
        }
      }
    }
    __syncthreads();
  }
}

// FP64: an octet's four entries against eight fibers are one m8n8k4 product on the FP64
// tensor pipe (T1 rows x coefficients); the coefficients come from global memory in fragment
// order, one value per lane, three steps ahead.
template <int FT>
__global__ void __launch_bounds__(WX_THREADS, 2)
k_wsparse_f64(const qc_wxitem *__restrict__ items, const qc_wxdelta *__restrict__ deltas,
              const qc_wxgrp *__restrict__ grps, const int *__restrict__ rows, const qc_wxdop *__restrict__ dops,
              const qc_wxoct *__restrict__ octs, const double *__restrict__ ent_w, const int *__restrict__ ent_r,
              const qc_op *__restrict__ ops, int maxR, int maxO, const double *__restrict__ A,
              double *__restrict__ C) {
  constexpr int GW = 32, NG = FT / GW, NT = GW / 8, P = wx_pitch<double, FT>();
  extern __shared__ __align__(16) unsigned char wx_smem[];
  WxTile<FT> &w = *reinterpret_cast<WxTile<FT> *>(wx_smem);
  qc_wxoct *const so = reinterpret_cast<qc_wxoct *>(&w + 1);                           // [maxO]
  double *const As = reinterpret_cast<double *>(so + maxO);                            // [R + 4][P], last rows zero
  int *const rowt = reinterpret_cast<int *>(As + (size_t)(maxR + 4) * P);             // [maxR]

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gr = lane >> 2, gk = lane & 3;
  const qc_wxitem it = items[blockIdx.x];
  const qc_wxdelta *const dl = deltas + it.delta;
  const int R = dl->R, dop_b = dl->dop_b;
  for (int r = tid; r < R; r += WX_THREADS) rowt[r] = rows[dl->row_b + r];
  for (int t = tid; t < 4 * P; t += WX_THREADS) As[R * P + t] = 0.0;
  wx_open_tile<FT>(w, it, grps, dl->grp_e);
  for (int op = it.op_b; op < it.op_e; ++op) {
    const qc_op o = ops[op];
    const qc_wxdop dop = dops[dop_b + op - it.op0];
    const int no = dop.noct;
    const qc_wxoct *const go = octs + dop.oct_b;
    wx_stage<double, FT>(w, rowt, R, A + o.a_base, As, go, so, no);
    const double *const ew = ent_w + 8 * dop.ent_b + lane;       // step s: [32 s]
    const int *const er = ent_r + dop.ent_b + gk;                // step s: [4 s]
    double *const Co = C + o.c_base;
    // the stream of this warp's steps, unit after unit, three steps ahead (an octet has one at
    // least: fe counts steps from the operator's first, fl ends the current unit's)
    const qc_wxoct *fo = go;                     // records: global memory until the staged ones are in
    const int nu = no * NG;
    int fp = 0, fu = wx_unit(0, warp), fe = 0, fl = 0;
    if (fu < nu) {
      fe = go[fu / NG].ent >> 2;
      fl = fe + (go[fu / NG].cnt >> 2);
    }
    auto fetch = [&](double &wv, int &rv) {
      if (fe < fl) {
        wv = ew[32 * fe];
        rv = er[4 * fe];
        if (++fe == fl) {
          fu = wx_unit(++fp, warp);
          if (fu < nu) {
            fe = fo[fu / NG].ent >> 2;
            fl = fe + (fo[fu / NG].cnt >> 2);
          }
        }
      }
    };
    double w0 = 0.0, w1 = 0.0, w2 = 0.0;
    int r0 = R, r1 = R, r2 = R;
    fetch(w0, r0);
    fetch(w1, r1);
    fetch(w2, r2);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    fo = so;
    int pass = 0, u = wx_unit(0, warp), left = 0, g0 = 0;
    double acc[NT][2];
    auto open_unit = [&]() {
      if (u < nu) {
        left = so[u / NG].cnt >> 2;
        g0 = (u % NG) * GW + gr;
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = 0.0;
      }
    };
    auto step = [&](double wv, int r) {
      const double *a = As + r * P + g0;
      double av[NT];
#pragma unroll
      for (int t = 0; t < NT; ++t) av[t] = a[8 * t];
#pragma unroll
      for (int t = 0; t < NT; ++t)
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                     : "+d"(acc[t][0]), "+d"(acc[t][1])
                     : "d"(av[t]), "d"(wv));
      if (--left == 0) {
        // lane: fiber 8 t + lane / 4 of every t, rows 2 (lane % 4) and the next one
        const qc_wxoct &x = so[u / NG];
        const int ra = x.row[2 * gk], rb = x.row[2 * gk + 1];
        const int *ta = w.c[max(ra, 0) >> 16] + g0, *tb = w.c[max(rb, 0) >> 16] + g0;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int fl = w.flo[g0 + 8 * t], oa = ta[8 * t], ob = tb[8 * t];
          if (ra >= 0 && oa >= 0) Co[oa + (ra & 0xffff) * fl] = acc[t][0];
          if (rb >= 0 && ob >= 0) Co[ob + (rb & 0xffff) * fl] = acc[t][1];
        }
        u = wx_unit(++pass, warp);
        open_unit();
      }
    };
    open_unit();
    // each of the three prefetched steps keeps its registers: a copy would wait for its load
    while (u < nu) {
      step(w0, r0);
      fetch(w0, r0);
      if (u >= nu) break;
      step(w1, r1);
      fetch(w1, r1);
      if (u >= nu) break;
      step(w2, r2);
      fetch(w2, r2);
    }
    __syncthreads();
  }
}

template <typename T, int FT>
size_t wx_smem_bytes(int maxR, int maxO) {
  return (size_t)(maxR + 4) * wx_pitch<T, FT>() * sizeof(T) + (size_t)maxO * sizeof(qc_wxoct) +
         (size_t)maxR * sizeof(int) + wx_fixed_smem<T, FT>();
}

struct WxArgs {
  const void *items;
  long long nitems;
  const void *deltas, *grps, *rows, *dops, *octs, *ent_w, *ent_r, *ops;
  int maxR, maxO;
};

template <typename T, typename W, auto Kernel>
int launch_kernel(size_t smem, const WxArgs &x, const T *A, T *C, cudaStream_t s) {
  if (smem > WX_MAXSMEM) return QC_ERR_ARG;
  // the limit belongs to a kernel on a device: raised once for each
  static std::atomic<bool> raised[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && (dev >= 64 || !raised[dev].load(std::memory_order_relaxed))) {
    e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WX_MAXSMEM);
    if (e == cudaSuccess && dev < 64) raised[dev].store(true, std::memory_order_relaxed);
  }
  if (e == cudaSuccess) {
    Kernel<<<(unsigned)x.nitems, WX_THREADS, smem, s>>>(
        (const qc_wxitem *)x.items, (const qc_wxdelta *)x.deltas, (const qc_wxgrp *)x.grps, (const int *)x.rows,
        (const qc_wxdop *)x.dops, (const qc_wxoct *)x.octs, (const W *)x.ent_w, (const int *)x.ent_r,
        (const qc_op *)x.ops, x.maxR, x.maxO, A, C);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    fprintf(stderr, "[qcgpu] qc_wsparse: %s\n", cudaGetErrorString(e));
    return QC_ERR_CUDA;
  }
  return QC_OK;
}

bool wx_bad(const WxArgs &x) {
  return x.nitems > 0x7fffffffLL || !x.items || !x.deltas || !x.grps || !x.rows || !x.dops || !x.octs || !x.ent_w ||
         !x.ent_r || !x.ops || x.maxR < 0 || x.maxO < 0 || x.maxO > WX_MAXOCT;
}

// ---- host: the sparse rows of S = W_i W_{i+1} for every (delta, operator) of one class
struct Nz {
  int j;
  double v;
};

// A packed W tensor [a, b, n', n] of one class; row0: where an allowed block's rows a stand in a
// NzRows (-1: not allowed), rows: all of them.
struct SparseW {
  int ns[4];
  const long long *nd[4];
  const long long *ioff;
  const int *allowed;
  std::vector<int> row0;
  int rows = 0;
  long long size = 0;          // elements of an operator

  void number_rows() {
    const int per = ns[1] * ns[2] * ns[3], nb = ns[0] * per;
    row0.assign(nb, -1);
    for (int b = 0; b < nb; ++b)
      if (allowed[b]) {
        row0[b] = rows;
        rows += (int)nd[0][b / per];
        size += nd[0][b / per] * nd[1][b / (ns[2] * ns[3]) % ns[1]];
      }
  }
};

// the non-zeros of one operator's tensor, row by row of its allowed blocks
struct NzRows {
  std::vector<int> start;
  std::unique_ptr<Nz[]> nz;
};

struct OpLists {
  std::vector<qc_wxdop> dops;
  std::vector<qc_wxoct> octs;
  std::vector<double> w;       // four entries a step: [step][row][entry of the step]
  std::vector<int> r;
};

void list_rows(const SparseW &W, const double *val, NzRows &out) {
  const int per = W.ns[1] * W.ns[2] * W.ns[3], nb = W.ns[0] * per;
  out.start.reserve(W.rows + 1);
  out.nz.reset(new Nz[W.size + 1]);
  Nz *q = out.nz.get();
  for (int b = 0; b < nb; ++b) {
    if (W.row0[b] < 0) continue;
    const int na = (int)W.nd[0][b / per], nbb = (int)W.nd[1][b / (W.ns[2] * W.ns[3]) % W.ns[1]];
    const double *p = val + W.ioff[b];
    for (int a = 0; a < na; ++a, p += nbb) {
      out.start.push_back((int)(q - out.nz.get()));
      for (int j = 0; j < nbb; ++j) {        // (written always: a branch is mispredicted at every other non-zero)
        *q = Nz{j, p[j]};
        q += p[j] != 0.0;
      }
    }
  }
  out.start.push_back((int)(q - out.nz.get()));
}

// What the rows of one delta are made of, for every operator of the class: products of the blocks
// (T1 block ib, MPO sector sb) -> T3 block kb that symmetry allows, and the rows' blocks.
struct DeltaPlan {
  struct Product {
    int k0, i0, na, r1, r2;    // first row k, first row i, rows i, rows of both blocks in their NzRows
  };
  int R, nrow = 0;
  std::vector<Product> products;
  std::vector<int> rowid, reach;     // block << 16 | c; T1 blocks that reach the row (one bit each)
};

void plan_deltas(const SparseW &W1, const SparseW &W2, int ndelta, const int *iblk, const int *kblk, const int *row0,
                 const int *Rs, std::vector<DeltaPlan> &out) {
  // sectors sb that (sa, n1', n1) connects to
  std::vector<std::vector<int>> via((size_t)W1.ns[0] * 16);
  for (int sa = 0; sa < W1.ns[0]; ++sa)
    for (int sb = 0; sb < W1.ns[1]; ++sb)
      for (int n = 0; n < 16; ++n)
        if (W1.row0[(sa * W1.ns[1] + sb) * 16 + n] >= 0) via[16 * sa + n].push_back(sb);
  out.resize(ndelta);
  for (int d = 0; d < ndelta; ++d) {
    DeltaPlan &x = out[d];
    x.R = Rs[d];
    for (int kb = 0; kb < 16; ++kb) {
      const int sc = kblk[16 * d + kb];
      if (sc < 0) continue;
      int reach = 0;
      for (int ib = 0; ib < 16; ++ib) {
        const int sa = iblk[16 * d + ib];
        if (sa < 0) continue;
        const int n = 4 * (kb >> 2) + (ib >> 2), m = 4 * (kb & 3) + (ib & 3);       // (n1', n1), (n2', n2)
        for (int sb : via[16 * sa + n]) {
          const int r1 = W1.row0[(sa * W1.ns[1] + sb) * 16 + n], r2 = W2.row0[(sb * W2.ns[1] + sc) * 16 + m];
          if (r2 < 0) continue;
          reach |= 1 << ib;
          x.products.push_back({x.nrow, row0[16 * d + ib], (int)W1.nd[0][sa], r1, r2});
        }
      }
      for (int c = 0; c < (int)W2.nd[1][sc]; ++c) x.rowid.push_back(kb << 16 | c);
      x.nrow = (int)x.rowid.size();
      x.reach.resize(x.nrow, reach);
    }
  }
}

void build_op(const SparseW &W1, const double *v1, const SparseW &W2, const double *v2,
              const std::vector<DeltaPlan> &deltas, OpLists &out) {
  NzRows l1, l2;
  list_rows(W1, v1, l1);
  list_rows(W2, v2, l2);
  std::vector<double> S;                 // rows of the current delta, dense in i
  std::vector<uint64_t> mask;
  std::vector<int> nnz, perm, bucket[4];
  std::vector<qc_wxoct> os;
  for (const DeltaPlan &dp : deltas) {
    const int R = dp.R, nrow = dp.nrow;
    const int words = (R + 63) / 64;
    const std::vector<int> &rowid = dp.rowid, &reach = dp.reach;
    S.assign((size_t)nrow * R, 0.0);
    mask.assign((size_t)nrow * words, 0);
    for (const auto &p : dp.products)
      for (int a = 0; a < p.na; ++a) {
        const int i = p.i0 + a;
        for (int x = l1.start[p.r1 + a]; x < l1.start[p.r1 + a + 1]; ++x) {
          const Nz u = l1.nz[x];
          for (int y = l2.start[p.r2 + u.j]; y < l2.start[p.r2 + u.j + 1]; ++y) {
            const Nz w = l2.nz[y];
            S[(size_t)(p.k0 + w.j) * R + i] += u.v * w.v;
            mask[(size_t)(p.k0 + w.j) * words + (i >> 6)] |= 1ull << (i & 63);
          }
        }
      }
    // products that cancelled exactly are no entries
    nnz.assign(nrow, 0);
    for (int k = 0; k < nrow; ++k)
      for (int wd = 0; wd < words; ++wd) {
        uint64_t m = mask[(size_t)k * words + wd], live = 0;
        while (m) {
          const int bit = __builtin_ctzll(m);
          m &= m - 1;
          if (S[(size_t)k * R + wd * 64 + bit] != 0.0) live |= 1ull << bit;
        }
        mask[(size_t)k * words + wd] = live;
        nnz[k] += __builtin_popcountll(live);
      }
    // rows of like pattern share an octet: longest first, equal patterns side by side.  A row's zero
    // coefficients meet the T1 rows of the other seven, so only rows that the same T1 blocks can
    // reach share one: an Inf or NaN of a T1 row then gets no further than in the two block products
    perm.resize(nrow);
    for (int k = 0; k < nrow; ++k) perm[k] = k;
    std::stable_sort(perm.begin(), perm.end(), [&](int x, int y) {
      if (reach[x] != reach[y]) return reach[x] > reach[y];
      if (nnz[x] != nnz[y]) return nnz[x] > nnz[y];
      for (int wd = 0; wd < words; ++wd) {
        const uint64_t mx = mask[(size_t)x * words + wd], my = mask[(size_t)y * words + wd];
        if (mx != my) return mx > my;
      }
      return false;
    });
    qc_wxdop rec;
    rec.ent_b = (long long)out.r.size();
    rec.oct_b = (int)out.octs.size();
    os.clear();
    for (int k0 = 0, nk; k0 < nrow; k0 += nk) {
      for (nk = 1; nk < std::min(8, nrow - k0) && reach[perm[k0 + nk]] == reach[perm[k0]];) ++nk;
      qc_wxoct x;
      memset(&x, 0, sizeof(x));
      x.ent = (int)((long long)out.r.size() - rec.ent_b);
      for (int k = 0; k < 8; ++k) x.row[k] = k < nk ? rowid[perm[k0 + k]] : -1;
      // the T1 rows any of the eight reads, in fours of different residues mod 4 where possible
      for (auto &b : bucket) b.clear();
      for (int wd = 0; wd < words; ++wd) {
        uint64_t m = 0;
        for (int k = 0; k < nk; ++k) m |= mask[(size_t)perm[k0 + k] * words + wd];
        while (m) {
          const int i = wd * 64 + __builtin_ctzll(m);
          m &= m - 1;
          bucket[i & 3].push_back(i);
        }
      }
      int rest = (int)(bucket[0].size() + bucket[1].size() + bucket[2].size() + bucket[3].size());
      // (one step of zero rows for an octet without entries)
      for (bool first = true; first || rest > 0; first = false) {
        bool used[4] = {false, false, false, false};
        out.w.resize(out.w.size() + 32, 0.0);
        double *const w = out.w.data() + out.w.size() - 32;
        for (int e = 0; e < 4; ++e) {
          int best = -1;
          for (int b = 0; b < 4; ++b)
            if (!used[b] && !bucket[b].empty() && (best < 0 || bucket[b].size() > bucket[best].size())) best = b;
          if (best < 0) {                         // residues used up: any row that is left
            for (int b = 0; b < 4; ++b)
              if (!bucket[b].empty() && (best < 0 || bucket[b].size() > bucket[best].size())) best = b;
          }
          if (best < 0) {                         // none left: a zero row of an unused residue
            int z = 0;
            while (z < 3 && used[(R + z) & 3]) ++z;
            used[(R + z) & 3] = true;
            out.r.push_back(R + z);
            continue;
          }
          used[best] = true;
          const int i = bucket[best].back();
          bucket[best].pop_back();
          --rest;
          out.r.push_back(i);
          for (int k = 0; k < nk; ++k) w[4 * k + e] = S[(size_t)perm[k0 + k] * R + i];
        }
      }
      x.cnt = (int)((long long)out.r.size() - rec.ent_b) - x.ent;
      os.push_back(x);
    }
    std::stable_sort(os.begin(), os.end(), [](const qc_wxoct &x, const qc_wxoct &y) { return x.cnt > y.cnt; });
    out.octs.insert(out.octs.end(), os.begin(), os.end());
    rec.noct = (int)os.size();
    out.dops.push_back(rec);
  }
}

struct WxBuild {
  struct Part {
    SparseW W1, W2;
    std::vector<DeltaPlan> deltas;
    const qc_wxpart *in;
    long long op0;
  };
  std::vector<Part> parts;
  std::vector<OpLists> ops;      // of all parts
};

// f(0) .. f(n - 1) on the host's threads; false if one of them threw.  The caller waits for the
// items, not for the threads: a CPU of a shared host that has to wake can take a scheduler tick
// or two to start one, which then finds nothing left.  Renormalisations from the right at K=24, D=16
// and 60 took 7.9 ms in the median with a join of the threads, in steps of 4 ms; 5.2 and 5.7 ms now
// (with the deltas planned once a class and the exchanged bonds kept, 7.3 and 7.4 without either).
// A thread touches f only for an item, and so only while the caller waits for it.
template <typename F>
bool wx_each(long long n, const F &f) {
  struct State {
    std::atomic<long long> next{0}, done{0};
    std::atomic<bool> bad{false};
    std::mutex m;
    std::condition_variable all;
  };
  const auto st = std::make_shared<State>();
  const F *const fp = &f;
  auto loop = [st, n, fp]() {
    for (long long i; (i = st->next.fetch_add(1)) < n;) {
      try {
        (*fp)(i);
      } catch (...) {
        st->bad = true;
      }
      if (st->done.fetch_add(1) + 1 == n) {
        std::lock_guard<std::mutex> l(st->m);
        st->all.notify_one();
      }
    }
  };
  const long long hw = std::max(1u, std::thread::hardware_concurrency());
  try {
    for (long long k = 1; k < std::min({8ll, hw, n / 4}); ++k) std::thread(loop).detach();
  } catch (...) {              // no more threads: the others do their share
  }
  loop();
  std::unique_lock<std::mutex> l(st->m);
  st->all.wait(l, [&]() { return st->done.load() >= n; });
  return !st->bad;
}

}  // namespace

// Sparse rows of W_i W_{i+1} for the operators of the given classes (qc_wxpart).  Returns per class
// the octets and entries to fetch with qc_wx_fetch, which frees the handle; the parts' arrays
// have to stay until then.
extern "C" int qc_wx_build(int nparts, const void *parts, void **handle, long long *nocts, long long *nents) {
  if (nparts < 1 || !parts || !handle || !nocts || !nents) return QC_ERR_ARG;
  const qc_wxpart *in = (const qc_wxpart *)parts;
  WxBuild *h = nullptr;
  try {
    h = new WxBuild;
    h->parts.resize(nparts);
    long long nops = 0;
    int rc = QC_OK;
    for (int q = 0; q < nparts && rc == QC_OK; ++q) {
      const qc_wxpart &x = in[q];
      if (x.nops < 1 || x.ndelta < 0 || !x.w1 || !x.off1 || !x.ns1 || !x.nd1 || !x.ioff1 || !x.allowed1 || !x.w2 ||
          !x.off2 || !x.ns2 || !x.nd2 || !x.ioff2 || !x.allowed2 ||
          (x.ndelta && (!x.iblk || !x.kblk || !x.row0 || !x.R))) {
        rc = QC_ERR_ARG;
        break;
      }
      if (x.ns1[2] != 4 || x.ns1[3] != 4 || x.ns2[2] != 4 || x.ns2[3] != 4 || x.ns1[1] != x.ns2[0]) {
        rc = QC_ERR_LAYOUT;
        break;
      }
      WxBuild::Part &p = h->parts[q];
      p.in = &x;
      p.op0 = nops;
      nops += x.nops;
      const long long *p1 = x.nd1, *p2 = x.nd2;
      for (int k = 0; k < 4; ++k) {
        p.W1.ns[k] = x.ns1[k];
        p.W2.ns[k] = x.ns2[k];
        p.W1.nd[k] = p1;
        p.W2.nd[k] = p2;
        p1 += x.ns1[k];
        p2 += x.ns2[k];
      }
      for (int k = 0; k < x.ns1[1]; ++k)
        if (p.W1.nd[1][k] != p.W2.nd[0][k]) rc = QC_ERR_LAYOUT;        // the bond between the sites
      p.W1.ioff = x.ioff1;
      p.W1.allowed = x.allowed1;
      p.W2.ioff = x.ioff2;
      p.W2.allowed = x.allowed2;
      for (int i = 0; i < 16 * x.ndelta; ++i) {
        const int sa = x.iblk[i], sc = x.kblk[i];
        if (sa >= x.ns1[0] || sc >= x.ns2[1] ||
            (sa >= 0 && (x.row0[i] < 0 || x.row0[i] + p.W1.nd[0][sa] > x.R[i / 16])))
          rc = QC_ERR_ARG;
      }
      if (rc != QC_OK) break;
      p.W1.number_rows();
      p.W2.number_rows();
      plan_deltas(p.W1, p.W2, x.ndelta, x.iblk, x.kblk, x.row0, x.R, p.deltas);
    }
    if (rc == QC_OK) {
      h->ops.resize(nops);
      const bool ok = wx_each(nops, [&](long long o) {
        const WxBuild::Part *p = h->parts.data() + nparts - 1;
        while (p->op0 > o) --p;
        const qc_wxpart &x = *p->in;
        build_op(p->W1, x.w1 + x.off1[o - p->op0], p->W2, x.w2 + x.off2[o - p->op0], p->deltas, h->ops[o]);
      });
      rc = ok ? QC_OK : QC_ERR_CAPACITY;
    }
    long long nq = 0;
    for (int q = 0; q < nparts && rc == QC_OK; ++q) {
      nocts[q] = nents[q] = 0;
      for (int o = 0; o < in[q].nops; ++o) {
        const OpLists &l = h->ops[h->parts[q].op0 + o];
        nocts[q] += (long long)l.octs.size();
        nents[q] += (long long)l.r.size();
      }
      nq += nocts[q];
    }
    if (nq > 0x7fffffffLL) rc = QC_ERR_CAPACITY;
    if (rc != QC_OK) {
      delete h;
      return rc;
    }
    *handle = h;
    return QC_OK;
  } catch (...) {
    delete h;
    return QC_ERR_CAPACITY;
  }
}

// Copies what qc_wx_build made, class after class, and frees it: dops [ndelta][nops] of every class,
// octets, T1 rows and the coefficients in the kernels' orders: FP64 fragments (w64: step by
// step, lane l the coefficient of entry l % 4 and row l / 4) and FP32 [nents][8] (w32); either
// may be null.
extern "C" int qc_wx_fetch(void *handle, void *dops, void *octs, double *w64, float *w32, int *r) {
  WxBuild *h = (WxBuild *)handle;
  if (!h) return QC_ERR_ARG;
  qc_wxdop *pd = (qc_wxdop *)dops;
  qc_wxoct *po = (qc_wxoct *)octs;
  long long ent0 = 0;
  int oct0 = 0;
  for (const auto &p : h->parts) {
    const int nops = p.in->nops;
    for (int o = 0; o < nops; ++o) {
      const OpLists &l = h->ops[p.op0 + o];
      for (int d = 0; d < p.in->ndelta; ++d) {
        qc_wxdop x = l.dops[d];
        x.ent_b += ent0;
        x.oct_b += oct0;
        pd[(long long)d * nops + o] = x;
      }
      const size_t n = l.r.size();
      if (!l.octs.empty()) memcpy(po + oct0, l.octs.data(), l.octs.size() * sizeof(qc_wxoct));
      if (n) memcpy(r + ent0, l.r.data(), n * sizeof(int));
      if (w64 && n) memcpy(w64 + 8 * ent0, l.w.data(), 64 * n);
      if (w32)
        for (size_t e = 0; e < n; ++e)
          for (int k = 0; k < 8; ++k) w32[8 * (ent0 + e) + k] = (float)l.w[(e & ~(size_t)3) * 8 + 4 * k + (e & 3)];
      ent0 += (long long)n;
      oct0 += (int)l.octs.size();
    }
    pd += (long long)p.in->ndelta * nops;
  }
  delete h;
  return QC_OK;
}

extern "C" int qc_wsparse_f64(const void *items, long long nitems, int tile, const void *deltas, const void *grps,
                              const void *rows, const void *dops, const void *octs, const void *ent_w,
                              const void *ent_r, const void *ops, int maxR, int maxO, const double *A, double *C,
                              void *stream) {
  if (nitems <= 0) return QC_OK;
  const WxArgs x = {items, nitems, deltas, grps, rows, dops, octs, ent_w, ent_r, ops, maxR, maxO};
  if (wx_bad(x)) return QC_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  switch (tile) {
    case 32: return launch_kernel<double, double, k_wsparse_f64<32>>(wx_smem_bytes<double, 32>(maxR, maxO), x, A, C, s);
    case 64: return launch_kernel<double, double, k_wsparse_f64<64>>(wx_smem_bytes<double, 64>(maxR, maxO), x, A, C, s);
    case 128: return launch_kernel<double, double, k_wsparse_f64<128>>(wx_smem_bytes<double, 128>(maxR, maxO), x, A, C, s);
    default: return QC_ERR_ARG;
  }
}

extern "C" int qc_wsparse_f32(const void *items, long long nitems, int tile, const void *deltas, const void *grps,
                              const void *rows, const void *dops, const void *octs, const void *ent_w,
                              const void *ent_r, const void *ops, int maxR, int maxO, const float *A, float *C,
                              void *stream) {
  if (nitems <= 0) return QC_OK;
  const WxArgs x = {items, nitems, deltas, grps, rows, dops, octs, ent_w, ent_r, ops, maxR, maxO};
  if (wx_bad(x)) return QC_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  switch (tile) {
    case 32: return launch_kernel<float, float4, k_wsparse_f32<32, 32>>(wx_smem_bytes<float, 32>(maxR, maxO), x, A, C, s);
    case 64: return launch_kernel<float, float4, k_wsparse_f32<64, 64>>(wx_smem_bytes<float, 64>(maxR, maxO), x, A, C, s);
    case 128: return launch_kernel<float, float4, k_wsparse_f32<128, 64>>(wx_smem_bytes<float, 128>(maxR, maxO), x, A, C, s);
    default: return QC_ERR_ARG;
  }
}
