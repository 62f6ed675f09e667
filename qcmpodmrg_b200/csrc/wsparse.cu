// The two MPO-site contractions of sigma as one sparse product: T3 = T1 . (W_i W_{i+1})
// (top2 and top3 of HVecQt, source/mpo_dmrg_kernelQt.py:303-306), without the
// intermediate T2.
//
// A fiber is one (l, r) pair of bond states.  For one fiber the two contractions are a
// matrix S[k, i] from its T1 rows i = (a, n1, n2) to its T3 rows k = (c, n1', n2'), and
// every fiber of one charge difference q(l) - q(r) meets the same S.  An ab-initio MPO
// fills about a tenth of the blocks of S that symmetry allows (K = 24: 20 310 of 230 000
// elements per operator, 13 per row k, against 74 multiply-adds per element of the two
// dense block contractions), so S is kept as a list: for every quad of four consecutive
// rows k, the T1 rows that any of the four reads and their four coefficients.
//
// One CTA takes a tile of 32 * FPT fibers of one charge difference (fibers of several
// sector pairs share a tile, so small sectors fill the lanes) and walks operators: the
// tile's T1 rows are staged in shared memory (cp.async, rows contiguous over fibers), a
// warp takes quads of S, lane = fiber, and every entry is one broadcast of (row,
// coefficients) against one conflict-free row read for 4 * FPT FMAs.  T3 keeps r as its
// fastest index, so results leave as contiguous rows straight from registers.
//
// Bound: T1 read and T3 written once.  Mid-chain dot of K=24, D=500 (1.22e9 elements each):
// FP64 8.1 ms, 2.4 TB/s, against 30.2 ms of the two dense stages; FP32 4.6 ms, 2.1 TB/s,
// against 15.5 ms.  The shared-memory pipe (72 % of its wavefronts: row reads and
// coefficient broadcasts) and the issue slots (71 %) bound it, not HBM.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <new>
#include <thread>
#include <vector>
#include "qc_types.h"

namespace {

constexpr int WX_WARPS = 8;
constexpr int WX_THREADS = 32 * WX_WARPS;
constexpr int WX_MAXQ = 1024;             // quads of one (delta, operator)

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

// The four coefficients of an entry: 16-byte vectors, one in FP32 and two in FP64, kept as
// separate arrays (half h of entry e at [h * n + e]) so that 32 lanes move them without bank
// conflicts and one broadcast load reads one.
template <typename T>
struct Coef;
template <>
struct Coef<float> {
  typedef float4 V;
  static constexpr int NV = 1;
  static __device__ __forceinline__ void get(const float4 *p, int, int e, float (&w)[4]) {
    const float4 x = p[e];
    w[0] = x.x;
    w[1] = x.y;
    w[2] = x.z;
    w[3] = x.w;
  }
  static __device__ __forceinline__ float4 zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
};
template <>
struct Coef<double> {
  typedef double2 V;
  static constexpr int NV = 2;
  static __device__ __forceinline__ void get(const double2 *p, int n, int e, double (&w)[4]) {
    const double2 x = p[e], y = p[n + e];
    w[0] = x.x;
    w[1] = x.y;
    w[2] = y.x;
    w[3] = y.y;
  }
  static __device__ __forceinline__ double2 zero() { return make_double2(0.0, 0.0); }
};

template <typename T, int FPT>
__host__ __device__ constexpr size_t wx_fixed_smem() {
  return 34 * 32 * FPT * sizeof(int) +                                             // tabA, tabC, fibF, fibO
         (size_t)WX_WARPS * 32 * (16 * Coef<T>::NV + sizeof(int));                // entry rings
}

template <typename T, int FPT>
__global__ void __launch_bounds__(WX_THREADS)
k_wsparse(const qc_wxitem *__restrict__ items, const qc_wxdelta *__restrict__ deltas,
          const qc_wxgrp *__restrict__ grps, const int *__restrict__ rows, const qc_wxdop *__restrict__ dops,
          const qc_wxquad *__restrict__ quads, const typename Coef<T>::V *__restrict__ ent_w, long long nent,
          const int *__restrict__ ent_r, const qc_op *__restrict__ ops, int maxR, int maxQ, const T *__restrict__ A,
          T *__restrict__ C) {
  typedef typename Coef<T>::V V;
  constexpr int NV = Coef<T>::NV;
  constexpr int FT = 32 * FPT;
  extern __shared__ __align__(16) unsigned char wx_smem[];
  T *const As = reinterpret_cast<T *>(wx_smem);                                  // [R + 1][FT], row R zero
  V *const ring_w0 = reinterpret_cast<V *>(As + (size_t)(maxR + 1) * FT);       // [warps][NV][32]
  qc_wxquad *const sq = reinterpret_cast<qc_wxquad *>(ring_w0 + WX_WARPS * NV * 32);  // [maxQ]
  int *const ring_r0 = reinterpret_cast<int *>(sq + maxQ);                       // [warps][32]
  int *const tabA = ring_r0 + WX_WARPS * 32;                                     // [16][FT]
  int *const tabC = tabA + 16 * FT;                                              // [16][FT]
  int *const fibF = tabC + 16 * FT;                                              // [FT]
  int *const fibO = fibF + FT;                                                   // [FT]
  int *const rowt = fibO + FT;                                                   // [maxR]
  __shared__ int s_start[FT + 1];
  __shared__ int s_grp[FT], s_f[FT];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const qc_wxitem it = items[blockIdx.x];
  const qc_wxdelta *const dl = deltas + it.delta;
  const int R = dl->R, row_b = dl->row_b, grp_e = dl->grp_e, dop_b = dl->dop_b;

  // ---- the tile's fibers: sector pair and fiber in it, then their block offsets
  for (int t = tid; t <= FT; t += WX_THREADS) {
    const int g = it.grp + t;
    s_start[t] = g < grp_e ? grps[g].start : 0x7fffffff;
  }
  for (int r = tid; r < R; r += WX_THREADS) rowt[r] = rows[row_b + r];
  __syncthreads();
  for (int t = tid; t < FT; t += WX_THREADS) {
    const int pos = s_start[0] + it.f0 + t;
    int lo = 0, hi = FT;                       // largest k with s_start[k] <= pos
    while (lo < hi) {
      const int m = (lo + hi + 1) >> 1;
      if (s_start[m] <= pos) lo = m; else hi = m - 1;
    }
    s_grp[t] = t < it.nf ? it.grp + lo : -1;
    s_f[t] = pos - s_start[lo];
    As[R * FT + t] = T(0);
  }
  __syncthreads();
  for (int e = tid; e < 16 * FT; e += WX_THREADS) {
    const int b = e / FT, t = e - b * FT;
    const int g = s_grp[t];
    int oa = -1, oc = -1;
    if (g >= 0) {
      const qc_wxgrp *gr = grps + g;
      const int f = s_f[t], flo = gr->flo;
      oa = gr->a[b];
      if (oa >= 0) oa += f;
      oc = gr->c[b];
      if (oc >= 0) oc += (f / flo) * gr->h[b] + f % flo;
      if (b == 0) {
        fibF[t] = gr->F;
        fibO[t] = flo;
      }
    } else if (b == 0) {
      fibF[t] = fibO[t] = 0;
    }
    tabA[e] = oa;
    tabC[e] = oc;
  }
  __syncthreads();

  V *const ring_w = ring_w0 + warp * NV * 32;
  int *const ring_r = ring_r0 + warp * 32;
  for (int op = it.op_b; op < it.op_e; ++op) {
    const qc_op o = ops[op];
    const qc_wxdop dop = dops[dop_b + op - it.op0];
    const T *const Ao = A + o.a_base;
    T *const Co = C + o.c_base;
    const V *const ew = ent_w + dop.ent_b;
    const int *const er = ent_r + dop.ent_b;
    const qc_wxquad *const gq = quads + dop.quad_b;
    const int nq = dop.nquad;
    // ---- stage the tile's T1 rows and the operator's quad records
    for (int r = warp; r < R; r += WX_WARPS) {
      const int rec = rowt[r];
      const int *ta = tabA + (rec >> 16) * FT;
      const int a = rec & 0xffff;
#pragma unroll
      for (int j = 0; j < FPT; ++j) {
        const int f = lane + 32 * j;
        const int off = ta[f];
        cp_async_el(As + r * FT + f, off >= 0 ? Ao + off + (long long)a * fibF[f] : A, off >= 0);
      }
    }
    for (int e = tid; e < nq; e += WX_THREADS) cp_async_16(sq + e, gq + e);
    asm volatile("cp.async.commit_group;" ::: "memory");
    // the warp's first quad and its first entries, while the rows are in flight; lanes past
    // the end hold the zero row with zero coefficients
    V pw[NV];
    int pr;
    auto fetch = [&](const qc_wxquad &x, int c0) {
#pragma unroll
      for (int h = 0; h < NV; ++h) pw[h] = Coef<T>::zero();
      pr = R;
      if (c0 + lane < x.cnt) {
#pragma unroll
        for (int h = 0; h < NV; ++h) pw[h] = ew[h * nent + x.ent + c0 + lane];
        pr = er[x.ent + c0 + lane];
      }
    };
    int q = warp;
    qc_wxquad cur;
    if (q < nq) {
      cur = gq[q];
      fetch(cur, 0);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    while (q < nq) {
      const qc_wxquad cq = cur;
      const int qn = q + WX_WARPS;
      if (qn < nq) cur = sq[qn];
      T acc[4][FPT];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < FPT; ++j) acc[k][j] = T(0);
      for (int c0 = 0;; c0 += 32) {
        const int n = min(32, cq.cnt - c0);
#pragma unroll
        for (int h = 0; h < NV; ++h) ring_w[32 * h + lane] = pw[h];
        ring_r[lane] = pr * FT;
        __syncwarp();
        const bool more = c0 + 32 < cq.cnt;
        if (more)
          fetch(cq, c0 + 32);
        else if (qn < nq)
          fetch(cur, 0);
        for (int e = 0; e < n; e += 4) {
          const int4 r4 = *reinterpret_cast<const int4 *>(ring_r + e);
          const int rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            T w[4], av[FPT];
            Coef<T>::get(ring_w, 32, e + u, w);
            const T *a = As + rr[u] + lane;
#pragma unroll
            for (int j = 0; j < FPT; ++j) av[j] = a[32 * j];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
              for (int j = 0; j < FPT; ++j) acc[k][j] = fma(w[k], av[j], acc[k][j]);
          }
        }
        __syncwarp();
        if (!more) break;
      }
      // ---- four rows of the block: fibers of one l are contiguous
      const int *tc = tabC + cq.blk * FT;
      const int nc = cq.c0nc & 0xff, cfirst = cq.c0nc >> 8;
#pragma unroll
      for (int j = 0; j < FPT; ++j) {
        const int off = tc[lane + 32 * j], fl = fibO[lane + 32 * j];
        if (off >= 0) {
          T *dst = Co + off + (long long)cfirst * fl;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k < nc) dst[(long long)k * fl] = acc[k][j];
        }
      }
      q = qn;
    }
    __syncthreads();
  }
}

template <typename T, int FPT>
size_t wx_smem_bytes(int maxR, int maxQ) {
  return (size_t)(maxR + 1) * 32 * FPT * sizeof(T) + (size_t)maxQ * sizeof(qc_wxquad) + (size_t)maxR * sizeof(int) +
         wx_fixed_smem<T, FPT>();
}

template <typename T, int FPT>
int launch_fpt(const void *items, long long nitems, const void *deltas, const void *grps, const void *rows,
               const void *dops, const void *quads, const void *ent_w, long long nent, const void *ent_r,
               const void *ops, int maxR, int maxQ, const T *A, T *C, cudaStream_t s) {
  const size_t smem = wx_smem_bytes<T, FPT>(maxR, maxQ);
  if (smem > 224 * 1024) return QC_ERR_ARG;
  cudaError_t e = cudaFuncSetAttribute(k_wsparse<T, FPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) {
    k_wsparse<T, FPT><<<(unsigned)nitems, WX_THREADS, smem, s>>>(
        (const qc_wxitem *)items, (const qc_wxdelta *)deltas, (const qc_wxgrp *)grps, (const int *)rows,
        (const qc_wxdop *)dops, (const qc_wxquad *)quads, (const typename Coef<T>::V *)ent_w, nent,
        (const int *)ent_r, (const qc_op *)ops, maxR, maxQ, A, C);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    fprintf(stderr, "[qcgpu] qc_wsparse: %s\n", cudaGetErrorString(e));
    return QC_ERR_CUDA;
  }
  return QC_OK;
}

template <typename T>
int launch_wsparse(const void *items, long long nitems, int fpt, const void *deltas, const void *grps,
                   const void *rows, const void *dops, const void *quads, const void *ent_w, long long nent,
                   const void *ent_r, const void *ops, int maxR, int maxQ, const T *A, T *C, cudaStream_t s) {
  if (nitems <= 0) return QC_OK;
  if (nitems > 0x7fffffffLL || !items || !deltas || !grps || !rows || !dops || !quads || !ent_w || !ent_r || !ops ||
      maxR < 0 || maxQ < 0 || maxQ > WX_MAXQ || nent < 0)
    return QC_ERR_ARG;
  switch (fpt) {
    case 1: return launch_fpt<T, 1>(items, nitems, deltas, grps, rows, dops, quads, ent_w, nent, ent_r, ops, maxR, maxQ, A, C, s);
    case 2: return launch_fpt<T, 2>(items, nitems, deltas, grps, rows, dops, quads, ent_w, nent, ent_r, ops, maxR, maxQ, A, C, s);
    case 4: return launch_fpt<T, 4>(items, nitems, deltas, grps, rows, dops, quads, ent_w, nent, ent_r, ops, maxR, maxQ, A, C, s);
    default: return QC_ERR_ARG;
  }
}

// ---- host: the sparse rows of S = W_i W_{i+1} for every (delta, operator) of one class
struct Nz {
  int j;
  double v;
};

// A packed W tensor [a, b, n', n] of one class: block (sa, sb, n', n) has its non-zeros
// listed row by row (row a or, for the second site, row b).
struct SparseW {
  int ns[4];
  const long long *nd[4];
  const long long *ioff;
  const int *allowed;
};

struct OpLists {
  std::vector<qc_wxdop> dops;
  std::vector<qc_wxquad> quads;
  std::vector<double> w;
  std::vector<int> r;
};

// rows of the non-zeros of every allowed block: start[block][row], flat lists
void list_rows(const SparseW &W, const double *val, std::vector<std::vector<int>> &start,
               std::vector<std::vector<Nz>> &nz) {
  const int nb = W.ns[0] * W.ns[1] * W.ns[2] * W.ns[3];
  start.assign(nb, std::vector<int>());
  nz.assign(nb, std::vector<Nz>());
  for (int b = 0; b < nb; ++b) {
    if (!W.allowed[b]) continue;
    const int sa = b / (W.ns[1] * W.ns[2] * W.ns[3]), sb = b / (W.ns[2] * W.ns[3]) % W.ns[1];
    const int na = (int)W.nd[0][sa], nbb = (int)W.nd[1][sb];
    const double *p = val + W.ioff[b];
    start[b].resize(na + 1);
    for (int a = 0; a < na; ++a) {
      start[b][a] = (int)nz[b].size();
      for (int j = 0; j < nbb; ++j)
        if (p[(long long)a * nbb + j] != 0.0) nz[b].push_back(Nz{j, p[(long long)a * nbb + j]});
    }
    start[b][na] = (int)nz[b].size();
  }
}

void build_op(const SparseW &W1, const double *v1, const SparseW &W2, const double *v2, int ndelta, const int *iblk,
              const int *kblk, const int *row0, const int *Rs, OpLists &out) {
  std::vector<std::vector<int>> st1, st2;
  std::vector<std::vector<Nz>> nz1, nz2;
  list_rows(W1, v1, st1, nz1);
  list_rows(W2, v2, st2, nz2);
  const int nsb = W1.ns[1];
  std::vector<double> S;
  std::vector<uint64_t> mask;
  std::vector<qc_wxquad> qs;
  for (int d = 0; d < ndelta; ++d) {
    const int R = Rs[d];
    const int words = (R + 63) / 64;
    qc_wxdop rec;
    rec.ent_b = (long long)out.r.size();
    rec.quad_b = (int)out.quads.size();
    qs.clear();
    for (int kb = 0; kb < 16; ++kb) {
      const int sc = kblk[16 * d + kb];
      if (sc < 0) continue;
      const int nc = (int)W2.nd[1][sc];
      const int nq = (nc + 3) / 4;
      S.assign((size_t)nq * 4 * R, 0.0);            // [row i][nc padded to quads]
      mask.assign((size_t)nq * words, 0);
      const int n1p = kb >> 2, n2p = kb & 3;
      for (int ib = 0; ib < 16; ++ib) {
        const int sa = iblk[16 * d + ib];
        if (sa < 0) continue;
        const int n1 = ib >> 2, n2 = ib & 3;
        const int na = (int)W1.nd[0][sa], r0 = row0[16 * d + ib];
        for (int sb = 0; sb < nsb; ++sb) {
          const int b1 = ((sa * W1.ns[1] + sb) * W1.ns[2] + n1p) * W1.ns[3] + n1;
          const int b2 = ((sb * W2.ns[1] + sc) * W2.ns[2] + n2p) * W2.ns[3] + n2;
          if (!W1.allowed[b1] || !W2.allowed[b2] || nz1[b1].empty() || nz2[b2].empty()) continue;
          for (int a = 0; a < na; ++a) {
            const int i = r0 + a;
            for (int x = st1[b1][a]; x < st1[b1][a + 1]; ++x) {
              const Nz u = nz1[b1][x];
              for (int y = st2[b2][u.j]; y < st2[b2][u.j + 1]; ++y) {
                const Nz w = nz2[b2][y];
                S[((size_t)(w.j >> 2) * R + i) * 4 + (w.j & 3)] += u.v * w.v;
                mask[(size_t)(w.j >> 2) * words + (i >> 6)] |= 1ull << (i & 63);
              }
            }
          }
        }
      }
      for (int q = 0; q < nq; ++q) {
        qc_wxquad x;
        x.ent = (int)((long long)out.r.size() - rec.ent_b);
        x.blk = kb;
        x.c0nc = (4 * q) << 8 | std::min(4, nc - 4 * q);
        for (int wd = 0; wd < words; ++wd) {
          uint64_t m = mask[(size_t)q * words + wd];
          while (m) {
            const int i = wd * 64 + __builtin_ctzll(m);
            m &= m - 1;
            const double *p = &S[((size_t)q * R + i) * 4];
            if (p[0] == 0.0 && p[1] == 0.0 && p[2] == 0.0 && p[3] == 0.0) continue;
            out.w.insert(out.w.end(), p, p + 4);
            out.r.push_back(i);
          }
        }
        x.cnt = (int)((long long)out.r.size() - rec.ent_b) - x.ent;
        qs.push_back(x);
      }
    }
    // longest first: warps take quads round-robin, so their loads come out even
    std::stable_sort(qs.begin(), qs.end(), [](const qc_wxquad &x, const qc_wxquad &y) { return x.cnt > y.cnt; });
    out.quads.insert(out.quads.end(), qs.begin(), qs.end());
    rec.nquad = (int)qs.size();
    out.dops.push_back(rec);
  }
}

struct WxBuild {
  std::vector<OpLists> ops;
  int ndelta;
};

}  // namespace

// Sparse rows of W_i W_{i+1} for the operators of one class.  w1 / w2: packed FP64 values
// (host) of operator o at off1[o] / off2[o]; ns / nd / ioff / allowed: the two layouts'
// sector counts, sector extents (four arrays back to back), block offsets and allowed
// blocks; iblk / kblk / row0 [ndelta][16]: left (right) MPO sector of every (n1, n2)
// ((n1', n2')) block of a delta (-1: none) and its first T1 row; R: T1 rows.  Returns the
// quads and entries to fetch with qc_wx_fetch, which frees the handle.
extern "C" int qc_wx_build(int nops, const double *w1, const long long *off1, const int *ns1, const long long *nd1,
                           const long long *ioff1, const int *allowed1, const double *w2, const long long *off2,
                           const int *ns2, const long long *nd2, const long long *ioff2, const int *allowed2,
                           int ndelta, const int *iblk, const int *kblk, const int *row0, const int *R, void **handle,
                           long long *nquads, long long *nents) {
  if (nops < 1 || ndelta < 0 || !w1 || !off1 || !ns1 || !nd1 || !ioff1 || !allowed1 || !w2 || !off2 || !ns2 || !nd2 ||
      !ioff2 || !allowed2 || (ndelta && (!iblk || !kblk || !row0 || !R)) || !handle || !nquads || !nents)
    return QC_ERR_ARG;
  if (ns1[2] != 4 || ns1[3] != 4 || ns2[2] != 4 || ns2[3] != 4 || ns1[1] != ns2[0]) return QC_ERR_LAYOUT;
  try {
    SparseW W1, W2;
    const long long *p1 = nd1, *p2 = nd2;
    for (int k = 0; k < 4; ++k) {
      W1.ns[k] = ns1[k];
      W2.ns[k] = ns2[k];
      W1.nd[k] = p1;
      W2.nd[k] = p2;
      p1 += ns1[k];
      p2 += ns2[k];
    }
    W1.ioff = ioff1;
    W1.allowed = allowed1;
    W2.ioff = ioff2;
    W2.allowed = allowed2;
    for (int d = 0; d < ndelta; ++d)
      for (int b = 0; b < 16; ++b) {
        const int sa = iblk[16 * d + b], sc = kblk[16 * d + b];
        if (sa >= ns1[0] || sc >= ns2[1]) return QC_ERR_ARG;
        if (sa >= 0 && (row0[16 * d + b] < 0 || row0[16 * d + b] + W1.nd[0][sa] > R[d])) return QC_ERR_ARG;
      }
    WxBuild *h = new WxBuild;
    h->ndelta = ndelta;
    h->ops.resize(nops);
    bool bad = false;
    auto work = [&](int o) {
      build_op(W1, w1 + off1[o], W2, w2 + off2[o], ndelta, iblk, kblk, row0, R, h->ops[o]);
    };
    const int nt = nops >= 4 ? std::min(8, std::min(nops, (int)std::max(1u, std::thread::hardware_concurrency()))) : 1;
    if (nt > 1) {
      std::vector<std::thread> th;
      std::vector<char> fail(nt, 0);
      int started = 0;
      try {
        for (; started < nt; ++started)
          th.emplace_back([&, started]() {
            try {
              for (int o = started; o < nops; o += nt) work(o);
            } catch (...) {
              fail[started] = 1;
            }
          });
      } catch (...) {          // no more threads: their operators are done below
      }
      for (auto &t : th) t.join();
      try {
        for (int k = started; k < nt; ++k)
          for (int o = k; o < nops; o += nt) work(o);
      } catch (...) {
        bad = true;
      }
      for (char f : fail) bad = bad || f;
    } else {
      try {
        for (int o = 0; o < nops; ++o) work(o);
      } catch (...) {
        bad = true;
      }
    }
    if (bad) {
      delete h;
      return QC_ERR_CAPACITY;
    }
    long long nq = 0, ne = 0;
    for (const OpLists &l : h->ops) {
      nq += (long long)l.quads.size();
      ne += (long long)l.r.size();
    }
    if (nq > 0x7fffffffLL) {
      delete h;
      return QC_ERR_CAPACITY;
    }
    *handle = h;
    *nquads = nq;
    *nents = ne;
    return QC_OK;
  } catch (...) {
    return QC_ERR_CAPACITY;
  }
}

// Copies what qc_wx_build made and frees it: dops [ndelta][nops] (entry and quad offsets from
// ent0 / quad0), quads, coefficients [nents][4] and T1 rows [nents].
extern "C" int qc_wx_fetch(void *handle, long long ent0, int quad0, void *dops, void *quads, double *w, int *r) {
  WxBuild *h = (WxBuild *)handle;
  if (!h) return QC_ERR_ARG;
  const int nops = (int)h->ops.size();
  qc_wxdop *pd = (qc_wxdop *)dops;
  qc_wxquad *pq = (qc_wxquad *)quads;
  for (int o = 0; o < nops; ++o) {
    const OpLists &l = h->ops[o];
    for (int d = 0; d < h->ndelta; ++d) {
      qc_wxdop x = l.dops[d];
      x.ent_b += ent0;
      x.quad_b += quad0;
      pd[(long long)d * nops + o] = x;
    }
    if (!l.quads.empty()) memcpy(pq, l.quads.data(), l.quads.size() * sizeof(qc_wxquad));
    if (!l.r.empty()) {
      memcpy(w, l.w.data(), l.w.size() * sizeof(double));
      memcpy(r, l.r.data(), l.r.size() * sizeof(int));
    }
    pq += l.quads.size();
    w += l.w.size();
    r += l.r.size();
    ent0 += (long long)l.r.size();
    quad0 += (int)l.quads.size();
  }
  delete h;
  return QC_OK;
}

extern "C" int qc_wsparse_f64(const void *items, long long nitems, int fpt, const void *deltas, const void *grps,
                              const void *rows, const void *dops, const void *quads, const void *ent_w,
                              long long nent, const void *ent_r, const void *ops, int maxR, int maxQ, const double *A,
                              double *C, void *stream) {
  return launch_wsparse<double>(items, nitems, fpt, deltas, grps, rows, dops, quads, ent_w, nent, ent_r, ops, maxR, maxQ,
                            A, C, (cudaStream_t)stream);
}

extern "C" int qc_wsparse_f32(const void *items, long long nitems, int fpt, const void *deltas, const void *grps,
                              const void *rows, const void *dops, const void *quads, const void *ent_w,
                              long long nent, const void *ent_r, const void *ops, int maxR, int maxQ, const float *A,
                              float *C, void *stream) {
  return launch_wsparse<float>(items, nitems, fpt, deltas, grps, rows, dops, quads, ent_w, nent, ent_r, ops, maxR, maxQ,
                            A, C, (cudaStream_t)stream);
}
