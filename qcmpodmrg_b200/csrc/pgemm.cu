// Dense panel GEMM (FP64 tensor pipe / FP32 FFMA) for contractions laid out as panels.
//
// The L.psi contraction of HVecQt (source/mpo_dmrg_kernelQt.py:301, top1 =
// tensordot(L, psi, axes=([2],[0]))) pairs every L block (a, l, l') with every
// psi block (l', n1, n2, r) of the same sector l'.  With the L blocks of one
// sector stacked into a row-major panel [M x K] (a per-dot permutation), each
// psi block is the row-major [K x N] operand of one dense GEMM whose [M x N]
// result is a run of T1 blocks.  No index maps are needed: the kernel is a plain
// tiled GEMM with a register-prefetch software pipeline (the next K-slice is
// loaded from global memory while the current one is multiplied out of shared
// memory) and one barrier per K-slice.
#include <cuda_runtime.h>
#include <cstdio>
#include "qc_types.h"

namespace {

template <typename T, int TM, int TN, int TK, int RM, int RN, int NT>
__global__ void __launch_bounds__(NT, 2)
k_pgemm(const qc_ptask *__restrict__ tasks, const qc_op *__restrict__ ops, const long long *__restrict__ crow,
        const T *__restrict__ A, const T *__restrict__ B, T *__restrict__ C) {
  constexpr int TX = TN / RN, TY = TM / RM;
  static_assert(TX * TY == NT, "thread tile");
  constexpr int LA = (TM * TK + NT - 1) / NT;       // A elements per thread per K-slice
  constexpr int LB = (TK * TN + NT - 1) / NT;
  __shared__ T As[2][TK][TM + 1];
  __shared__ T Bs[2][TK][TN + 1];

  const qc_ptask t = tasks[blockIdx.x];
  const int op = t.op_b + (int)blockIdx.y;
  if (op >= t.op_e) return;
  const qc_op o = ops[op];
  const T *Ab = A + o.a_base + t.a_off;
  const T *Bb = B + o.b_base + t.b_off;
  const T alpha = T(o.alpha);
  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;
  const int M = t.M, N = t.N, K = t.K;
  const long long lda = t.lda > 0 ? t.lda : K;

  T ra[LA], rb[LB];
  auto load = [&](int k0) {
#pragma unroll
    for (int e = 0; e < LA; ++e) {       // A: TK consecutive k of one row per TK threads
      const int idx = tid + e * NT;
      const int kk = idx % TK, i = idx / TK;
      const int m = t.m0 + i, k = k0 + kk;
      ra[e] = (idx < TM * TK && m < M && k < K) ? Ab[(long long)m * lda + k] : T(0);
    }
#pragma unroll
    for (int e = 0; e < LB; ++e) {       // B: consecutive n of one k row
      const int idx = tid + e * NT;
      const int j = idx % TN, kk = idx / TN;
      const int n = t.n0 + j, k = k0 + kk;
      rb[e] = (idx < TK * TN && n < N && k < K) ? Bb[(long long)k * N + n] : T(0);
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int e = 0; e < LA; ++e) {
      const int idx = tid + e * NT;
      if (idx < TM * TK) As[buf][idx % TK][idx / TK] = ra[e];
    }
#pragma unroll
    for (int e = 0; e < LB; ++e) {
      const int idx = tid + e * NT;
      if (idx < TK * TN) Bs[buf][idx / TN][idx % TN] = rb[e];
    }
  };

  T acc[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) acc[i][j] = T(0);

  const int nsteps = (K + TK - 1) / TK;
  load(0);
  for (int s = 0; s < nsteps; ++s) {
    const int buf = s & 1;
    store(buf);
    __syncthreads();
    if (s + 1 < nsteps) load((s + 1) * TK);
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      T av[RM], bv[RN];
#pragma unroll
      for (int i = 0; i < RM; ++i) av[i] = As[buf][kk][ty + i * TY];
#pragma unroll
      for (int j = 0; j < RN; ++j) bv[j] = Bs[buf][kk][tx + j * TX];
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
    }
  }
  T *Cb = C + o.c_base;
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int m = t.m0 + ty + i * TY;
    if (m >= M) continue;
    const long long row = (t.crow >= 0) ? crow[t.crow + m] : t.c_off + (long long)m * N;
#pragma unroll
    for (int j = 0; j < RN; ++j) {
      const int n = t.n0 + tx + j * TX;
      if (n < N) Cb[row + n] = alpha * acc[i][j];
    }
  }
}

// ---- FP64 on the tensor pipe (mma.sync f64)
//
// The same tasks with 8 x 8 x 4 FP64 tensor-core products.  The FP64 tensor pipe has the
// rate of the DFMA pipe (37 against 33 TFLOP/s measured on dependent-free streams), but one
// instruction does 256 multiply-adds on operands of one register each, so shared memory
// and issue slots no longer bound the kernel.  A warp owns 16 rows x TN columns: the
// column tiles past N are skipped by all warps alike, and so are the 4-wide K steps past K
// (panels of small sectors are a few columns wide and a few k deep).  Operands arrive by a
// three-stage cp.async ring, 16 bytes at a time where the panel's rows allow it.
// Mid-chain dot of K=24, D=500, all panels of L.psi and .R: 31.3 -> 21.6 ms.
constexpr int DG_BK = 16, DG_STAGES = 3, DG_THREADS = 256;
constexpr int DG_PA = DG_BK + 4;       // row pitch of A (doubles): 8 rows x 4 k touch every bank pair once
template <int TN>
__host__ __device__ constexpr int dg_pb() { return TN + 4; }
template <int TN>
__host__ __device__ constexpr int dg_stage() { return 128 * DG_PA + DG_BK * dg_pb<TN>(); }

__device__ __forceinline__ void dg_cp(unsigned dst, const double *src, int bytes16, int valid) {
  if (bytes16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <int TN>
__global__ void __launch_bounds__(DG_THREADS, 2)
k_dgemm(const qc_ptask *__restrict__ tasks, const qc_op *__restrict__ ops, const long long *__restrict__ crow,
        const double *__restrict__ A, const double *__restrict__ B, double *__restrict__ C) {
  constexpr int NT = TN / 8, PB = dg_pb<TN>(), ST = dg_stage<TN>();
  extern __shared__ __align__(16) double dg_smem[];
  const qc_ptask t = tasks[blockIdx.x];
  const int op = t.op_b + (int)blockIdx.y;
  if (op >= t.op_e) return;
  const qc_op o = ops[op];
  const int M = t.M, N = t.N, K = t.K;
  const long long lda = t.lda > 0 ? t.lda : K;
  const double *const Ab = A + o.a_base + t.a_off + (long long)t.m0 * lda;
  const double *const Bb = B + o.b_base + t.b_off + t.n0;
  const int mrem = min(128, M - t.m0), nrem = min(TN, N - t.n0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(dg_smem);
  const bool va = !(lda & 1) && !((unsigned long long)Ab & 15);
  const bool vb = !(N & 1) && !((unsigned long long)Bb & 15);

  auto load = [&](int kt, int st) {
    const int k0 = kt * DG_BK, kr = K - k0;
    const unsigned sa = sbase + (unsigned)(st * ST) * 8u, sb = sa + 128u * DG_PA * 8u;
    if (va) {
#pragma unroll
      for (int e = 0; e < 128 * DG_BK / 2 / DG_THREADS; ++e) {
        const int idx = tid + e * DG_THREADS, k = 2 * (idx % (DG_BK / 2)), m = idx / (DG_BK / 2);
        const int v = (m < mrem) ? max(0, min(2, kr - k)) * 8 : 0;
        dg_cp(sa + (unsigned)(m * DG_PA + k) * 8u, v ? Ab + m * lda + k0 + k : A, 1, v);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 128 * DG_BK / DG_THREADS; ++e) {
        const int idx = tid + e * DG_THREADS, k = idx % DG_BK, m = idx / DG_BK;
        const int v = (m < mrem && k < kr) ? 8 : 0;
        dg_cp(sa + (unsigned)(m * DG_PA + k) * 8u, v ? Ab + m * lda + k0 + k : A, 0, v);
      }
    }
    if (vb) {
      for (int idx = tid; idx < DG_BK * TN / 2; idx += DG_THREADS) {
        const int n = 2 * (idx % (TN / 2)), k = idx / (TN / 2);
        const int v = (k < kr) ? max(0, min(2, nrem - n)) * 8 : 0;
        dg_cp(sb + (unsigned)(k * PB + n) * 8u, v ? Bb + (long long)(k0 + k) * N + n : B, 1, v);
      }
    } else {
      for (int idx = tid; idx < DG_BK * TN; idx += DG_THREADS) {
        const int n = idx % TN, k = idx / TN;
        const int v = (k < kr && n < nrem) ? 8 : 0;
        dg_cp(sb + (unsigned)(k * PB + n) * 8u, v ? Bb + (long long)(k0 + k) * N + n : B, 0, v);
      }
    }
  };

  double acc[2][NT][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  const int nk = (K + DG_BK - 1) / DG_BK;
#pragma unroll
  for (int s = 0; s < DG_STAGES - 1; ++s) {
    if (s < nk) load(s, s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const int gr = lane >> 2, gk = lane & 3;         // fragment row (or column) and k of this lane
  const int nt = (nrem + 7) >> 3;
  const bool live = warp * 16 < mrem;
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(DG_STAGES - 2) : "memory");
    __syncthreads();
    if (kt + DG_STAGES - 1 < nk) load(kt + DG_STAGES - 1, (kt + DG_STAGES - 1) % DG_STAGES);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (live) {
      const double *as = dg_smem + (kt % DG_STAGES) * ST + (warp * 16 + gr) * DG_PA + gk;
      const double *bs = dg_smem + (kt % DG_STAGES) * ST + 128 * DG_PA + gk * PB + gr;
      const int k4 = min(DG_BK / 4, (K - kt * DG_BK + 3) >> 2);
#pragma unroll
      for (int kk = 0; kk < DG_BK / 4; ++kk) {
        if (kk < k4) {
          const double a0 = as[4 * kk], a1 = as[8 * DG_PA + 4 * kk];
#pragma unroll
          for (int j = 0; j < NT; ++j)
            if (j < nt) {
              const double b = bs[4 * kk * PB + 8 * j];
              dmma884(acc[0][j], a0, b);
              dmma884(acc[1][j], a1, b);
            }
        }
      }
    }
  }
  // the accumulator of lane l: row l / 4, columns 2 (l % 4) and the next one
  double *const Cb = C + o.c_base;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int ml = warp * 16 + 8 * i + gr;
    if (ml >= mrem) continue;
    const int m = t.m0 + ml;
    double *dst = Cb + ((t.crow >= 0) ? crow[t.crow + m] : t.c_off + (long long)m * N) + t.n0;
    const bool v2 = !((unsigned long long)dst & 15);
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int n = 8 * j + 2 * gk;
      const double x = o.alpha * acc[i][j][0], y = o.alpha * acc[i][j][1];
      if (n + 1 < nrem && v2) {
        *reinterpret_cast<double2 *>(dst + n) = make_double2(x, y);
      } else {
        if (n < nrem) dst[n] = x;
        if (n + 1 < nrem) dst[n + 1] = y;
      }
    }
  }
}

template <int TN>
int launch_dg(dim3 grid, const qc_ptask *tk, const qc_op *op, const long long *crow, const double *A, const double *B,
              double *C, cudaStream_t s) {
  const int smem = DG_STAGES * dg_stage<TN>() * 8;
  if (cudaFuncSetAttribute(k_dgemm<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return QC_ERR_CUDA;
  k_dgemm<TN><<<grid, DG_THREADS, smem, s>>>(tk, op, crow, A, B, C);
  return QC_OK;
}

int launch_dgemm(const void *tasks, long long ntasks, int opspan, const void *ops, const long long *crow,
                 const double *A, const double *B, double *C, int cfg, cudaStream_t s) {
  if (ntasks <= 0) return QC_OK;
  if (ntasks > 0x7fffffffLL || opspan < 1 || opspan > 65535) return QC_ERR_ARG;
  dim3 grid((unsigned)ntasks, (unsigned)opspan);
  const qc_ptask *tk = (const qc_ptask *)tasks;
  const qc_op *op = (const qc_op *)ops;
  int rc = QC_ERR_ARG;
  switch (cfg) {
    case 0: rc = launch_dg<64>(grid, tk, op, crow, A, B, C, s); break;   // N > 32
    case 1: rc = launch_dg<32>(grid, tk, op, crow, A, B, C, s); break;   // 16 < N <= 32
    case 2: rc = launch_dg<16>(grid, tk, op, crow, A, B, C, s); break;   // N <= 16
    default: return rc;
  }
  cudaError_t e = cudaGetLastError();
  if (rc != QC_OK || e != cudaSuccess) {
    fprintf(stderr, "[qcgpu] qc_pgemm_f64: %s\n", cudaGetErrorString(e));
    return QC_ERR_CUDA;
  }
  return QC_OK;
}

template <typename T>
int launch_pgemm(const void *tasks, long long ntasks, int opspan, const void *ops, const long long *crow, const T *A,
                 const T *B, T *C, int cfg, cudaStream_t s) {
  if (ntasks <= 0) return QC_OK;
  if (ntasks > 0x7fffffffLL || opspan < 1 || opspan > 65535) return QC_ERR_ARG;
  dim3 grid((unsigned)ntasks, (unsigned)opspan);
  const qc_ptask *tk = (const qc_ptask *)tasks;
  const qc_op *op = (const qc_op *)ops;
  constexpr int KT = 16;
  switch (cfg) {
    case 0: k_pgemm<T, 128, 64, KT, 8, 4, 256><<<grid, 256, 0, s>>>(tk, op, crow, A, B, C); break;   // N > 32
    case 1: k_pgemm<T, 128, 32, KT, 8, 2, 256><<<grid, 256, 0, s>>>(tk, op, crow, A, B, C); break;   // 16 < N <= 32
    case 2: k_pgemm<T, 128, 16, KT, 4, 2, 256><<<grid, 256, 0, s>>>(tk, op, crow, A, B, C); break;   // N <= 16
    default: return QC_ERR_ARG;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    fprintf(stderr, "[qcgpu] qc_pgemm: %s\n", cudaGetErrorString(e));
    return QC_ERR_CUDA;
  }
  return QC_OK;
}

}  // namespace

extern "C" int qc_pgemm_f64(const void *tasks, long long ntasks, int opspan, const void *ops, const long long *crow,
                            const double *A, const double *B, double *C, int cfg, void *stream) {
  return launch_dgemm(tasks, ntasks, opspan, ops, crow, A, B, C, cfg, (cudaStream_t)stream);
}

extern "C" int qc_pgemm_f32(const void *tasks, long long ntasks, int opspan, const void *ops, const long long *crow,
                            const float *A, const float *B, float *C, int cfg, void *stream) {
  return launch_pgemm<float>(tasks, ntasks, opspan, ops, crow, A, B, C, cfg, (cudaStream_t)stream);
}
