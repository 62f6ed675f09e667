// Orthonormalisation of one vector against the rows of a Davidson basis (dvdson_ortho,
// source/tools/pdvdson.py:350-390): `times` passes of r -= V^T (V r), then r / |r| twice.
//
// Bound: launches at small sizes, times + 1 readings of V at large ones (it stays in L2).  A pass
// needs all of V r before it can change r, so passes are separate launches; each one finishes
// the pass before it (sums the blocks' partial products, in a fixed order, and updates its part of
// r) and forms the next products from the values of V that it holds in registers: 8 launches
// for 5 passes where matrix products, subtractions and norms were 20, and V is read once a
// pass.  A vector of the K=8, D=32 sweep: 490 us before (host time, one sync included), 87 now.
#include <cuda_runtime.h>
#include <cstdio>
#include "qc_types.h"

namespace {

constexpr int OR_THREADS = 256, OR_BLOCKS = 296, OR_CHUNK = 512, OR_MAXM = 32;

// sum of p[b * m + j] over the blocks b, by one warp
__device__ __forceinline__ double or_sum(const double *p, int blocks, int m, int j) {
  double s = 0.0;
  for (int b = threadIdx.x & 31; b < blocks; b += 32) s += p[(long long)b * m + j];
#pragma unroll
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

__device__ __forceinline__ void or_block_sum(double v, double *s_red, double *out) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < OR_THREADS / 32; ++w) s += s_red[w];
    *out = s;
  }
  __syncthreads();
}

// r -= V^T c with c the sums of pin (none: r as it is); then the products V r of this block's
// elements, or the sum of their squares.
template <int MB>
__global__ void __launch_bounds__(OR_THREADS)
k_ortho_pass(const double *__restrict__ V, int m, long long n, const double *rin, double *rout,
             const double *__restrict__ pin, double *__restrict__ pout, int squares) {
  __shared__ double s_c[MB], s_red[OR_THREADS / 32];
  const int warp = threadIdx.x >> 5;
  if (pin)
    for (int j = warp; j < m; j += OR_THREADS / 32) {
      const double c = or_sum(pin, gridDim.x, m, j);
      if ((threadIdx.x & 31) == 0) s_c[j] = c;
    }
  __syncthreads();
  double acc[MB];
#pragma unroll
  for (int j = 0; j < MB; ++j) acc[j] = 0.0;
  for (long long i = blockIdx.x * (long long)OR_THREADS + threadIdx.x; i < n; i += (long long)gridDim.x * OR_THREADS) {
    double r = rin[i], v[MB];
#pragma unroll
    for (int j = 0; j < MB; ++j) v[j] = j < m ? V[j * n + i] : 0.0;
    if (pin) {
      double d = 0.0;
#pragma unroll
      for (int j = 0; j < MB; ++j)
        if (j < m) d += s_c[j] * v[j];
      r -= d;
    }
    rout[i] = r;
    if (squares)
      acc[0] += r * r;
    else
#pragma unroll
      for (int j = 0; j < MB; ++j) acc[j] += v[j] * r;
  }
  if (squares)
    or_block_sum(acc[0], s_red, pout + blockIdx.x);
  else
#pragma unroll
    for (int j = 0; j < MB; ++j)
      if (j < m) or_block_sum(acc[j], s_red, pout + (long long)blockIdx.x * m + j);
}

// r /= sqrt(sum of pin); the sums of squares of the result and (first block) the norm
__global__ void __launch_bounds__(OR_THREADS)
k_ortho_scale(long long n, double *__restrict__ r, const double *__restrict__ pin, double *__restrict__ pout,
              double *__restrict__ norm) {
  __shared__ double s_n, s_red[OR_THREADS / 32];
  if (threadIdx.x < 32) {
    const double s = sqrt(or_sum(pin, gridDim.x, 1, 0));
    if (threadIdx.x == 0) s_n = s;
  }
  __syncthreads();
  const double d = s_n;
  if (norm && blockIdx.x == 0 && threadIdx.x == 0) *norm = d;
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)OR_THREADS + threadIdx.x; i < n; i += (long long)gridDim.x * OR_THREADS) {
    const double x = r[i] / d;
    r[i] = x;
    acc += x * x;
  }
  if (pout) or_block_sum(acc, s_red, pout + blockIdx.x);
}

unsigned or_grid(long long n) {
  const long long g = (n + OR_CHUNK - 1) / OR_CHUNK;
  return (unsigned)(g < 1 ? 1 : g > OR_BLOCKS ? OR_BLOCKS : g);
}

template <int MB>
void or_run(const double *V, int m, long long n, const double *r, double *out, double *work, int times,
            cudaStream_t s) {
  const unsigned g = or_grid(n);
  double *p[2] = {work + 1, work + 1 + (long long)OR_BLOCKS * OR_MAXM};
  for (int t = 0; t <= times; ++t)
    k_ortho_pass<MB><<<g, OR_THREADS, 0, s>>>(V, m, n, t ? out : r, out, t ? p[(t + 1) & 1] : nullptr, p[t & 1],
                                              t == times);
  k_ortho_scale<<<g, OR_THREADS, 0, s>>>(n, out, p[times & 1], p[(times + 1) & 1], work);
  k_ortho_scale<<<g, OR_THREADS, 0, s>>>(n, out, p[(times + 1) & 1], nullptr, nullptr);
}

}  // namespace

// doubles of qc_ortho's work buffer (its first one receives |r|)
extern "C" long long qc_ortho_work(void) { return 1 + 2LL * OR_BLOCKS * OR_MAXM; }

extern "C" int qc_ortho(const double *V, int m, long long n, const double *r, double *out, double *work, int times,
                        void *stream) {
  if (!V || !r || !out || !work || m < 1 || m > OR_MAXM || n < 1 || times < 1 || out == r) return QC_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (m <= 4) or_run<4>(V, m, n, r, out, work, times, s);
  else if (m <= 8) or_run<8>(V, m, n, r, out, work, times, s);
  else if (m <= 16) or_run<16>(V, m, n, r, out, work, times, s);
  else or_run<32>(V, m, n, r, out, work, times, s);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    fprintf(stderr, "[qcgpu] qc_ortho: %s\n", cudaGetErrorString(e));
    return QC_ERR_CUDA;
  }
  return QC_OK;
}
