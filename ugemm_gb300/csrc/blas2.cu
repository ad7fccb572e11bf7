// blas2.cu -- SAXPY and SGEMV on the GPU (the reference's saxpy_cpu and
// sgemv_cpu, ugemm.h:86-160).  Both are HBM-bound: every element of x / A is
// read once with coalesced loads; reductions are done in a fixed order, so
// results are deterministic.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"

namespace cg = cooperative_groups;

namespace ugemm {
namespace {

// y[i*incy] += alpha * x[i*incx]  (ugemm.h:86-97)
__global__ void saxpy_kernel(int n, float alpha, const float* __restrict__ x, int incx,
                             float* __restrict__ y, int incy) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (incx == 1 && incy == 1 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0) {
    const long long n4 = n / 4;
    for (long long v = i; v < n4; v += stride) {
      const float4 a = reinterpret_cast<const float4*>(x)[v];
      float4 b = reinterpret_cast<float4*>(y)[v];
      b.x += alpha * a.x; b.y += alpha * a.y; b.z += alpha * a.z; b.w += alpha * a.w;
      reinterpret_cast<float4*>(y)[v] = b;
    }
    for (long long t = n4 * 4 + i; t < n; t += stride) y[t] += alpha * x[t];
    return;
  }
  for (; i < n; i += stride) y[i * incy] += alpha * x[i * incx];
}

// 'N': A is column-major M x N (A[m + n*lda]); y[m] = alpha * sum_n A[m,n] x[n]
// + beta * y[m].  A block owns 32 V rows (V = 4: 16-byte loads, 512 bytes of a
// column at a time); its W warps take every Wth column, U loads in flight
// each, and the partial sums are added in a fixed order.  HBM-bound: what counts
// is bytes in flight and long runs of a column, so where row blocks are few a
// cluster of kGemvCluster blocks shares the columns of each, the sums passing
// through distributed shared memory in rank order.
constexpr int kGemvCluster = 8;
template <int V, int W, int U>
__global__ void __launch_bounds__(W * 32)
    sgemv_n_kernel(int M, int N, float alpha, const float* __restrict__ A, int lda,
                   const float* __restrict__ x, int incx, float beta, float* __restrict__ y,
                   int incy, int share) {
  __shared__ float part[W][32 * V + 1];
  __shared__ float sum[32 * V];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int rank = share > 1 ? blockIdx.x % share : 0;
  const int m0 = (blockIdx.x / share) * 32 * V, m = m0 + lane * V;
  const int step = W * share;
  float s[V];
#pragma unroll
  for (int e = 0; e < V; ++e) s[e] = 0.f;
  if (m < M) {  // (V = 4: M is a multiple of 4)
    const float* col = A + m;
    auto load = [&](int n, float (&v)[V]) {
      const float* p = col + static_cast<long long>(n) * lda;
      if constexpr (V == 4) {
        const float4 q = __ldcs(reinterpret_cast<const float4*>(p));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
      } else {
        v[0] = *p;
      }
    };
    int n = w * share + rank;
    for (; n + (U - 1) * step < N; n += U * step) {
      float v[U][V];
#pragma unroll
      for (int u = 0; u < U; ++u) load(n + u * step, v[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float b = x[static_cast<long long>(n + u * step) * incx];
#pragma unroll
        for (int e = 0; e < V; ++e) s[e] += v[u][e] * b;
      }
    }
    if (n < N) {  // fewer than U: together all the same, beyond N zeros
      float v[U][V];
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int e = 0; e < V; ++e) v[u][e] = 0.f;
        if (n + u * step < N) load(n + u * step, v[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float b = n + u * step < N ? x[static_cast<long long>(n + u * step) * incx] : 0.f;
#pragma unroll
        for (int e = 0; e < V; ++e) s[e] += v[u][e] * b;
      }
    }
  }
#pragma unroll
  for (int e = 0; e < V; ++e) part[w][lane * V + e] = s[e];
  __syncthreads();
  const int r = threadIdx.x;  // a row of the block
  float t = 0.f;
  if (r < 32 * V) {
    // in pairs: a chain of 16 rounds twice as much (64 x 64: 8.2e-8, in
    // pairs 6.6e-8)
    float p[W];
#pragma unroll
    for (int j = 0; j < W; ++j) p[j] = part[j][r];
#pragma unroll
    for (int d = W / 2; d > 0; d /= 2)
#pragma unroll
      for (int j = 0; j < d; ++j) p[j] += p[j + d];
    t = p[0];
    sum[r] = t;
  }
  if (share > 1) {
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    if (rank == 0 && r < 32 * V) {
      t = 0.f;
      for (int c = 0; c < share; ++c) t += cl.map_shared_rank(sum, c)[r];
    }
    cl.sync();  // the others' shared memory stays until it has been read
  }
  if (rank == 0 && r < 32 * V && m0 + r < M) {
    float* yp = y + static_cast<long long>(m0 + r) * incy;
    *yp = (beta == 0.f) ? alpha * t : alpha * t + beta * *yp;
  }
}

// 'T': A is column-major N x M (A[n + m*lda]); y[m] = alpha * sum_n A[n,m] x[n]
// + beta * y[m].  WPC warps per output, coalesced along the column: 16-byte
// loads, U in flight, where A's columns and x allow them (VEC), else of four
// bytes; reduced by a fixed tree.  HBM-bound (8192 x 8192: one scalar
// load in flight 53 us, 5.1 TB/s; now 41); short columns by the loads' latency
// and the warps in flight, which U = 8 halves.
template <int WPC, bool VEC, int U>
__global__ void __launch_bounds__(256) sgemv_t_kernel(int M, int N, float alpha,
                                                      const float* __restrict__ A, int lda,
                                                      const float* __restrict__ x, int incx,
                                                      float beta, float* __restrict__ y, int incy) {
  __shared__ float part[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int m = blockIdx.x * (8 / WPC) + w / WPC;
  const int t = (w % WPC) * 32 + lane;  // this thread among the output's
  constexpr int T = WPC * 32;
  float s = 0.f;
  if (m < M) {
    const float* col = A + static_cast<long long>(m) * lda;
    if (VEC) {
      const float4* c4 = reinterpret_cast<const float4*>(col);
      const float4* x4 = reinterpret_cast<const float4*>(x);
      const int n4 = N / 4;
      auto add = [&](const float4& a, const float4& b) {
        s += a.x * b.x; s += a.y * b.y; s += a.z * b.z; s += a.w * b.w;
      };
      int i = t;
      for (; i + (U - 1) * T < n4; i += U * T) {
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = __ldcs(c4 + i + u * T);
#pragma unroll
        for (int u = 0; u < U; ++u) add(v[u], x4[i + u * T]);
      }
      if constexpr (U <= 2) {
        if (i < n4) add(__ldcs(c4 + i), x4[i]);
      } else {
        for (; i < n4; i += T) add(c4[i], x4[i]);
      }
      for (int n = 4 * n4 + t; n < N; n += T) s += col[n] * x[n];
    } else {
      constexpr int L = U;  // loads in flight
      int n = t;
      for (; n + (L - 1) * T < N; n += L * T) {
        float v[L];
#pragma unroll
        for (int u = 0; u < L; ++u) v[u] = col[n + u * T];
#pragma unroll
        for (int u = 0; u < L; ++u) s += v[u] * x[static_cast<long long>(n + u * T) * incx];
      }
      if (n < N) {
        float v[L];
#pragma unroll
        for (int u = 0; u < L; ++u) v[u] = n + u * T < N ? col[n + u * T] : 0.f;
#pragma unroll
        for (int u = 0; u < L; ++u)
          s += v[u] * (n + u * T < N ? x[static_cast<long long>(n + u * T) * incx] : 0.f);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (WPC > 1) {
    if (lane == 0) part[w] = s;
    __syncthreads();
    float p[WPC];
#pragma unroll
    for (int j = 0; j < WPC; ++j) p[j] = part[w / WPC * WPC + j];
#pragma unroll
    for (int d = WPC / 2; d > 0; d /= 2)
#pragma unroll
      for (int j = 0; j < d; ++j) p[j] += p[j + d];
    s = p[0];
  }
  if (t == 0 && m < M) {
    float* yp = y + static_cast<long long>(m) * incy;
    *yp = (beta == 0.f) ? alpha * s : alpha * s + beta * *yp;
  }
}

template <int WPC>
void launch_gemv_t(int M, int N, float alpha, const float* A, int lda, const float* x, int incx,
                   float beta, float* y, int incy, cudaStream_t st) {
  const bool vec = (lda & 3) == 0 && incx == 1 &&
                   ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(x)) & 15) == 0;
  const int grid = cdiv(M, 8 / WPC);
  auto kern = !vec ? (N <= 64 * WPC ? sgemv_t_kernel<WPC, false, 2> : sgemv_t_kernel<WPC, false, 8>)
              : N <= 256 * WPC ? sgemv_t_kernel<WPC, true, 2> : sgemv_t_kernel<WPC, true, 8>;
  kern<<<grid, 256, 0, st>>>(M, N, alpha, A, lda, x, incx, beta, y, incy);
}

// Clusters of blocks share the columns when the row blocks are few: as many as
// keep the blocks within 2.5 an SM, and 64 columns a block.  (More blocks than
// that lose more to the clusters' barriers than they gain: 16384 x 1024 in
// blocks of 32 rows 11 us alone, 31 in eights; 2048 x 2048 7.8 alone, 5.7 in fours;
// 8192 x 8192 in blocks of 128 rows 45 us in fours, 53 in eights.)
template <int V, int W, int U>
cudaError_t launch_gemv_nw(int M, int N, float alpha, const float* A, int lda, const float* x,
                           int incx, float beta, float* y, int incy, int share, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(cdiv(M, 32 * V)) * share);
  cfg.blockDim = dim3(W * 32);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = share;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = share > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, sgemv_n_kernel<V, W, U>, M, N, alpha, A, lda, x, incx, beta, y, incy,
                            share);
}

template <int V>
cudaError_t launch_gemv_n(int M, int N, float alpha, const float* A, int lda, const float* x,
                          int incx, float beta, float* y, int incy, cudaStream_t st) {
  const int rows = cdiv(M, 32 * V), sms = device_sms();
  int share = kGemvCluster;
  while (share > 1 && (2LL * rows * share > 5LL * sms || N < 64 * share)) share /= 2;
  // few columns of many rows: 8 warps a block, whose sums are half the work
  // (40000 x 64, unaligned: 5.4 us with 16, 3.6)
  if (V == 1 && N <= 256 && rows >= 4 * sms)
    return launch_gemv_nw<1, 8, 4>(M, N, alpha, A, lda, x, incx, beta, y, incy, 1, st);
  return launch_gemv_nw<V, 16, V == 4 ? 4 : 8>(M, N, alpha, A, lda, x, incx, beta, y, incy, share, st);
}

}  // namespace
}  // namespace ugemm

using namespace ugemm;

extern "C" {

UGEMM_API int ugemm_saxpy(int N, float alpha, const float* x, int incx, float* y, int incy,
                          void* stream) {
  if (N < 0 || incx <= 0 || incy <= 0) return UGEMM_ERR_ARG;
  if (N == 0) return UGEMM_OK;
  if (!x || !y) return UGEMM_ERR_ARG;
  const int grid = static_cast<int>(std::min<long long>((N + 1023) / 1024, 152LL * 16));
  prof_begin(static_cast<cudaStream_t>(stream));
  saxpy_kernel<<<std::max(grid, 1), 256, 0, static_cast<cudaStream_t>(stream)>>>(N, alpha, x, incx,
                                                                                y, incy);
  prof_end(static_cast<cudaStream_t>(stream), kProfAux);
  return cudaPeekAtLastError() == cudaSuccess ? UGEMM_OK : UGEMM_ERR_CUDA;
}

UGEMM_API int ugemm_sgemv(char trans, int M, int N, float alpha, const float* A, int lda,
                          const float* x, int incx, float beta, float* y, int incy,
                          void* stream) {
  const bool t = (trans == 'T' || trans == 't');
  if (!t && trans != 'N' && trans != 'n') return UGEMM_ERR_ARG;
  if (M < 0 || N < 0 || incx <= 0 || incy <= 0) return UGEMM_ERR_ARG;
  if (lda < std::max(1, t ? N : M)) return UGEMM_ERR_ARG;
  if (M == 0) return UGEMM_OK;
  if (!y || (N > 0 && (!A || !x))) return UGEMM_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  prof_begin(st);
  // 16-byte loads, but where columns are few and blocks of 32 rows share the SMs more
  // evenly than blocks of 128 (100000 x 100: 8.1 us, 8.7)
  const bool even = N <= 256 && cdiv(M, 128) >= 4 * device_sms();
  if (!t && ((M | lda) & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0 && M >= 512 && !even)
    (void)launch_gemv_n<4>(M, N, alpha, A, lda, x, incx, beta, y, incy, st);
  else if (!t)
    (void)launch_gemv_n<1>(M, N, alpha, A, lda, x, incx, beta, y, incy, st);
  else {
    // warps an output: one up to 2048 long where the outputs fill the SMs, and up to
    // 1024 where they do not, so that no thread has fewer than 16 products and its
    // share of the tree (2000 x 100: 3.3 us in eights, 1.9)
    const bool few = M < 16 * device_sms();
    if (N > (few ? 4095 : 4096)) launch_gemv_t<8>(M, N, alpha, A, lda, x, incx, beta, y, incy, st);
    else if (N > (few ? 2047 : 2048)) launch_gemv_t<4>(M, N, alpha, A, lda, x, incx, beta, y, incy, st);
    else if (few && N > 1023) launch_gemv_t<2>(M, N, alpha, A, lda, x, incx, beta, y, incy, st);
    else launch_gemv_t<1>(M, N, alpha, A, lda, x, incx, beta, y, incy, st);
  }
  prof_end(st, kProfAux);
  return cudaPeekAtLastError() == cudaSuccess ? UGEMM_OK : UGEMM_ERR_CUDA;
}

}  // extern "C"
