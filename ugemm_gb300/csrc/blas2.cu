// blas2.cu -- SAXPY and SGEMV on the GPU (the reference's saxpy_cpu and
// sgemv_cpu, ugemm.h:86-160).  Both are HBM-bound: every element of x / A is
// read once with coalesced loads; reductions are done in a fixed order, so
// results are deterministic.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

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

// Four floats of A.  A matrix that L2 cannot hold streams past what it does
// hold (8192 x 8192: 41 us, 43 without); a smaller one stays for the next call, which
// finds it there (16384 x 1024 transposed: 8.2 us, 14.4 when it may not stay).
template <bool STREAM>
__device__ __forceinline__ float4 load_a4(const float4* p) {
  return STREAM ? __ldcs(p) : __ldg(p);
}

// Whether A is larger than the current device's L2 (looked up once per device).
bool beyond_l2(int M, int N) {
  static std::atomic<int> cached[64];
  int dev = 0, bytes = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  bytes = cached[dev].load(std::memory_order_relaxed);
  if (bytes == 0) {
    if (cudaDeviceGetAttribute(&bytes, cudaDevAttrL2CacheSize, dev) != cudaSuccess || bytes <= 0)
      return false;
    cached[dev].store(bytes, std::memory_order_relaxed);
  }
  return 4LL * M * N > bytes;
}

// 'N': A is column-major M x N (A[m + n*lda]); y[m] = alpha * sum_n A[m,n] x[n]
// + beta * y[m].  A block owns 32 V rows (V = 4: 16-byte loads, 512 bytes of a
// column at a time); its W warps take every Wth column, U loads in flight
// each, and the partial sums are added in a fixed order.  HBM-bound: what counts
// is bytes in flight and long runs of a column, so where row blocks are few a
// cluster of kGemvCluster blocks shares the columns of each, the sums passing
// through distributed shared memory in rank order.
constexpr int kGemvCluster = 8;
template <int V, int W, int U, bool CLUSTER, bool STREAM>
__global__ void __launch_bounds__(W * 32)
    sgemv_n_kernel(int M, int N, float alpha, const float* __restrict__ A, int lda,
                   const float* __restrict__ x, int incx, float beta, float* __restrict__ y,
                   int incy, int cluster) {
  const int share = CLUSTER ? cluster : 1;
  __shared__ float part[W][32 * V + 1];
  __shared__ float sum[32 * V];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int rank = CLUSTER ? blockIdx.x % share : 0;
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
        const float4 q = load_a4<STREAM>(reinterpret_cast<const float4*>(p));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
      } else {
        v[0] = *p;
      }
    };
    // U columns' products: one after the other, or, where few warps make long
    // chains, in pairs first
    auto add = [&](const float (&v)[U][V], const float (&b)[U]) {
#pragma unroll
      for (int e = 0; e < V; ++e) {
        if constexpr (W >= 8) {
#pragma unroll
          for (int u = 0; u < U; ++u) s[e] += v[u][e] * b[u];
        } else {
          float p[U];
#pragma unroll
          for (int u = 0; u < U; ++u) p[u] = v[u][e] * b[u];
#pragma unroll
          for (int d = U / 2; d > 0; d /= 2)
#pragma unroll
            for (int u = 0; u < d; ++u) p[u] += p[u + d];
          s[e] += p[0];
        }
      }
    };
    int n = w * share + rank;
    for (; n + (U - 1) * step < N; n += U * step) {
      float v[U][V];
#pragma unroll
      for (int u = 0; u < U; ++u) load(n + u * step, v[u]);
      float b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) b[u] = x[static_cast<long long>(n + u * step) * incx];
      add(v, b);
    }
    if (n < N) {  // fewer than U: together all the same, beyond N zeros
      float v[U][V];
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int e = 0; e < V; ++e) v[u][e] = 0.f;
        if (n + u * step < N) load(n + u * step, v[u]);
      }
      float b[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        b[u] = n + u * step < N ? x[static_cast<long long>(n + u * step) * incx] : 0.f;
      add(v, b);
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
    if (CLUSTER) sum[r] = t;
  }
  if constexpr (CLUSTER) {
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

// The same for at most kGemvColumns columns: a thread has V rows to itself, all
// its loads in flight, and adds the products in pairs.  Nothing is shared, so
// the blocks are bound by the loads alone (1000000 x 1: 3.6 us, 21 where eight
// warps share a block's rows; 100000 x 8: 1.8 and 4.2).
constexpr int kGemvColumns = 8;
template <int V>
__global__ void __launch_bounds__(128)
    sgemv_rows_kernel(int M, int N, float alpha, const float* __restrict__ A, int lda,
                      const float* __restrict__ x, int incx, float beta, float* __restrict__ y,
                      int incy) {
  const long long m = (blockIdx.x * 128LL + threadIdx.x) * V;
  if (m >= M) return;  // (V = 4: M is a multiple of 4)
  float p[kGemvColumns][V];
#pragma unroll
  for (int n = 0; n < kGemvColumns; ++n) {
#pragma unroll
    for (int e = 0; e < V; ++e) p[n][e] = 0.f;
    if (n < N) {
      const float* c = A + m + static_cast<long long>(n) * lda;
      if constexpr (V == 4) {
        const float4 q = load_a4<false>(reinterpret_cast<const float4*>(c));
        p[n][0] = q.x; p[n][1] = q.y; p[n][2] = q.z; p[n][3] = q.w;
      } else {
        p[n][0] = *c;
      }
    }
  }
#pragma unroll
  for (int n = 0; n < kGemvColumns; ++n) {
    const float b = n < N ? x[static_cast<long long>(n) * incx] : 0.f;
#pragma unroll
    for (int e = 0; e < V; ++e) p[n][e] *= b;
  }
#pragma unroll
  for (int d = kGemvColumns / 2; d > 0; d /= 2)
#pragma unroll
    for (int n = 0; n < d; ++n)
#pragma unroll
      for (int e = 0; e < V; ++e) p[n][e] += p[n + d][e];
#pragma unroll
  for (int e = 0; e < V; ++e) {
    float* yp = y + (m + e) * incy;
    *yp = (beta == 0.f) ? alpha * p[0][e] : alpha * p[0][e] + beta * *yp;
  }
}

// 'T': A is column-major N x M (A[n + m*lda]); y[m] = alpha * sum_n A[n,m] x[n]
// + beta * y[m].  WPC warps per output, coalesced along the column: 16-byte
// loads, U in flight, where A's columns and x allow them (VEC), else of four
// bytes; reduced by a fixed tree.  HBM-bound (8192 x 8192: one scalar
// load in flight 53 us, 5.1 TB/s; now 41); short columns by the loads' latency
// and the warps in flight, which U = 8 halves.
template <int WPC, bool VEC, int U, bool STREAM>
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
        for (int u = 0; u < U; ++u) v[u] = load_a4<STREAM>(c4 + i + u * T);
#pragma unroll
        for (int u = 0; u < U; ++u) add(v[u], x4[i + u * T]);
      }
      if constexpr (U <= 2) {
        if (i < n4) add(load_a4<STREAM>(c4 + i), x4[i]);
      } else {
        for (; i < n4; i += T) add(load_a4<STREAM>(c4 + i), x4[i]);
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
  // eight loads in flight leave fewer warps an SM: where one warp an output makes
  // many blocks, two 16-byte ones are faster (144896 x 416: 43 us, 51); of four bytes
  // as many as a short column has (94016 x 96: four 10.0 us, eight 13.1)
  const bool many = grid > 5 * device_sms();
  const bool stream = vec && beyond_l2(M, N);
  auto kern = stream ? sgemv_t_kernel<WPC, true, 8, true>
              : vec  ? sgemv_t_kernel<WPC, true, 8, false>
                     : sgemv_t_kernel<WPC, false, 8, false>;
  if constexpr (WPC == 1) {
    if (vec && (N <= 256 || many))
      kern = stream ? sgemv_t_kernel<1, true, 2, true> : sgemv_t_kernel<1, true, 2, false>;
    else if (!vec && N <= 96)
      kern = N <= 32 ? sgemv_t_kernel<1, false, 2, false> : sgemv_t_kernel<1, false, 4, false>;
  }
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
  auto kern = share > 1 ? sgemv_n_kernel<V, W, U, true, false> : sgemv_n_kernel<V, W, U, false, false>;
  if constexpr (V == 4)
    if (beyond_l2(M, N))
      kern = share > 1 ? sgemv_n_kernel<4, W, U, true, true> : sgemv_n_kernel<4, W, U, false, true>;
  return cudaLaunchKernelEx(&cfg, kern, M, N, alpha, A, lda, x, incx, beta, y, incy, share);
}

// vec: 16-byte loads are possible.
cudaError_t launch_gemv_n(int M, int N, float alpha, const float* A, int lda, const float* x,
                          int incx, float beta, float* y, int incy, bool vec, cudaStream_t st) {
  const int sms = device_sms(), blocks = cdiv(M, 128);  // of 128 rows, by 16-byte loads
  if (N <= kGemvColumns) {
    if (vec && blocks >= 16 * sms)
      sgemv_rows_kernel<4><<<cdiv(M, 512), 128, 0, st>>>(M, N, alpha, A, lda, x, incx, beta, y, incy);
    else
      sgemv_rows_kernel<1><<<blocks, 128, 0, st>>>(M, N, alpha, A, lda, x, incx, beta, y, incy);
    return cudaPeekAtLastError();
  }
  if (N <= 256) {
    // few columns: no clusters, whose barriers take longer than the columns (1312 x 160
    // 2.3 us alone, 3.0 in twos); 16-byte loads where their blocks reach most SMs
    // (16384 x 256 3.5 us, 4.5 without; 4096 x 256 3.3 and 2.6); fewer warps a block where
    // there are many blocks, whose sums then cost more than the loads (100000 x 100 5.1
    // us in fours, 6.0 in sixteens; 134571 x 48, unaligned, 6.6 and 13.8; 952 x 32 1.45 in
    // eights, 1.69)
    if (vec && blocks >= 4 * sms)
      return launch_gemv_nw<4, 4, 8>(M, N, alpha, A, lda, x, incx, beta, y, incy, 1, st);
    if (vec && 2 * blocks >= sms)
      return launch_gemv_nw<4, 16, 4>(M, N, alpha, A, lda, x, incx, beta, y, incy, 1, st);
    if (blocks >= sms)
      return launch_gemv_nw<1, 4, 8>(M, N, alpha, A, lda, x, incx, beta, y, incy, 1, st);
    if (N <= 32 || (N <= 96 && 2 * blocks >= sms))
      return launch_gemv_nw<1, 8, 4>(M, N, alpha, A, lda, x, incx, beta, y, incy, 1, st);
    if (N <= 96)  // few blocks: most of a warp's columns in flight (64 x 64 1.67 us, 1.76 in fours)
      return launch_gemv_nw<1, 8, 8>(M, N, alpha, A, lda, x, incx, beta, y, incy, 1, st);
    return launch_gemv_nw<1, 16, 8>(M, N, alpha, A, lda, x, incx, beta, y, incy, 1, st);
  }
  const bool wide = vec && M >= 512;
  const int rows = wide ? blocks : cdiv(M, 32);
  int share = kGemvCluster;
  while (share > 1 && (2LL * rows * share > 5LL * sms || N < 64 * share)) share /= 2;
  if (wide)
    return launch_gemv_nw<4, 16, 4>(M, N, alpha, A, lda, x, incx, beta, y, incy, share, st);
  return launch_gemv_nw<1, 16, 8>(M, N, alpha, A, lda, x, incx, beta, y, incy, share, st);
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
  const int grid = static_cast<int>(std::min<long long>((N + 1023) / 1024, 16LL * device_sms()));
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
  if (!t) {
    const bool vec = ((M | lda) & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
    (void)launch_gemv_n(M, N, alpha, A, lda, x, incx, beta, y, incy, vec, st);
  } else {
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
