// simt.cu -- plain FP32 SIMT SGEMM for sm_103a (the "plain" form).
//
// Replaces the reference's OpenCL gemm_rnn (sgemm_ocl2.h:17-90: 16x16 tile,
// one output per work-item, two local-memory loads per FMA) and its separate
// transpose pass (sgemm_ocl2.h:95-128, :180-199).  Here:
//   * one CTA computes a tile of C: 128 x 256 or 128 x 192 (8 x 16 or 8 x 12
//     registers of a thread, packed FP32 FMAs), 128 x 128 for the columns and the
//     last wave that those leave, or 64 x 64 for small outputs (np_tiles,
//     simt_pick_tile); 16 x 16 compute threads, whose thread 0 issues the copies
//     (64 x 64 and grouped tiles: a ninth warp does);
//   * A and B k-slices (BK = 32) are staged by TMA into a 4-deep shared-memory
//     ring guarded by mbarriers; k-contiguous tiles use the 128-byte swizzle
//     so the float4 fragment reads are bank-conflict free;
//   * transposed operands are handled by the tile layout (an m- or
//     n-contiguous tile) -- no transpose kernel, no extra HBM pass;
//   * ragged edges: TMA zero-fills out-of-range rows/columns/k, the epilogue
//     guards its stores; alpha/beta are fused into the epilogue and C is not
//     read when beta == 0 (sgemm_ocl2.h:86-88).
// Operands whose base or leading dimension break TMA's 16-byte rules are
// first copied into an aligned scratch buffer (simt_scratch_bytes).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "internal.h"
#include "ptx.cuh"
#include "simt.cuh"

namespace ugemm {
namespace {

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

// Position of the 16-byte chunk `q` of row `r` in a 128-byte-row tile written
// by TMA with CU_TENSOR_MAP_SWIZZLE_128B (address bits [4,7) ^= bits [7,10)).
__device__ __forceinline__ int swz_chunk(int r, int q) { return q ^ (r & 7); }

// Two FP32 accumulators side by side in one 64-bit register, and the packed
// FMA that updates both (fma.rn.f32x2: each half rounds as fmaf does).  A
// packed FMA takes one issue slot and one set of register reads for two
// products, which leaves the issue slots that the fragment loads and the
// moves need; scalar FMAs stalled at dispatch at 68% of the FMA pipe.
using Acc2 = unsigned long long;
__device__ __forceinline__ Acc2 pack2(float lo, float hi) {
  Acc2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(Acc2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(Acc2& acc, Acc2 a, Acc2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// Which dimension a pair of accumulators spans.  The operand whose fragment
// already lies in register pairs (float4 loads of consecutive rows or columns)
// is the paired one, and the other is broadcast, which costs nothing.  Where
// both operands are k-contiguous there is none: pairs assembled from two loads
// cost a move each (4096^3 NT: 35 TFLOP/s, 49 with scalar FMAs), and an even and
// an odd k of one element, summed apart, would be another order of summation.
enum class Pair { kN, kM, kNone };
template <bool AK, bool BKM>
constexpr Pair pair_of() { return !BKM ? Pair::kN : !AK ? Pair::kM : Pair::kNone; }

template <int TM, int TN, Pair P>
struct AccTile {
  static constexpr int R = P == Pair::kM ? TM / 2 : TM, C = P == Pair::kN ? TN / 2 : TN;
  Acc2 v[R][C];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < C; ++j) v[i][j] = 0;
  }
  __device__ __forceinline__ float get(int i, int j) const {
    float lo, hi;
    unpack2(v[P == Pair::kM ? i / 2 : i][P == Pair::kN ? j / 2 : j], lo, hi);
    return ((P == Pair::kM ? i : j) & 1) ? hi : lo;
  }
};
template <int TM, int TN>
struct AccTile<TM, TN, Pair::kNone> {
  float v[TM][TN];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) v[i][j] = 0.f;
  }
  __device__ __forceinline__ float get(int i, int j) const { return v[i][j]; }
};

// One k-slice (kBK deep) of the register-blocked product, consumed from a
// staged tile pair.  AK: op(A) rows are k-contiguous (ta == 'N').  BKM: op(B)
// columns are k-contiguous (tb == 'T').  k-contiguous operands are read as
// float4 of 4 k, eight columns of B at a time; the other layout is read per
// k, so few fragment values are live beside the accumulators.
// BOX: columns of B to a box of its map, [32][BOX] in the stage.
template <int TM, int TN, bool AK, bool BKM, int BOX>
__device__ __forceinline__ void simt_consume(const float* As, const float* Bs,
                                             AccTile<TM, TN, pair_of<AK, BKM>()>& acc) {
  constexpr Pair P = pair_of<AK, BKM>();
  constexpr int BM = 16 * TM;
  constexpr int JG = BKM && TN > 8 ? (TN % 8 ? 4 : 8) : TN;  // columns of a B fragment
  constexpr bool A4 = AK || BKM;              // A's fragment covers the 4 k of a step
  const int tid = threadIdx.x;
  const int ty = tid >> 4, tx = tid & 15;
#pragma unroll
  for (int q = 0; q < kBK / 4; ++q) {
    float4 a4[A4 ? TM : 1];   // AK: [row] of 4 k; else [k][TM / 4] of 4 rows
    auto load_a = [&](int kk, float4* v) {  // [32][BM]: rows 64 g + 4 ty + {0..3}
#pragma unroll
      for (int g = 0; g < TM / 4; ++g)
        v[g] = *reinterpret_cast<const float4*>(As + (4 * q + kk) * BM + 64 * g + 4 * ty);
    };
    if constexpr (AK) {  // [BM][32], 128-byte swizzled rows; thread rows ty + 16 i
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int r = ty + 16 * i;
        a4[i] = *reinterpret_cast<const float4*>(As + r * kBK + 4 * swz_chunk(ty, q));
      }
    } else if constexpr (A4) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) load_a(kk, a4 + kk * (TM / 4));
    }
    auto el = [](const float4& v, int e) { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; };
#pragma unroll
    for (int jg = 0; jg < TN / JG; ++jg) {
      float4 b4[BKM ? JG : TN / 4];
      if constexpr (BKM) {  // [BN][32], 128-byte swizzled rows; thread columns tx + 16 j
#pragma unroll
        for (int j = 0; j < JG; ++j) {
          const int c = tx + 16 * (jg * JG + j);
          b4[j] = *reinterpret_cast<const float4*>(Bs + c * kBK + 4 * swz_chunk(tx, q));
        }
      }
      if constexpr (P == Pair::kNone) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < JG; ++j)
              acc.v[i][jg * JG + j] = fmaf(el(a4[i], kk), el(b4[j], kk), acc.v[i][jg * JG + j]);
      } else {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          float4 ak[TM / 4];
          if constexpr (!A4) load_a(kk, ak);
          if constexpr (P == Pair::kN) {
            // thread columns 64 g + 4 tx + {0..3}
#pragma unroll
            for (int g = 0; g < TN / 4; ++g)
              b4[g] = *reinterpret_cast<const float4*>(
                  Bs + 64 * g / BOX * BOX * kBK + (4 * q + kk) * BOX + 64 * g % BOX + 4 * tx);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
              const float v = AK ? el(a4[A4 ? i : 0], kk) : el(ak[i / 4], i % 4);
              const Acc2 a2 = pack2(v, v);
#pragma unroll
              for (int j = 0; j < TN / 2; ++j)
                fma2(acc.v[i][j], a2, j % 2 == 0 ? pack2(b4[j / 2].x, b4[j / 2].y)
                                                 : pack2(b4[j / 2].z, b4[j / 2].w));
            }
          } else {  // Pair::kM: rows from a4, columns broadcast
#pragma unroll
            for (int j = 0; j < JG; ++j) {
              const float v = el(b4[j], kk);
              const Acc2 b2 = pack2(v, v);
#pragma unroll
              for (int i = 0; i < TM / 2; ++i) {
                const float4& x = a4[A4 ? kk * (TM / 4) + i / 2 : 0];
                fma2(acc.v[i][jg * JG + j], i % 2 == 0 ? pack2(x.x, x.y) : pack2(x.z, x.w), b2);
              }
            }
          }
        }
      }
    }
  }
}

// One BM x BN tile's k loop, consuming the TMA ring from stage counter `it`
// (which keeps running across the tiles of a persistent CTA).
template <int TM, int TN, bool AK, bool BKM>
__device__ __forceinline__ bool simt_mainloop(const uint8_t* smem, uint64_t* full, uint64_t* empty,
                                              int nkt, uint32_t& it,
                                              AccTile<TM, TN, pair_of<AK, BKM>()>& acc, int* err) {
  using S = SimtShape<TM, TN>;
  const int lane = threadIdx.x & 31;
  acc.clear();
  for (int kt = 0; kt < nkt; ++kt, ++it) {
    const int s = it % kStages;
    if (!mbar_wait(&full[s], (it / kStages) & 1, err, kDevTimeoutFull)) return false;
    const float* As = reinterpret_cast<const float*>(smem + s * S::STAGE_BYTES);
    simt_consume<TM, TN, AK, BKM, S::BN>(As, As + S::A_BYTES / 4, acc);
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
  }
  return true;
}

// alpha/beta epilogue of one tile from registers; C is not read when beta == 0.
template <int TM, int TN, bool AK, bool BKM>
__device__ __forceinline__ void simt_store(const AccTile<TM, TN, pair_of<AK, BKM>()>& tile,
                                           float* C, int M, int N, int ldc, float alpha, float beta, int m0, int n0,
                                           const Epilogue& epi) {
  const int tid = threadIdx.x;
  const int ty = tid >> 4, tx = tid & 15;
  const bool vec = ((ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int row = m0 + (AK ? ty + 16 * i : 64 * (i / 4) + 4 * ty + (i % 4));
    if (row >= M) continue;
    float* crow = C + static_cast<size_t>(row) * ldc;
    float acc[TN];
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[j] = tile.get(i, j);
    if (BKM) {
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int col = n0 + tx + 16 * j;
        if (col < N) {
          float v = alpha * acc[j];
          if (beta != 0.f) v += beta * crow[col];
          crow[col] = epilogue_apply(v, epi, row);
        }
      }
    } else {
#pragma unroll
      for (int g = 0; g < TN / 4; ++g) {
        const int col = n0 + 64 * g + 4 * tx;
        if (vec && col + 3 < N) {
          float4 v = make_float4(alpha * acc[4 * g], alpha * acc[4 * g + 1],
                                 alpha * acc[4 * g + 2], alpha * acc[4 * g + 3]);
          if (beta != 0.f) {
            const float4 o = *reinterpret_cast<const float4*>(crow + col);
            v.x += beta * o.x; v.y += beta * o.y; v.z += beta * o.z; v.w += beta * o.w;
          }
          v.x = epilogue_apply(v.x, epi, row); v.y = epilogue_apply(v.y, epi, row);
          v.z = epilogue_apply(v.z, epi, row); v.w = epilogue_apply(v.w, epi, row);
          *reinterpret_cast<float4*>(crow + col) = v;
        } else {
#pragma unroll
          for (int jj = 0; jj < 4; ++jj)
            if (col + jj < N) {
              float v = alpha * acc[4 * g + jj];
              if (beta != 0.f) v += beta * crow[col + jj];
              crow[col + jj] = epilogue_apply(v, epi, row);
            }
        }
      }
    }
  }
}

__device__ __forceinline__ void raster_tile(int local, int tiles_m, int tiles_n, int& tile_m,
                                            int& tile_n) {
  const int per_group = kRaster * tiles_n;
  const int first_m = (local / per_group) * kRaster;
  const int group_rows = min(tiles_m - first_m, kRaster);
  tile_m = first_m + (local % per_group) % group_rows;
  tile_n = (local % per_group) / group_rows;
}

template <int TM, int TN, bool AK, bool BKM>
__global__ void __launch_bounds__(kThreads, AK && BKM ? 1 : 2)
    simt_sgemm_kernel(const __grid_constant__ CUtensorMap tmA,
                      const __grid_constant__ CUtensorMap tmB, float* __restrict__ C, int M,
                      int N, int K, int ldc, float alpha, float beta, Epilogue epi, int tiles_m,
                      int tiles_n, int* err) {
  using S = SimtShape<TM, TN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * S::STAGE_BYTES);
  uint64_t* empty = full + kStages;
  int tile_m, tile_n;
  raster_tile(blockIdx.x, tiles_m, tiles_n, tile_m, tile_n);
  const int m0 = tile_m * S::BM, n0 = tile_n * S::BN;
  const int nkt = (K + kBK - 1) / kBK;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kConsumerWarps);
    }
    fence_barrier_init();
  }
  __syncthreads();

  if (warp == kConsumerWarps) {  // ---------------- TMA producer warp
    if (lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      for (int kt = 0; kt < nkt; ++kt) {
        const int s = kt % kStages;
        const uint32_t ph = (kt / kStages) & 1;
        if (!mbar_wait(&empty[s], ph ^ 1, err, kDevTimeoutEmpty)) break;
        uint8_t* sa = smem + s * S::STAGE_BYTES;
        uint8_t* sb = sa + S::A_BYTES;
        mbar_arrive_expect_tx(&full[s], S::STAGE_BYTES);
        if (AK) tma_load_2d(sa, &tmA, &full[s], kt * kBK, m0);
        else    tma_load_2d(sa, &tmA, &full[s], m0, kt * kBK);
        if (BKM) tma_load_2d(sb, &tmB, &full[s], kt * kBK, n0);
        else     tma_load_2d(sb, &tmB, &full[s], n0, kt * kBK);
      }
    }
    return;
  }
  AccTile<TM, TN, pair_of<AK, BKM>()> acc;
  uint32_t it = 0;
  if (!simt_mainloop<TM, TN, AK, BKM>(smem, full, empty, nkt, it, acc, err)) return;
  simt_store<TM, TN, AK, BKM>(acc, C, M, N, ldc, alpha, beta, m0, n0, epi);
}

// Producer-less variant: 8 warps only.  With no ninth warp every thread may
// hold up to 255 registers (a ninth warp caps each scheduler's share at 168),
// room for the 8 x 16 register block.  Thread 0 issues the TMA for stage
// kt + S - 1 once all warps released the stage they consumed at kt - 1.
//
// What bounds it: a 128-bit shared load costs a warp four wavefronts, so an
// 8 x 8 block (16 words read for 64 FMAs) keeps the shared-memory pipe as
// busy as the FMA pipe and both reach about 70%; an 8 x 16 block reads 24
// words for 128 FMAs, three quarters of that.  128 x 256 tiles are coarse,
// so the last of them, which would not fill a wave of SMs, run as two
// 128 x 128 tiles each (CTAs from `wide_tiles` on); 8 x 12 blocks, 128 x 192
// tiles, fill the waves of some outputs better (np_tiles).
template <int TM, int TN, bool AK, bool BKM, int BOX>
__device__ __forceinline__ void simt_np_tile(uint8_t* smem, const CUtensorMap& tmA,
                                             const CUtensorMap& tmB, float* __restrict__ C, int M,
                                             int N, int K, int ldc, float alpha, float beta,
                                             const Epilogue& epi, int m0, int n0, int* err) {
  using S = SimtShape<TM, TN>;
  using W = SimtShape<8, 16>;  // the ring's layout (and the barriers') is the wide tile's
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * W::STAGE_BYTES);
  uint64_t* empty = full + kStages;
  const int nkt = (K + kBK - 1) / kBK;
  const int tid = threadIdx.x, lane = tid & 31;
  auto issue = [&](int kt) {
    const int s = kt % kStages;
    uint8_t* sa = smem + s * W::STAGE_BYTES;
    uint8_t* sb = sa + S::A_BYTES;
    mbar_arrive_expect_tx(&full[s], S::STAGE_BYTES);
    if (AK) tma_load_2d(sa, &tmA, &full[s], kt * kBK, m0);
    else    tma_load_2d(sa, &tmA, &full[s], m0, kt * kBK);
#pragma unroll
    for (int h = 0; h < S::BN / BOX; ++h) {
      if (BKM) tma_load_2d(sb + h * BOX * kBK * 4, &tmB, &full[s], kt * kBK, n0 + BOX * h);
      else     tma_load_2d(sb + h * BOX * kBK * 4, &tmB, &full[s], n0 + BOX * h, kt * kBK);
    }
  };
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kConsumerWarps);
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int kt = 0; kt < min(kStages - 1, nkt); ++kt) issue(kt);  // first use of each stage
  }
  __syncthreads();
  AccTile<TM, TN, pair_of<AK, BKM>()> acc;
  acc.clear();
  for (int kt = 0; kt < nkt; ++kt) {
    if (tid == 0) {
      const int kn = kt + kStages - 1;
      if (kn < nkt) {
        if (!mbar_wait(&empty[kn % kStages], ((kn / kStages) & 1) ^ 1, err, kDevTimeoutEmpty))
          return;
        issue(kn);
      }
    }
    const int s = kt % kStages;
    if (!mbar_wait(&full[s], (kt / kStages) & 1, err, kDevTimeoutFull)) return;
    const float* As = reinterpret_cast<const float*>(smem + s * W::STAGE_BYTES);
    simt_consume<TM, TN, AK, BKM, BOX>(As, As + S::A_BYTES / 4, acc);
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
  }
  simt_store<TM, TN, AK, BKM>(acc, C, M, N, ldc, alpha, beta, m0, n0, epi);
}

template <bool AK, bool BKM, int WT>
__global__ void __launch_bounds__(kConsumerWarps * 32, 1)
    simt_sgemm_np_kernel(const __grid_constant__ CUtensorMap tmA,
                         const __grid_constant__ CUtensorMap tmB, float* __restrict__ C, int M,
                         int N, int K, int ldc, float alpha, float beta, Epilogue epi,
                         int tiles_m, int tiles_n, int wide_tiles, int* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  // tiles_m x tiles_n tiles of 128 x W in raster order
  constexpr int W = 16 * WT, BOX = W % 128 == 0 ? 128 : 64;
  const int b = blockIdx.x;
  int tile_m, tile_n;
  if (b < wide_tiles) {
    if constexpr (pair_of<AK, BKM>() != Pair::kNone) {
      raster_tile(b, tiles_m, tiles_n, tile_m, tile_n);
      simt_np_tile<8, WT, AK, BKM, BOX>(smem, tmA, tmB, C, M, N, K, ldc, alpha, beta, epi,
                                   tile_m * 128, tile_n * W, err);
    }
  } else {
    raster_tile(wide_tiles + (b - wide_tiles) / 2, tiles_m, tiles_n, tile_m, tile_n);
    const int n0 = tile_n * W + ((b - wide_tiles) & 1) * 128;
    const int n1 = min(N, (tile_n + 1) * W);  // the next tile's columns are not this one's
    if (n0 < n1)
      simt_np_tile<8, 8, AK, BKM, BOX>(smem, tmA, tmB, C, M, n1, K, ldc, alpha, beta, epi,
                                  tile_m * 128, n0, err);
  }
}

// Persistent grouped SIMT GEMM: one CTA per SM walks the tiles of all
// problems.  The batched pre-pass packed every operand row-contiguous per k
// (A as K x M, B as K x N), the layout with 512-byte TMA rows that this kernel
// reads fastest, so all problems use the (!AK, !BKM) path.
template <int TM, int TN>
__global__ void __launch_bounds__(kThreads, 1)
    simt_grouped_kernel(const CUtensorMap* __restrict__ maps, const SimtProblem* __restrict__ probs,
                        int nprob, int total_tiles, int* err) {
  using S = SimtShape<TM, TN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * S::STAGE_BYTES);
  uint64_t* empty = full + kStages;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kConsumerWarps);
    }
    fence_barrier_init();
  }
  __syncthreads();
  auto locate = [&](int t, SimtProblem& P, int& p, int& m0, int& n0) {
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (probs[mid].tile_start <= t) lo = mid; else hi = mid - 1;
    }
    p = lo;
    P = probs[lo];
    int tm, tn;
    raster_tile(t - P.tile_start, P.tiles_m, P.tiles_n, tm, tn);
    m0 = tm * S::BM;
    n0 = tn * S::BN;
  };
  if (warp == kConsumerWarps) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < total_tiles; t += gridDim.x) {
        SimtProblem P;
        int p, m0, n0;
        locate(t, P, p, m0, n0);
        const CUtensorMap* ma = &maps[2 * p];
        const CUtensorMap* mb = &maps[2 * p + 1];
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(
                         reinterpret_cast<uint64_t>(ma)) : "memory");
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(
                         reinterpret_cast<uint64_t>(mb)) : "memory");
        for (int kt = 0; kt < P.nkt; ++kt, ++it) {
          const int s = it % kStages;
          const uint32_t ph = (it / kStages) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, err, kDevTimeoutEmpty)) { ok = false; break; }
          uint8_t* sa = smem + s * S::STAGE_BYTES;
          mbar_arrive_expect_tx(&full[s], S::STAGE_BYTES);
          tma_load_2d(sa, ma, &full[s], m0, (P.kt0 + kt) * kBK);
          tma_load_2d(sa + S::A_BYTES, mb, &full[s], n0, (P.kt0 + kt) * kBK);
        }
      }
    }
    return;
  }
  uint32_t it = 0;
  for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
    SimtProblem P;
    int p, m0, n0;
    locate(t, P, p, m0, n0);
    AccTile<TM, TN, Pair::kN> acc;
    if (!simt_mainloop<TM, TN, false, false>(smem, full, empty, P.nkt, it, acc, err)) return;
    simt_store<TM, TN, false, false>(acc, P.C, P.M, P.N, P.ldc, P.alpha, P.beta, m0, n0, P.epi);
  }
}

// Batched pre-pass of the grouped SIMT form: copy op(X) (element (r, k) at
// src[r*sr + k*sk]) to dst[k*ld + r] (rows contiguous per k), 32 x 64 tiles
// through shared memory so both source layouts read and write coalesced.
__global__ void __launch_bounds__(256) pack_kmajor_batched_kernel(const PackJob* __restrict__ jobs,
                                                                  int njobs, int total_tiles) {
  __shared__ float tile[32][65];
  __shared__ int starts[2048];
  const int cached = min(njobs, 2048);
  for (int i = threadIdx.x; i < cached; i += blockDim.x) starts[i] = jobs[i].tile_start;
  __syncthreads();
  for (int b = blockIdx.x; b < total_tiles; b += gridDim.x) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const int st = njobs <= 2048 ? starts[mid] : jobs[mid].tile_start;
    if (st <= b) lo = mid; else hi = mid - 1;
  }
  const PackJob j = jobs[lo];
  const int local = b - j.tile_start;
  const int tiles_k = (j.K + 63) / 64;
  const int r0 = (local / tiles_k) * 32, k0 = (local % tiles_k) * 64;
  const int t = threadIdx.x;
  if (j.gather) {  // implicit im2col: this thread's pixel is fixed, taps vary
    const int pix = j.gather == 2 ? k0 + (t & 63) : r0 + (t & 31);
    const Im2colPix px = im2col_pix(j.im, pix);
    const int npix = j.gather == 2 ? j.K : j.rows;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (j.gather == 2) {  // rows are taps
        const int rr = (t >> 6) + 4 * i, r = r0 + rr;
        tile[rr][t & 63] = (r < j.rows && pix < npix) ? im2col_load(j.im, im2col_tap(j.im, r), px)
                                                       : 0.f;
      } else {              // rows are pixels
        const int kk = (t >> 5) + 8 * i, k = k0 + kk;
        tile[t & 31][kk] = (k < j.K && pix < npix) ? im2col_load(j.im, im2col_tap(j.im, k), px)
                                                    : 0.f;
      }
    }
  } else if (j.sk == 1) {
    const int k = k0 + (t & 63);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int rr = (t >> 6) + 4 * i, r = r0 + rr;
      tile[rr][t & 63] = (r < j.rows && k < j.K) ? j.src[r * j.sr + k] : 0.f;
    }
  } else {
    const int rr = t & 31, r = r0 + rr;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int kk = (t >> 5) + 8 * i, k = k0 + kk;
      tile[rr][kk] = (r < j.rows && k < j.K) ? j.src[r * j.sr + k * j.sk] : 0.f;
    }
  }
  __syncthreads();
  {
    const int rr = t & 31, r = r0 + rr;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int kk = (t >> 5) + 8 * i, k = k0 + kk;
      if (r < j.rows && k < j.K) j.dst[static_cast<size_t>(k) * j.ld + r] = tile[rr][kk];
    }
  }
  __syncthreads();  // the tile buffer is refilled by the next iteration
  }
}

// Copy a rows x cols row-major matrix into a dense buffer whose rows are
// `ldd` floats (a multiple of 4) so that TMA can describe it.
__global__ void pack_rows_kernel(const float* __restrict__ src, int lds, float* __restrict__ dst,
                                 int ldd, int rows, int cols) {
  const size_t total = static_cast<size_t>(rows) * ldd;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total;
       i += size_t(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / ldd), c = static_cast<int>(i % ldd);
    dst[i] = (c < cols) ? src[static_cast<size_t>(r) * lds + c] : 0.f;
  }
}

__global__ void scale_kernel(float* __restrict__ C, int M, int N, int ldc, float beta) {
  const size_t total = static_cast<size_t>(M) * N;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total;
       i += size_t(gridDim.x) * blockDim.x) {
    float* p = C + (i / N) * static_cast<size_t>(ldc) + (i % N);
    *p = (beta == 0.f) ? 0.f : beta * *p;
  }
}

bool tma_ok(const void* p, int ld) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && (ld % 4) == 0;
}

// Stored shape (rows, cols) of an operand.
void stored_a(const Gemm& g, int& rows, int& cols) {
  if (g.ta == 'N') { rows = g.M; cols = g.K; } else { rows = g.K; cols = g.M; }
}
void stored_b(const Gemm& g, int& rows, int& cols) {
  if (g.tb == 'N') { rows = g.K; cols = g.N; } else { rows = g.N; cols = g.K; }
}

// The producer-less kernel's tiles for an M x N output.  Costs in k of a full wave
// of 128 x 256 tiles (174 us per 1024), K in whole stages: each width's share per k,
// and what a wave takes beside (prologue, stores; less of it in the first wave, whose
// stores go to L2), fitted to ten outputs at K = 8 to 1024.  Shallow products are bound by
// the latter: 4096 x 4096 x 32 takes 47 us in 128 x 128 tiles and 56 in wide ones,
// 6000 x 6000 x 32 101 and 129.  Without pairs there are no wide tiles.  Wide
// tiles fill whole waves of SMs; what is left of them runs as narrow ones when
// those fit in one wave, and everything runs narrow where that takes less time (a
// right edge that leaves half of the wide tiles empty).
constexpr double kWideFixed = 100, kWideFirst = 0.42;
constexpr double kNarrowCost = 0.56, kNarrowFixed = 27.5;  // 128 wide
constexpr double kMiddleCost = 0.78, kMiddleFixed = 55;  // 192 wide
// 64 x 64 tiles, two CTAs to an SM: a round of two to an SM, or of one at most;
// slower where both operands are k-contiguous (4096 x 4096 x 32: 84 us, 49 otherwise)
constexpr double kSmallCost = 0.375, kSmallHalfCost = 0.29, kSmallFixed = 11.4;
constexpr double kSmallCostNT = 0.40, kSmallFixedNT = 21.5;
struct NpTiles {
  int width = 256;             // of the wide tiles
  int tiles_m = 0, tiles_n = 0, wide = 0;  // wide tiles, and how many run as such
  double cost = 0;
};
NpTiles np_tiles(int M, int N, int K, bool wide_ok, int sms) {
  K = cdiv(K, kBK) * kBK;
  const double narrow = kNarrowCost * K + kNarrowFixed;  // a wave of 128 x 128 tiles
  NpTiles best;
  best.tiles_m = cdiv(M, 128);
  best.tiles_n = cdiv(N, 256);
  best.cost = narrow * cdiv(best.tiles_m * cdiv(N, 128), sms);
  for (int width : {256, 192}) {
    if (!wide_ok) break;
    NpTiles t;
    t.width = width;
    t.tiles_m = cdiv(M, 128);
    t.tiles_n = cdiv(N, width);
    const int total = t.tiles_m * t.tiles_n, rest = total % sms;
    const bool tail = rest > 0 && 2 * rest <= sms;
    const double fixed = width == 256 ? kWideFixed : kMiddleFixed;
    const double wave = (width == 256 ? 1.0 : kMiddleCost) * K + fixed;
    const int waves = total / sms + (rest > 0 && !tail ? 1 : 0);
    t.wide = tail ? total - rest : total;
    t.cost = wave * waves + (tail ? narrow : 0.0) - (waves > 0 ? kWideFirst * fixed : 0.0);
    if (t.cost < best.cost) best = t;
  }
  return best;
}

// Boxes of 32 k by rows_a rows of op(A), rows_b columns of op(B).
template <bool AK, bool BKM>
bool encode_operands(const Gemm& g, const float* A, int lda, const float* B, int ldb, int rows_a,
                     int rows_b, CUtensorMap* ta, CUtensorMap* tb) {
  const CUtensorMapDataType f32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  return (AK ? encode_tmap_2d(ta, f32, 4, A, g.K, g.M, lda * 4ull, kBK, rows_a,
                              CU_TENSOR_MAP_SWIZZLE_128B)
             : encode_tmap_2d(ta, f32, 4, A, g.M, g.K, lda * 4ull, rows_a, kBK,
                              CU_TENSOR_MAP_SWIZZLE_NONE)) &&
         (BKM ? encode_tmap_2d(tb, f32, 4, B, g.K, g.N, ldb * 4ull, kBK, rows_b,
                               CU_TENSOR_MAP_SWIZZLE_128B)
              : encode_tmap_2d(tb, f32, 4, B, g.N, g.K, ldb * 4ull, rows_b, kBK,
                               CU_TENSOR_MAP_SWIZZLE_NONE));
}

// tile: kSimt64x64 (a producer warp), or the producer-less kernel.
template <bool AK, bool BKM>
ugemm_status launch_t(const Gemm& g, int tile, const float* A, int lda, const float* B, int ldb,
                      int* dev_err, cudaStream_t st) {
  CUtensorMap ta, tb;
  if (tile == kSimt64x64) {
    using S = SimtShape<4, 4>;
    if (!encode_operands<AK, BKM>(g, A, lda, B, ldb, S::BM, S::BN, &ta, &tb)) return UGEMM_ERR_CUDA;
    auto kern = simt_sgemm_kernel<4, 4, AK, BKM>;
    static std::atomic<uint64_t> attr_done{0};  // per instantiation and device
    if (!smem_attr_once(kern, S::SMEM, attr_done)) return UGEMM_ERR_CUDA;
    const int tiles_m = cdiv(g.M, S::BM), tiles_n = cdiv(g.N, S::BN);
    prof_begin(st);
    kern<<<tiles_m * tiles_n, kThreads, S::SMEM, st>>>(ta, tb, g.C, g.M, g.N, g.K, g.ldc, g.alpha,
                                                       g.beta, g.epi, tiles_m, tiles_n, dev_err);
  } else {
    using S = SimtShape<8, 16>;
    constexpr bool wide_ok = pair_of<AK, BKM>() != Pair::kNone;
    NpTiles t = np_tiles(g.M, g.N, g.K, wide_ok, device_sms());
    if (tile != kSimtMixed) {
      t.width = 256;
      t.tiles_n = cdiv(g.N, 256);
      t.wide = tile == kSimt128x256 && wide_ok ? t.tiles_m * t.tiles_n : 0;
    }
    if (!encode_operands<AK, BKM>(g, A, lda, B, ldb, 128, t.width == 192 ? 64 : 128, &ta, &tb))
      return UGEMM_ERR_CUDA;
    auto kern = t.width == 192 ? simt_sgemm_np_kernel<AK, BKM, 12> : simt_sgemm_np_kernel<AK, BKM, 16>;
    static std::atomic<uint64_t> attr_done[2];  // per instantiation and device
    if (!smem_attr_once(kern, S::SMEM, attr_done[t.width == 192])) return UGEMM_ERR_CUDA;
    const int total = t.tiles_m * t.tiles_n;
    prof_begin(st);
    kern<<<t.wide + 2 * (total - t.wide), kConsumerWarps * 32, S::SMEM, st>>>(
        ta, tb, g.C, g.M, g.N, g.K, g.ldc, g.alpha, g.beta, g.epi, t.tiles_m, t.tiles_n, t.wide,
        dev_err);
  }
  prof_end(st, kProfSimt);
  return cudaPeekAtLastError() == cudaSuccess ? UGEMM_OK : UGEMM_ERR_CUDA;
}

}  // namespace

size_t simt_scratch_bytes(const Gemm& g) {
  size_t bytes = 0;
  int r, c;
  if (!tma_ok(g.A, g.lda)) { stored_a(g, r, c); bytes += align_up(size_t(r) * align_up(c, 4) * 4, 256); }
  if (!tma_ok(g.B, g.ldb)) { stored_b(g, r, c); bytes += align_up(size_t(r) * align_up(c, 4) * 4, 256); }
  return bytes;
}

int simt_pick_tile(const Gemm& g) {
  static const int forced = [] {
    const char* e = std::getenv("UGEMM_SIMT_TILE");
    const int v = e ? std::atoi(e) : -1;
    return v >= 0 && v < kSimtTileCount ? v : -1;
  }();
  if (forced >= 0) return forced;
  // whichever needs less time by the waves' measured costs (2048^3 NN: 348 us
  // mixed, 464 in 64x64 tiles; 1024^3: 99 and 74)
  const int sms = device_sms();
  const long small = long(cdiv(g.M, 64)) * cdiv(g.N, 64);
  const bool wide_ok = !(g.ta == 'N' && g.tb == 'T');
  const double fixed = wide_ok ? kSmallFixed : kSmallFixedNT, k = cdiv(g.K, kBK) * kBK;
  const double small_cost =
      small <= sms ? kSmallHalfCost * k + fixed
                   : ((wide_ok ? kSmallCost : kSmallCostNT) * k + fixed) *
                         ((small + 2 * sms - 1) / (2 * sms));
  return np_tiles(g.M, g.N, g.K, wide_ok, sms).cost < small_cost ? kSimtMixed : kSimt64x64;
}

ugemm_status simt_launch(const Gemm& g, int tile, Scratch ws, int* dev_err, cudaStream_t st) {
  const float* A = g.A;
  const float* B = g.B;
  int lda = g.lda, ldb = g.ldb;
  uint8_t* wp = static_cast<uint8_t*>(ws.ptr);
  size_t used = 0;
  int r, c;
  if (!tma_ok(A, lda)) {
    stored_a(g, r, c);
    const int ld = static_cast<int>(align_up(c, 4));
    const size_t need = align_up(size_t(r) * ld * 4, 256);
    if (used + need > ws.bytes) return UGEMM_ERR_ARENA_TOO_SMALL;
    float* dst = reinterpret_cast<float*>(wp + used);
    prof_begin(st);
    pack_rows_kernel<<<std::min<size_t>(4096, (size_t(r) * ld + 255) / 256), 256, 0, st>>>(
        A, lda, dst, ld, r, c);
    prof_end(st, kProfAux);
    A = dst; lda = ld; used += need;
  }
  if (!tma_ok(B, ldb)) {
    stored_b(g, r, c);
    const int ld = static_cast<int>(align_up(c, 4));
    const size_t need = align_up(size_t(r) * ld * 4, 256);
    if (used + need > ws.bytes) return UGEMM_ERR_ARENA_TOO_SMALL;
    float* dst = reinterpret_cast<float*>(wp + used);
    prof_begin(st);
    pack_rows_kernel<<<std::min<size_t>(4096, (size_t(r) * ld + 255) / 256), 256, 0, st>>>(
        B, ldb, dst, ld, r, c);
    prof_end(st, kProfAux);
    B = dst; ldb = ld; used += need;
  }
  const bool ak = g.ta == 'N', bk = g.tb == 'T';
  if (ak && !bk) return launch_t<true, false>(g, tile, A, lda, B, ldb, dev_err, st);
  if (ak && bk) return launch_t<true, true>(g, tile, A, lda, B, ldb, dev_err, st);
  if (!ak && !bk) return launch_t<false, false>(g, tile, A, lda, B, ldb, dev_err, st);
  return launch_t<false, true>(g, tile, A, lda, B, ldb, dev_err, st);
}

ugemm_status scale_c_launch(const Gemm& g, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0 || g.beta == 1.f) return UGEMM_OK;
  const size_t total = size_t(g.M) * g.N;
  prof_begin(st);
  scale_kernel<<<std::min<size_t>(4096, (total + 255) / 256), 256, 0, st>>>(g.C, g.M, g.N, g.ldc,
                                                                            g.beta);
  prof_end(st, kProfAux);
  return cudaPeekAtLastError() == cudaSuccess ? UGEMM_OK : UGEMM_ERR_CUDA;
}

int simt_block(int tile) { return tile == kSimt64x64 ? 64 : 128; }

bool simt_encode_grouped(int tile, const float* a, int M, const float* b, int N, int K, int ld_a,
                         int ld_b, CUtensorMap* ta, CUtensorMap* tb) {
  const int bm = simt_block(tile);
  return encode_tmap_2d(ta, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a, M, std::max(K, 1), ld_a * 4ull,
                        bm, kBK, CU_TENSOR_MAP_SWIZZLE_NONE) &&
         encode_tmap_2d(tb, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, b, N, std::max(K, 1), ld_b * 4ull,
                        bm, kBK, CU_TENSOR_MAP_SWIZZLE_NONE);
}

namespace {
template <int TM, int TN>
ugemm_status grouped_t(const CUtensorMap* maps, const SimtProblem* probs, int nprob, int total,
                       int max_ctas, int* dev_err, cudaStream_t st) {
  using S = SimtShape<TM, TN>;
  auto kern = simt_grouped_kernel<TM, TN>;
  static std::atomic<uint64_t> attr_done{0};  // per instantiation and device
  if (!smem_attr_once(kern, S::SMEM, attr_done)) return UGEMM_ERR_CUDA;
  const int grid = std::max(1, std::min(total, max_ctas > 0 ? max_ctas : device_sms()));
  prof_begin(st);
  kern<<<grid, kThreads, S::SMEM, st>>>(maps, probs, nprob, total, dev_err);
  prof_end(st, kProfGrouped);
  return cudaPeekAtLastError() == cudaSuccess ? UGEMM_OK : UGEMM_ERR_CUDA;
}
}  // namespace

ugemm_status simt_grouped_launch(int tile, const CUtensorMap* maps, const SimtProblem* probs,
                                 int nprob, int total_tiles, int max_ctas, int* dev_err,
                                 cudaStream_t st) {
  if (total_tiles <= 0) return UGEMM_OK;
  if (tile == kSimt64x64) return grouped_t<4, 4>(maps, probs, nprob, total_tiles, max_ctas, dev_err, st);
  return grouped_t<8, 8>(maps, probs, nprob, total_tiles, max_ctas, dev_err, st);
}

ugemm_status pack_batched_launch(const PackJob* jobs, int njobs, int total_tiles, cudaStream_t st) {
  if (total_tiles <= 0) return UGEMM_OK;
  prof_begin(st);
  pack_kmajor_batched_kernel<<<std::min(total_tiles, device_sms() * 8), 256, 0, st>>>(jobs, njobs,
                                                                             total_tiles);
  prof_end(st, kProfSplitPrep);
  return cudaPeekAtLastError() == cudaSuccess ? UGEMM_OK : UGEMM_ERR_CUDA;
}

}  // namespace ugemm
