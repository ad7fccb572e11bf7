// multi.cu -- a few split-precision GEMMs, and split-K slices of them, in one
// persistent launch of the grouped tensor-core kernel, with all scratch in
// the caller's workspace: no plan, no allocation, nothing read from host
// memory at run time (the problem table is the GEMM kernel's parameter), so
// it is usable inside stream capture.
//
// Used where one GEMM launch at a time leaves SMs idle:
//   * ugemm_sgemm_backward: dA = alpha dC op(B)^T and dB = alpha op(A)^T dC
//     share one launch, so the tiles of both fill the GPU together;
//   * single GEMMs whose whole tiles leave SMs idle: narrower tiles, or k
//     slices whose FP32 partial tiles one reduce launch sums in a fixed order.
// Each GEMM may also be computed transposed (C^T = op(B)^T op(A)^T) when
// that wastes less of the 128-row tiles, as in grouped plans.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstring>

#include "internal.h"
#include "split_tc.cuh"

namespace ugemm {
namespace {

static_assert(sizeof(MultiTable) <= 16384, "a kernel parameter, copied at every launch");

MultiTable empty_table() {
  MultiTable t;
  std::memset(&t, 0, sizeof t);
  for (TcProblem& p : t.probs) p.tile_start = INT_MAX;
  return t;
}

double padded(int rows, int cols, int bn) {
  return double(align_up(rows, 128)) * ((cols / bn) * bn + align_up(cols % bn, 16));
}

// Slices whose partial tiles take 512 MiB.
int most_slices(const Gemm& g) {
  return std::max(1, static_cast<int>(std::min(1e9, double(512 << 20) / (double(g.M) * g.N * 4))));
}

// The tiles that several GEMMs share an SM's time by: 256-wide unless every
// output is narrow in its better orientation.
struct Shared {
  int block_n = 256;
  bool swap[kMultiMax];
  int nkb[kMultiMax];
  double fair = 0;  // half an SM's share of the stages
};
Shared shared_tiles(const Gemm* gs, int n, int pieces, int sms) {
  Shared h;
  int widest = 0;
  for (int i = 0; i < n; ++i) {
    const Gemm& g = gs[i];
    widest = std::max(widest, padded(g.N, g.M, 256) < padded(g.M, g.N, 256) ? g.M : g.N);
  }
  h.block_n = widest > 128 ? 256 : 128;
  for (int i = 0; i < n; ++i) {
    const Gemm& g = gs[i];
    const bool sw = h.swap[i] = padded(g.N, g.M, h.block_n) < padded(g.M, g.N, h.block_n);
    h.nkb[i] = split_nkb(pieces, g.K);
    h.fair += double(cdiv(sw ? g.N : g.M, kTcBM)) * cdiv(sw ? g.M : g.N, h.block_n) * h.nkb[i];
  }
  h.fair /= 2.0 * sms;
  return h;
}

// The longest chain of FP32 sums of one GEMM (choose_geometry): its slice, were
// it cut so that its tiles are half an SM's share each.
int longest_sum(const Gemm& g, int pieces, int sms) {
  const Shared h = shared_tiles(&g, 1, pieces, sms);
  return slice_blocks(h.nkb[0], h.fair, std::min(kMultiSubs, most_slices(g)));
}

}  // namespace

// One GEMM: the tile width and slices of the least time by the stage times.
// Several: slices no longer than half an SM's fair share, which round robin
// then balances (2048 x 8192 x 1024 backward: 342 us, 435 with whole tiles on
// each GEMM's share of the SMs).
MultiLayout multi_layout(const Gemm* gs, int n, const SplitPlan& p, bool whole_k) {
  MultiLayout L;
  const int sms = device_sms();
  if (n == 1) {
    const int slices = whole_k ? 1 : std::min(kMultiSubs, most_slices(gs[0]));
    const int nkb = split_nkb(p.pieces, gs[0].K);
    // (without slices, only 64-wide tiles, three pieces', keep the sums short)
    const int longest = L.longest =
        whole_k && p.pieces != 3 ? nkb : longest_sum(gs[0], p.pieces, sms);
    L.us = 1e300;
    for (int bn : {64, 128, 256}) {
      if (bn == 64 && p.pieces != 3) continue;
      const GeoChoice c = choose_geometry(p.pieces, gs[0].M, gs[0].N, nkb, sms, bn, true, slices,
                                          longest);
      if (c.us >= L.us) continue;
      L.us = c.us;
      L.block_n = bn;
      L.geo[0] = c;
    }
    // the pieces' traffic (16 bytes an element) against slower stages: fused
    // where one side of the output is short
    L.us += split_pass_us((double(gs[0].M) + gs[0].N) * gs[0].K);
    if (p.pieces == 3 && p.products == 6 && fusable(gs[0]) && !writes_operands(gs, 1)) {
      GeoChoice c;
      c.us = fused_us(gs[0], sms, &c.swap, &c.slices, slices, longest);
      if (c.us < L.us) {
        c.per = cdiv(nkb, c.slices);
        L.us = c.us;
        L.block_n = 128;
        L.geo[0] = c;
        L.fused = true;
      }
    }
  } else {
    const Shared h = shared_tiles(gs, n, p.pieces, sms);
    L.block_n = h.block_n;
    int subs = n;
    for (int i = 0; i < n; ++i) {
      GeoChoice& o = L.geo[i];
      o.swap = h.swap[i];
      o.per = slice_blocks(h.nkb[i], h.fair, std::min(kMultiSubs - (subs - 1), most_slices(gs[i])));
      o.slices = cdiv(h.nkb[i], o.per);
      subs += o.slices - 1;
    }
  }
  size_t off = 0;
  for (int i = 0; i < n; ++i) {
    L.a_off[i] = L.b_off[i] = off;
    if (L.fused) continue;  // no pieces in memory
    off += split_operand_bytes(p.pieces, gs[i].M, gs[i].K);
    L.b_off[i] = off;
    off += split_operand_bytes(p.pieces, gs[i].N, gs[i].K);
  }
  for (int i = 0; i < n; ++i) {
    L.part_off[i] = off;
    if (L.geo[i].slices > 1) off += align_up(size_t(L.geo[i].slices) * gs[i].M * gs[i].N * 4, 256);
  }
  L.total = align_up(off, 256);
  return L;
}

TailPlan tail_plan(const Gemm& g, const SplitPlan& p) {
  TailPlan t;
  if (g.M == 0 || g.N == 0 || g.K == 0 || g.alpha == 0.f) return t;
  const int sms = device_sms();
  const int tiles_m = cdiv(g.M, kTcBM), tiles_n = cdiv(g.N, p.block_n);
  const int tiles = tiles_m * tiles_n, rem = tiles % sms;
  if (tiles <= sms || rem == 0 || split_nkb(p.pieces, g.K) < 2 * kMinSlice) return t;
  // the raster order ends with the last group of tile rows, column by column
  const int first_m = ((tiles_m - 1) / kTcRaster) * kTcRaster, rows = tiles_m - first_m;
  const int cols = cdiv(rem, rows);             // whole tile columns of that group
  if (cols >= tiles_n || 2 * cols * rows > sms) return t;
  t.use = true;
  t.main_tiles = tiles - cols * rows;
  t.r0 = first_m * kTcBM;
  t.c0 = (tiles_n - cols) * p.block_n;
  return t;
}

size_t tail_scratch_bytes(const Gemm& g, const SplitPlan& p) {
  const TailPlan t = tail_plan(g, p);
  if (!t.use) return 0;
  return align_up(2 * size_t(g.M - t.r0) * (g.N - t.c0) * 4, 256);
}

ugemm_status tail_launch(const Gemm& g, const SplitPlan& p, const TailPlan& tail,
                         const void* a_pieces, const void* b_pieces, void* scratch, int* dev_err,
                         cudaStream_t st) {
  const int Mt = g.M - tail.r0, Nt = g.N - tail.c0, Kp = split_kp(g.K);
  const size_t mn = size_t(Mt) * Nt;
  float* part = static_cast<float*>(scratch);
  MultiTable t = empty_table();
  const size_t row_bytes = size_t(Kp) * piece_bytes(p.pieces);
  const auto* ap = static_cast<const uint8_t*>(a_pieces) + size_t(tail.r0) * row_bytes;
  const auto* bp = static_cast<const uint8_t*>(b_pieces) + size_t(tail.c0) * row_bytes;
  if (!split_encode_view(p.pieces, kTcBM, ap, Mt, g.M, g.K, &t.maps[0]) ||
      !split_encode_view(p.pieces, p.block_n, bp, Nt, g.N, g.K, &t.maps[1]))
    return UGEMM_ERR_CUDA;
  const int nkb = split_nkb(p.pieces, g.K), per = cdiv(nkb, 2);
  int tiles = 0;
  for (int s = 0; s < 2; ++s) {
    TcProblem& tp = t.probs[s];
    tp.C = part + s * mn;
    tp.M = Mt;
    tp.N = Nt;
    tp.ldc = Nt;
    tp.alpha = g.alpha;
    tp.beta = 0.f;
    tp.kb0 = s * per;
    tp.nkb = std::min(per, nkb - tp.kb0);
    tp.tiles_m = cdiv(Mt, kTcBM);
    tp.tiles_n = cdiv(Nt, p.block_n);
    tp.tile_start = tiles;
    if (p.f16) {  // the views' rows and columns keep the whole operands' scales
      tp.fmax_a = split_fmax_word(a_pieces, p.pieces, g.M, g.K) + tail.r0;
      tp.fmax_b = split_fmax_word(b_pieces, p.pieces, g.N, g.K) + tail.c0;
    }
    tiles += tp.tiles_m * tp.tiles_n;
  }
  Epilogue epi = g.epi;
  if (epi.bias) epi.bias += tail.r0;
  const ReduceJob red{part, g.C + size_t(tail.r0) * g.ldc + tail.c0, Mt, Nt, g.ldc, 2, g.beta, epi};
  SplitPlan q = p;
  q.epi = false;
  CUtensorMap dummy;
  std::memset(&dummy, 0, sizeof dummy);
  TcProblem single{};
  const int chunk =
      split_chunk_stages(p.pieces, p.chunk_kb > 0 ? p.chunk_kb : split_default_chunk_kb(g.K));
  const ugemm_status s =
      split_gemm_launch(q, dummy, dummy, single, nullptr, nullptr, nullptr, tiles, chunk,
                        std::max(1, std::min(tiles, device_sms())), dev_err, st, nullptr, &t);
  return s != UGEMM_OK ? s
                       : splitk_reduce_param_launch(&red, 1, static_cast<long long>(mn), st);
}

namespace {

// Whether L's narrower tiles or k slices are faster than one launch of whole
// 256- (or, up to 128 columns, 128-) wide tiles by the stage times, as they are
// where whole tiles leave SMs idle (1024^3: 32 tiles of 256).
bool faster_than_whole(const Gemm& g, const SplitPlan& p, const MultiLayout& L) {
  const int nkb = split_nkb(p.pieces, g.K);
  const GeoChoice whole =
      choose_geometry(p.pieces, g.M, g.N, nkb, device_sms(), p.block_n, false, 1, nkb);
  return L.us < 0.95 * (whole.us + split_pass_us((double(g.M) + g.N) * g.K));
}

// Whole tiles of g, or 0 if it does not run here at all.
int whole_tiles(const Gemm& g, const SplitPlan& p) {
  if (g.M == 0 || g.N == 0 || g.K == 0 || g.alpha == 0.f) return 0;
  const double tiles = double(cdiv(g.M, kTcBM)) * cdiv(g.N, p.block_n);
  return tiles > 4 * device_sms() ? 0 : static_cast<int>(tiles);
}

}  // namespace

bool multi_faster(const Gemm& g, const SplitPlan& p, MultiLayout* L) {
  if (whole_tiles(g, p) == 0) return false;
  *L = multi_layout(&g, 1, p);
  return faster_than_whole(g, p, *L);
}

// Where that is faster, and where the tiles are fewer than the SMs and k is deep,
// so that slices or sums of sums (choose_geometry's `longest`) cost little and are
// nearer FP64 (2048^3 in BF16x6: one wave of 128 whole tiles is 1.29e-7 from
// it, sums of a third of k each 1.16e-7).
bool multi_wanted(const Gemm& g, const SplitPlan& p, MultiLayout* L) {
  const int tiles = whole_tiles(g, p);
  if (tiles == 0) return false;
  *L = multi_layout(&g, 1, p);
  return (tiles < device_sms() && L->longest < split_nkb(p.pieces, g.K)) ||
         faster_than_whole(g, p, *L);
}

ugemm_status multi_launch(const Gemm* gs, int n, const SplitPlan& plan, const MultiLayout& L,
                          Scratch ws, int* dev_err, cudaStream_t st) {
  if (n < 1 || n > kMultiMax) return UGEMM_ERR_ARG;
  for (int i = 0; i < n; ++i)
    if (gs[i].M == 0 || gs[i].N == 0 || gs[i].K == 0 || gs[i].alpha == 0.f) return UGEMM_ERR_ARG;
  if (L.total > ws.bytes) return UGEMM_ERR_ARENA_TOO_SMALL;
  uint8_t* base = static_cast<uint8_t*>(ws.ptr);
  SplitPlan p = plan;
  p.block_n = L.block_n;
  p.epi = false;
  p.fused = L.fused;

  MultiTable t = empty_table();
  ReduceJob red[kMultiMax];
  SplitJobTable jt{};
  static_assert(2 * kMultiMax <= kSplitTableJobs, "two operands per GEMM");
  int nj = 0, split_tiles = 0;
  int nsub = 0, nred = 0, tiles = 0;
  long long red_max = 0;
  for (int i = 0; i < n; ++i) {
    const Gemm& g = gs[i];
    const GeoChoice& o = L.geo[i];
    const int nkb = split_nkb(p.pieces, g.K);
    void* ap = base + L.a_off[i];
    void* bp = base + L.b_off[i];
    long long a_sr, a_sk, b_sr, b_sk;
    split_operand_strides(g, &a_sr, &a_sk, &b_sr, &b_sk);
    int kc[2] = {1, 1};
    if (L.fused) {  // nothing to split beforehand
    } else if (p.f16) {  // the FP16x3 split needs each operand's row maxima first
      ugemm_status s = split_operand_launch(p.pieces, g.A, a_sr, a_sk, g.M, g.K, ap, st, true);
      if (s == UGEMM_OK) s = split_operand_launch(p.pieces, g.B, b_sr, b_sk, g.N, g.K, bp, st, true);
      if (s != UGEMM_OK) return s;
    } else {  // every operand in one split launch (below)
      const int kp = split_kp(g.K), tk = cdiv(kp, 64);
      jt.jobs[nj++] = SplitJob{g.A, a_sr, a_sk, static_cast<__nv_bfloat16*>(ap), g.M, g.K, kp,
                               split_tiles};
      split_tiles += cdiv(g.M, 32) * tk;
      jt.jobs[nj++] = SplitJob{g.B, b_sr, b_sk, static_cast<__nv_bfloat16*>(bp), g.N, g.K, kp,
                               split_tiles};
      split_tiles += cdiv(g.N, 32) * tk;
    }
    bool ok;
    if (L.fused) {
      TcProblem layouts{};
      ok = fused_encode_problem(g, o.swap, p.block_n, &t.maps[2 * i], &layouts);
      kc[0] = layouts.kc_a;
      kc[1] = layouts.kc_b;
    } else if (o.swap) {
      ok = split_encode_maps(p.pieces, p.block_n, bp, g.N, ap, g.M, g.K, &t.maps[2 * i],
                             &t.maps[2 * i + 1]);
    } else {
      ok = split_encode_maps(p.pieces, p.block_n, ap, g.M, bp, g.N, g.K, &t.maps[2 * i],
                             &t.maps[2 * i + 1]);
    }
    if (!ok) return UGEMM_ERR_CUDA;
    const bool sliced = o.slices > 1;
    float* part = reinterpret_cast<float*>(base + L.part_off[i]);
    for (int sidx = 0; sidx < o.slices; ++sidx) {
      TcProblem& tp = t.probs[nsub++];
      tp.C = sliced ? part + size_t(sidx) * g.M * g.N : g.C;
      tp.M = o.swap ? g.N : g.M;
      tp.N = o.swap ? g.M : g.N;
      tp.ldc = sliced ? g.N : g.ldc;
      tp.alpha = g.alpha;
      tp.beta = sliced ? 0.f : g.beta;
      tp.kb0 = sidx * o.per;
      tp.nkb = std::min(o.per, nkb - tp.kb0);
      tp.tiles_m = cdiv(tp.M, kTcBM);
      tp.tiles_n = cdiv(tp.N, p.block_n);
      tp.swap = o.swap ? 1 : 0;
      tp.sum_kb = o.sum;
      tp.map = i;
      tp.kc_a = kc[0];
      tp.kc_b = kc[1];
      tp.epi = sliced ? Epilogue{} : g.epi;
      p.epi |= tp.epi.bias != nullptr || tp.epi.act != 0;
      if (p.f16) {  // kernel operand a is op(B)^T's pieces when swapped
        unsigned* wa = split_fmax_word(ap, p.pieces, g.M, g.K);
        unsigned* wb = split_fmax_word(bp, p.pieces, g.N, g.K);
        tp.fmax_a = o.swap ? wb : wa;
        tp.fmax_b = o.swap ? wa : wb;
      }
    }
    if (sliced) {
      red[nred++] = ReduceJob{part, g.C, g.M, g.N, g.ldc, o.slices, g.beta, g.epi};
      red_max = std::max(red_max, static_cast<long long>(g.M) * g.N);
    }
  }
  int min_k = gs[0].K;  // the chunk rule follows the shallowest GEMM (the most accurate choice)
  for (int i = 1; i < n; ++i) min_k = std::min(min_k, gs[i].K);
  // longest k first; tile offsets in that order
  std::stable_sort(t.probs, t.probs + nsub,
                   [](const TcProblem& a, const TcProblem& b) { return a.nkb > b.nkb; });
  for (int j = 0; j < nsub; ++j) {
    t.probs[j].tile_start = tiles;
    tiles += t.probs[j].tiles_m * t.probs[j].tiles_n;
  }
  // the operands' bf16 / TF32 pieces: one launch for all of them (four
  // launches of one operand each left a ramp and a tail apiece)
  if (nj > 0) {
    const ugemm_status s = split_param_launch(p.pieces, jt, nj, split_tiles, st);
    if (s != UGEMM_OK) return s;
  }
  CUtensorMap dummy;
  std::memset(&dummy, 0, sizeof dummy);
  TcProblem single{};
  int chunk =
      split_chunk_stages(p.pieces, p.chunk_kb > 0 ? p.chunk_kb : split_default_chunk_kb(min_k));
  // chunks no deeper than those of the longest sum on average (its last may be
  // short); three pieces' not of a single stage for that, as twice the sums round
  // more than they save (2048 x 2048 x 928: 1.09e-7 of FP64, 9.7e-8 in twos), and
  // as they are where k is not to be cut
  if (n == 1 && !(p.pieces == 3 && L.longest >= split_nkb(3, min_k)))
    chunk = std::max(p.pieces == 3 ? std::min(chunk, 2) : 1, L.longest / cdiv(L.longest, chunk));
  const ugemm_status s =
      split_gemm_launch(p, dummy, dummy, single, nullptr, nullptr, nullptr, tiles, chunk,
                        std::max(1, std::min(tiles, device_sms())), dev_err, st, nullptr, &t);
  return s != UGEMM_OK ? s : splitk_reduce_param_launch(red, nred, red_max, st);
}

}  // namespace ugemm
