// Host-side enqueue sequences of the radix select / top-k kernels (topk.cuh), shared by the
// C ABI and the serving runtime.  Scratch comes from the context's buffers (aux0: candidate
// keys, aux1: SelectState, aux2: tile counts), which the serving runtime binds to
// slices of its arena.
#pragma once
#include <algorithm>
#include <cmath>

#include "sort_host.cuh"
#include "topk.cuh"

namespace hpcs {

// Grid of the passes over the keys: SEL_CTAS_PER_SM CTAs per SM, fewer for small inputs.
inline int select_grid(hpcs_ctx* ctx, int64_t n, int key_bytes) {
  const int64_t per_cta = int64_t(SEL_NT) * SEL_VPT * (16 / key_bytes);
  const int64_t want = (n + per_cta - 1) / per_cta;
  const int64_t cap = int64_t(ctx->sms) * SEL_CTAS_PER_SM;
  return int(want < 1 ? 1 : (want > cap ? cap : want));
}

inline int stream_capturing(cudaStream_t s, bool* capturing) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  HPCS_CUDA(cudaStreamIsCapturing(s, &cap));
  *capturing = cap != cudaStreamCaptureStatusNone;
  return HPCS_OK;
}

template <class U>
inline int64_t win_tiles(int64_t n) {
  return (n + win_tile<U>() - 1) / win_tile<U>();
}

// Launches the finishing kernel as one cluster.
template <class U, int KIND>
inline int launch_select_finish(hpcs_ctx* ctx, bool chained, const U* cand, int64_t n, int64_t rank, SelectState* st,
                                int open_top, U* out, int64_t k, cudaStream_t s) {
  auto kern = select_finish_kernel<U, KIND>;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS_MAX_CTAS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.blockDim = dim3(FIN_NT, 1, 1);
  cfg.dynamicSmemBytes = sizeof(FinishSmem);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  static int ctas_by_dev[64] = {0};
  int& ctas = ctas_by_dev[ctx->device & 63];
  if (!ctas) {
    HPCS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(FinishSmem))));
    HPCS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cfg.gridDim = dim3(CS_MAX_CTAS, 1, 1);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) cudaGetLastError();
    ctas = clusters > 0 ? CS_MAX_CTAS : 8;
  }
  attr[0].val.clusterDim.x = unsigned(ctas);
  cfg.gridDim = dim3(unsigned(ctas), 1, 1);
  cfg.numAttrs = chained ? 2 : 1;
  HPCS_CUDA(cudaLaunchKernelEx(&cfg, kern, cand, n, rank, st, open_top, out, k));
  return HPCS_OK;
}

// The select of rank `rank` among n keys: sample, window read (with a copy of the keys and the tiles'
// counts if wanted), the levels.  rlo, rhi: sample ranks of the window's ends; open_top: rank n - k of
// the k largest, which go to out[0..k) (unsorted).  Up to FIN_MAX_CANDIDATES expected candidates the
// levels (and the gather) run in one cluster; more take a launch per level over all SMs.
template <class U, int KIND>
inline int enqueue_window_select(hpcs_ctx* ctx, const U* d, int64_t n, int64_t rank, int64_t rlo, int64_t rhi,
                                 bool open_top, U* cand, SelectState* st, U* copy, WinTile* tiles, U* out, int64_t k,
                                 cudaStream_t s) {
  constexpr int BITS = int(sizeof(U) * 8);
  constexpr int S = select_sample_size<U>();
  bool capturing = false;
  const int rc = stream_capturing(s, &capturing);
  if (rc != HPCS_OK) return rc;
  const bool chained = !capturing;
  const int grid = select_grid(ctx, n, int(sizeof(U)));
  // the sample lies in the candidate buffer (at least 4 S keys) until the window read
  select_gather_kernel<U, KIND><<<S / 512, 512, 0, s>>>(d, n, cand, st);
  HPCS_CUDA(cudaGetLastError());
  if (n >= int64_t(4) * S)
    HPCS_CUDA(launch_chained(chained, select_sample_kernel<U>, 1, SAMPLE_NT, 0, s, static_cast<const U*>(cand), rlo, rhi, st));
  const int ctas = int(win_tiles<U>(n));
  // the k largest with at most one candidate per warp expected need no CTA-wide slots
  const bool sparse = open_top && n >= int64_t(4) * S && (S - rlo) * (win_tile<U>() / (WIN_NT / 32)) <= S;
  const int steps = sparse && ctas >= 16 * ctx->sms ? 4 : 1;  // (the barrier's share; small inputs spread out)
  HPCS_CUDA(sparse ? launch_chained(chained, select_window_kernel<U, KIND, false, false>, (ctas + steps - 1) / steps, WIN_NT, 0, s, d, n, cand, st, copy, tiles, steps)
            : copy ? launch_chained(chained, select_window_kernel<U, KIND, true, true>, ctas, WIN_NT, 0, s, d, n, cand, st, copy, tiles, 1)
                   : launch_chained(chained, select_window_kernel<U, KIND, false, true>, ctas, WIN_NT, 0, s, d, n, cand, st, copy, tiles, 1));
  const U* c = cand;
  const int open = open_top ? 1 : 0;
  const int64_t width = (rhi >= S ? S : rhi + 1) - (rlo < 0 ? 0 : rlo);
  const int64_t expect = n < int64_t(4) * S || width >= S ? n : int64_t(double(width) / S * double(n));
  const bool finish = expect <= FIN_MAX_CANDIDATES;
  // More candidates than the sample explains (its count of a window of `width` samples is off by one part
  // in sqrt(width)): level 0 deals with them on all SMs.  But not a few that the cluster reads as fast: with
  // both ends given their common digits need no level (select among 1 Mi f32 keys, half of them zero: 524 Ki
  // candidates, 82 us in the cluster, 88 on all SMs), with the top open every level reads them (the 2^18
  // largest of 1 Mi u32 keys, half of them the largest value: 112 and 92).
  const int64_t few = open_top ? FIN_MAX_CANDIDATES * 3 / 4 : 2 * FIN_MAX_CANDIDATES;
  const int64_t limit = std::max(few, int64_t(double(expect) * (1.0 + 6.0 / std::sqrt(double(width)))) + 32768);
  for (int shift = BITS - 8; shift >= 0; shift -= 8) {
    if (!finish)
      HPCS_CUDA(launch_chained(chained, select_level_kernel<U, KIND, false>, grid, SEL_NT, 0, s, d, n, c, rank, st, shift, open, limit));
    else if (shift == BITS - 8)
      HPCS_CUDA(launch_chained(chained, select_level_kernel<U, KIND, true>, grid, SEL_NT, 0, s, d, n, c, rank, st, shift, open, limit));
    if (shift == BITS - 8)
      HPCS_CUDA(launch_chained(chained, select_compact_kernel<U, KIND>, grid, SEL_NT, 0, s, d, n, cand, st, out, k));
  }
  if (finish) return launch_select_finish<U, KIND>(ctx, chained, c, n, rank, st, open, out, k, s);
  if (out) {
    const int cgrid = select_grid(ctx, 2 * expect, int(sizeof(U)));
    HPCS_CUDA(launch_chained(chained, topk_gather_kernel<U, KIND>, cgrid, SEL_NT, 0, s, c, k, st, out));
  }
  return HPCS_OK;
}

// Radix select of the key of 0-based rank `rank` among n keys at device pointer d.  Leaves the
// SelectState in ctx->aux1 (prefix = the ordered bits of the selected key, less/eq counts), the
// candidates in ctx->aux0 and the tiles' counts in ctx->aux2 for the partition.  With `copy` (n keys),
// d's keys are copied there on the way.
template <class U, int KIND>
inline int enqueue_select(hpcs_ctx* ctx, const U* d, int64_t n, int64_t rank, cudaStream_t s, SelectState** out,
                          U* copy = nullptr) {
  constexpr int S = select_sample_size<U>();
  int rc;
  if ((rc = ensure(ctx, ctx->aux1, sizeof(SelectState))) != HPCS_OK) return rc;
  if ((rc = ensure(ctx, ctx->aux0, size_t(n) * sizeof(U))) != HPCS_OK) return rc;
  const int64_t tiles = win_tiles<U>(n);
  if ((rc = ensure(ctx, ctx->aux2, size_t(tiles) * (sizeof(uint2) + sizeof(WinTile)))) != HPCS_OK) return rc;
  SelectState* st = static_cast<SelectState*>(ctx->aux1.ptr);
  WinTile* wt = reinterpret_cast<WinTile*>(static_cast<uint2*>(ctx->aux2.ptr) + tiles);
  // the sample rank of the selected key has standard deviation sqrt(S p (1 - p)), p = rank / n;
  // the window reaches 6 of them plus 9 samples to each side
  const double p = n > 0 ? double(rank) / double(n) : 0.0;
  const int64_t m = int64_t(6.0 * std::sqrt(double(S) * p * (1.0 - p)) + 9.0) + 1;
  const int64_t rs = rank * S / n;  // expected sample rank of the selected key
  KernelTimer kt(ctx, s, HPCS_K_TOPK);
  rc = enqueue_window_select<U, KIND>(ctx, d, n, rank, rs - m, rs + m, false, static_cast<U*>(ctx->aux0.ptr), st, copy, wt,
                                      nullptr, 0, s);
  *out = st;
  return rc;
}

// Stable three-way partition of d[0..n) around the key that enqueue_select selected among the same
// keys, into out (which the select read, if it copied them to d).
template <class U, int KIND>
inline int enqueue_partition(hpcs_ctx* ctx, const U* d, int64_t n, SelectState* st, U* out, cudaStream_t s) {
  const int64_t tiles = win_tiles<U>(n);
  uint2* counts = static_cast<uint2*>(ctx->aux2.ptr);
  const WinTile* wt = reinterpret_cast<const WinTile*>(counts + tiles);
  bool capturing = false;
  const int rc = stream_capturing(s, &capturing);
  if (rc != HPCS_OK) return rc;
  const bool chained = !capturing;
  const SelectState* cst = st;
  KernelTimer kt(ctx, s, HPCS_K_TOPK);
  HPCS_CUDA(launch_chained(chained, partition_count_kernel<U, KIND>, int((tiles + 7) / 8), 256, 0, s, d, n,
                           static_cast<const U*>(ctx->aux0.ptr), cst, wt, tiles, counts));
  HPCS_CUDA(launch_chained(chained, partition_scan_kernel, 1, 1024, 0, s, counts, tiles));
  HPCS_CUDA(launch_chained(chained, partition_scatter_kernel<U, KIND>, int(tiles), PART_NT, 0, s, d, n, cst,
                           static_cast<const uint2*>(counts), out));
  return HPCS_OK;
}

// The k largest of in[0..n) into out[0..k), ascending (device pointers).  One read of the keys
// in the common case: a sampled threshold, one filtering read, the radix select over the
// candidates (topk.cuh); the two-read select over all keys when the candidates fall short.
template <class T, class U, int KIND>
inline int topk_largest_enqueue(hpcs_ctx* ctx, const U* d, int64_t n, int64_t k, U* out, cudaStream_t s) {
  constexpr int S = select_sample_size<U>();
  int rc;
  if ((rc = ensure(ctx, ctx->aux1, sizeof(SelectState))) != HPCS_OK) return rc;
  if ((rc = ensure(ctx, ctx->aux0, size_t(n) * sizeof(U))) != HPCS_OK) return rc;
  SelectState* st = static_cast<SelectState*>(ctx->aux1.ptr);
  U* cand = static_cast<U*>(ctx->aux0.ptr);
  // sampled keys expected at or above the threshold: enough that fewer than k candidates
  // (k keys sampled at rate S/n, Poisson) is many standard deviations away
  const double ks = double(k) * S / double(n);
  const int64_t m = int64_t(1.5 * ks + 6.0 * std::sqrt(ks) + 8.0) + 1;
  const bool one_cta = k <= topk_small_sort_max<U>();
  {
    KernelTimer kt(ctx, s, HPCS_K_TOPK);
    if ((rc = enqueue_window_select<U, KIND>(ctx, d, n, n - k, S - m, S, true, cand, st, nullptr, nullptr, out, k, s)) != HPCS_OK)
      return rc;
    bool capturing = false;
    if ((rc = stream_capturing(s, &capturing)) != HPCS_OK) return rc;
    if (one_cta)
      HPCS_CUDA(launch_chained(!capturing, topk_small_sort_kernel<U, KIND>, 1, TOPK_SMALL_SORT_NT, 0, s, out, int(k)));
  }
  if (one_cta) return HPCS_OK;
  return enqueue_sort<U, KIND, NoValue>(ctx, out, nullptr, k, s);
}

}  // namespace hpcs
