// Host-side launch logic for the LSD sort kernels: context state, scratch buffers,
// per-dtype kernel configuration and the enqueue sequence K1 -> K3 x P -> finalize.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/hpcs_gpu.h"
#include "chunk_pass.cuh"
#include "cluster_sort.cuh"
#include "lookback_pass.cuh"
#include "radix_kernels.cuh"

namespace hpcs {

// ---- thread-local error text ---------------------------------------------------------
void set_error(const std::string& msg);
int fail(int status, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);

#define HPCS_CUDA(call)                                  \
  do {                                                   \
    cudaError_t e_ = (call);                             \
    if (e_ != cudaSuccess) return ::hpcs::cuda_fail(e_, #call); \
  } while (0)

// Grow-only device buffer owned by a context.  A borrowed buffer is a slice of memory that
// someone else owns (the serving arena): it is never grown or freed by the context.
struct DevBuf {
  void* ptr = nullptr;
  size_t bytes = 0;
  bool borrowed = false;
};

}  // namespace hpcs

namespace hpcs {
struct HostStager;
}

struct hpcs_ctx {
  int device = 0;
  int sms = 0;
  int rank_mode = 1;  // hpcs::RankMode actually used
  hpcs_config cfg{};
  cudaStream_t stream = nullptr;
  cudaStream_t last_stream = nullptr;
  cudaEvent_t order_event = nullptr;
  size_t held_bytes = 0;
  // tile trace (debug)
  uint64_t* trace = nullptr;
  int trace_pass = -1;
  int trace_capacity = 0;
  // per-kernel timing
  bool profile = false;
  struct Timed {
    int cls;
    cudaEvent_t a, b;
  };
  std::vector<Timed> timed;
  std::vector<cudaEvent_t> event_pool;
  // scratch
  hpcs::DevBuf keys_a, keys_b, vals_a, vals_b, status0, status1, plan, counts, err_accum;
  hpcs::DevBuf aux0, aux1, aux2;
  // pinned ring and copy threads for host arrays in pageable memory (host_copy.cuh)
  hpcs::HostStager* stager = nullptr;
  // batched segmented sort: variant per (key width, length class), and the helper streams
  // and events that run the launches of different variants concurrently
  hpcs_seg_tuning seg_tuning{};
  bool seg_tuning_set = false;  // by the caller: followed as it is
  static constexpr int SEG_BRANCHES = 4;
  cudaStream_t seg_streams[SEG_BRANCHES] = {};
  cudaEvent_t seg_fork = nullptr;
  cudaEvent_t seg_join[SEG_BRANCHES] = {};
  // the grid-level path of the batched sort runs on its own branch
  cudaStream_t seg_grid_stream = nullptr;
  cudaEvent_t seg_grid_fork = nullptr, seg_grid_join = nullptr;
};

namespace hpcs {

int ensure(hpcs_ctx* ctx, DevBuf& b, size_t bytes);

// Brackets one kernel launch with an event pair when the context profiles.
struct KernelTimer {
  hpcs_ctx* ctx;
  cudaStream_t s;
  int cls;
  cudaEvent_t a = nullptr, b = nullptr;
  KernelTimer(hpcs_ctx* c, cudaStream_t st, int k);
  ~KernelTimer();
};
// Orders work on `s` after all earlier work of the context (scratch is shared).
int enter_stream(hpcs_ctx* ctx, cudaStream_t s);
uint32_t* device_error_word(hpcs_ctx* ctx);

// Look-back tile shapes: threads, keys per thread of the large tile, keys per thread whose shared
// accesses are in flight together.  The large tile fills the two tile buffers (a tile costs ~1600
// clocks of barriers and latency whatever its size: u32 keys 2^28, us per pass: 40 keys 592, 32 keys
// 650, 24 keys 703, 16 keys 953; 42 no better than 40).  The peer-mask ranking's 32 KiB of lane masks
// leave less room.  The 32-bit keys-only shape can be overridden at build time.
#ifndef HPCS_K32_KPT
#define HPCS_K32_KPT 40
#endif
template <class U, class V, int MODE>
struct SortConfig;
template <>
struct SortConfig<uint32_t, NoValue, RANK_ORDERED_ATOMIC> {
  static constexpr int NT = 512, KPT = HPCS_K32_KPT, BATCH = 8;
};
template <>
struct SortConfig<uint64_t, NoValue, RANK_ORDERED_ATOMIC> {
  static constexpr int NT = 512, KPT = 24, BATCH = 4;
};
template <>
struct SortConfig<uint32_t, uint32_t, RANK_ORDERED_ATOMIC> {
  static constexpr int NT = 512, KPT = 24, BATCH = 8;
};
template <>
struct SortConfig<uint64_t, uint32_t, RANK_ORDERED_ATOMIC> {
  static constexpr int NT = 512, KPT = 16, BATCH = 8;
};
template <>
struct SortConfig<uint32_t, NoValue, RANK_PEER_MASK> {
  static constexpr int NT = 512, KPT = 32, BATCH = 8;
};
template <>
struct SortConfig<uint64_t, NoValue, RANK_PEER_MASK> {
  static constexpr int NT = 512, KPT = 16, BATCH = 4;
};
template <>
struct SortConfig<uint32_t, uint32_t, RANK_PEER_MASK> {
  static constexpr int NT = 512, KPT = 16, BATCH = 8;
};
template <>
struct SortConfig<uint64_t, uint32_t, RANK_PEER_MASK> {
  static constexpr int NT = 512, KPT = 12, BATCH = 4;
};
// Keys per thread of the tile a sort of n keys takes: 8 while one such tile per SM holds the keys, 16
// up to two tiles per SM, then the large tile.  Smaller tiles put more SMs to work and their passes
// are shorter chains (u32 pass, us, 8 / 16 / 40 keys: 300 Ki keys 12.8 / 12.8 / 20.9, 1 Mi 16.7 / 15.0
// / 21.0, 3 M 27.1 / 20.8 / 21.2, 10 M 68 / 43.7 / 35.6).  The peer-mask ranking has one tile.
template <class U, class V, int MODE>
inline int lookback_kpt(int64_t n, int sms) {
  using C = SortConfig<U, V, MODE>;
  if (MODE == RANK_PEER_MASK) return C::KPT;
  if (n <= int64_t(sms) * C::NT * 8) return 8;
  return n <= int64_t(2) * sms * C::NT * 16 ? 16 : C::KPT;
}

// Chunked-pass tile shapes (threads x keys per thread).  Every shape keeps its two stage
// buffers within 128 KiB, which leaves room for 148 ranges x 512 bytes of next-digit
// counters within the 227 KiB of shared memory a CTA may use.
#ifndef HPCS_C32_NT
#define HPCS_C32_NT 512
#endif
#ifndef HPCS_C32_KPT
#define HPCS_C32_KPT 32
#endif
#ifndef HPCS_C64_KPT
#define HPCS_C64_KPT 16
#endif
#ifndef HPCS_CP32_KPT
#define HPCS_CP32_KPT 16
#endif
#ifndef HPCS_CP64_KPT
#define HPCS_CP64_KPT 10
#endif
template <class U, class V, int MODE>
struct ChunkConfig;
template <>
struct ChunkConfig<uint32_t, NoValue, RANK_ORDERED_ATOMIC> {
  static constexpr int NT = HPCS_C32_NT, KPT = HPCS_C32_KPT;
};
template <>
struct ChunkConfig<uint32_t, NoValue, RANK_PEER_MASK> {  // + lane masks: fewer warps
  static constexpr int NT = 512, KPT = 20;
};
template <>
struct ChunkConfig<uint64_t, NoValue, RANK_ORDERED_ATOMIC> {
  static constexpr int NT = 512, KPT = HPCS_C64_KPT;
};
template <>
struct ChunkConfig<uint32_t, uint32_t, RANK_ORDERED_ATOMIC> {
  static constexpr int NT = 512, KPT = HPCS_CP32_KPT;
};
template <>
struct ChunkConfig<uint64_t, uint32_t, RANK_ORDERED_ATOMIC> {
  static constexpr int NT = 512, KPT = HPCS_CP64_KPT;
};
// peer-mask ranking: 32 KiB of lane masks on top, 48 KiB stages
template <>
struct ChunkConfig<uint64_t, NoValue, RANK_PEER_MASK> {
  static constexpr int NT = 512, KPT = 12;
};
template <>
struct ChunkConfig<uint32_t, uint32_t, RANK_PEER_MASK> {
  static constexpr int NT = 512, KPT = 12;
};
template <>
struct ChunkConfig<uint64_t, uint32_t, RANK_PEER_MASK> {
  static constexpr int NT = 512, KPT = 8;
};
constexpr size_t MAX_DYN_SMEM = 232448;  // 227 KiB per CTA on sm_100

template <class U, class V, int MODE>
struct ChunkShape {
  using C = ChunkConfig<U, V, MODE>;
  using L = ChunkSmem<U, V, C::NT, C::KPT, MODE>;
  static constexpr int TILE = L::TILE;
  static constexpr int MAX_RANGES = 2 * int((MAX_DYN_SMEM - L::BASE_BYTES) / (RADIX * 4));
};

// Launches kernel k; chained: as a programmatic dependent of the kernel before it on the stream (k
// calls chain_wait before it touches memory).
template <class... P, class... A>
cudaError_t launch_chained(bool chained, void (*k)(P...), int grid, int block, size_t smem, cudaStream_t s, A... a) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(grid), 1, 1);
  cfg.blockDim = dim3(unsigned(block), 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, a...);
}

constexpr int HIST_NT = 1024;

// Launches K1 (one CTA per SM, 128 KiB of lane-private counters).
template <class U, int KIND>
int launch_histogram(hpcs_ctx* ctx, const U* keys, int64_t n, uint32_t* hist_out, const SortArgs& args,
                     int make_plan, cudaStream_t s);

template <class U, int KIND>
int launch_histogram(hpcs_ctx* ctx, const U* keys, int64_t n, uint32_t* hist_out, const SortArgs& args,
                     int make_plan, cudaStream_t s) {
  auto k = hist_all_digits_kernel<U, KIND, HIST_NT>;
  static int attr_set[64] = {0};
  if (!attr_set[ctx->device & 63]) {
    HPCS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(HistSmem<U>::BYTES)));
    attr_set[ctx->device & 63] = 1;
  }
  const int64_t vec = n * int64_t(sizeof(U)) / 16;
  const int64_t want = (vec + HIST_NT * 4 - 1) / (HIST_NT * 4);
  int grid = int(want < 1 ? 1 : (want > ctx->sms ? ctx->sms : want));
  if (args.chunk_hist) grid = args.chunks;  // CTA j counts key range j
  k<<<grid, HIST_NT, HistSmem<U>::BYTES, s>>>(keys, n, hist_out, args, make_plan);
  HPCS_CUDA(cudaGetLastError());
  return HPCS_OK;
}

// CTAs of a look-back pass: a persistent grid of one CTA per SM, one of them the scanner, at most
// one per tile besides it; a single tile needs no scanner.
inline int lookback_grid(int num_tiles, int sms) {
  const int want = num_tiles > 1 ? num_tiles + 1 : 1;
  return want < sms ? want : (sms > 1 ? sms : 2);
}

// Look-back launches for every digit pass, with tiles of KPT keys per thread.
template <class U, int KIND, class V, int MODE, int KPT>
int launch_lookback_tiles(hpcs_ctx* ctx, SortArgs args, bool chained, cudaStream_t s) {
  using C = SortConfig<U, V, MODE>;
  using L = LookbackSmem<U, V, C::NT, KPT, MODE>;
  static_assert(L::BYTES <= MAX_DYN_SMEM, "two tile buffers fit");
  constexpr int P = int(sizeof(U));
  auto k = lookback_pass_kernel<U, KIND, V, C::NT, KPT, MODE, C::BATCH>;
  static int attr_set[64] = {0};
  if (!attr_set[ctx->device & 63]) {
    HPCS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(L::BYTES)));
    attr_set[ctx->device & 63] = 1;
  }
  const int grid = lookback_grid(args.num_tiles, ctx->sms);
  for (int p = 0; p < P; p++) {
    args.pass = p;
    KernelTimer kt(ctx, s, HPCS_K_LOOKBACK);
    HPCS_CUDA(launch_chained(chained, k, grid, C::NT, L::BYTES, s, args));
  }
  return HPCS_OK;
}

template <class U, int KIND, class V, int MODE>
int launch_lookback_passes(hpcs_ctx* ctx, const SortArgs& args, int kpt, bool chained, cudaStream_t s) {
  constexpr int LARGE = SortConfig<U, V, MODE>::KPT;
  constexpr bool ONE = MODE == RANK_PEER_MASK;
  switch (kpt) {
    case 8: return launch_lookback_tiles<U, KIND, V, MODE, ONE ? LARGE : 8>(ctx, args, chained, s);
    case 16: return launch_lookback_tiles<U, KIND, V, MODE, ONE ? LARGE : 16>(ctx, args, chained, s);
    default: return launch_lookback_tiles<U, KIND, V, MODE, LARGE>(ctx, args, chained, s);
  }
}

// Chunked digit passes: one CTA per key range, one launch per digit.
template <class U, int KIND, class V, int MODE>
int launch_chunk_passes(hpcs_ctx* ctx, SortArgs args, cudaStream_t s) {
  using C = ChunkConfig<U, V, MODE>;
  using L = ChunkSmem<U, V, C::NT, C::KPT, MODE>;
  constexpr int P = int(sizeof(U));
  auto k = chunk_pass_kernel<U, KIND, V, C::NT, C::KPT, MODE>;
  static int attr_set[64] = {0};
  if (!attr_set[ctx->device & 63]) {
    HPCS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(MAX_DYN_SMEM)));
    attr_set[ctx->device & 63] = 1;
  }
  const size_t bytes = L::bytes(args.chunks);
  for (int p = 0; p < P; p++) {
    args.pass = p;
    KernelTimer kt(ctx, s, HPCS_K_ONESWEEP);
    k<<<args.chunks, C::NT, bytes, s>>>(args);
    HPCS_CUDA(cudaGetLastError());
  }
  return HPCS_OK;
}

// Key ranges of the chunked passes: as many as there are SMs (capped by the counters'
// shared memory), each a whole number of tiles.
struct ChunkGeometry {
  int chunks;
  uint32_t chunk_keys;
  uint32_t magic;
};
inline ChunkGeometry chunk_geometry(int64_t n, int tile, int max_ranges) {
  const int64_t tiles = (n + tile - 1) / tile;
  const int64_t per = (tiles + max_ranges - 1) / max_ranges;  // tiles per range
  ChunkGeometry g;
  g.chunks = int((tiles + per - 1) / per);
  g.chunk_keys = uint32_t(per * tile);
  g.magic = uint32_t(((uint64_t(1) << 32) + g.chunk_keys - 1) / g.chunk_keys);
  return g;
}

// Slice shapes of the one-launch small sort, in keys per thread.  One slice up to 8192 keys, with the
// smallest of 4, 8 and 16 that holds them (u32 keys, us per call: 1000 keys 6.3 / 8.3 / 10.4, 4096 keys
// 14.5 (two slices) / 8.3 / 12.4; 16384 keys in one slice of 32 per thread 22.7, in four of 8 18.6);
// beyond, the smallest of 8, 16 and (32-bit keys alone) 32 of which 16 slices hold them: fewer keys per
// CTA make shorter passes (65536 keys 20.6 / 24.7 / 39.0, 131072 keys - / 26.8 / 39.3, 262144 keys 41.1
// with 32, 52 on the look-back passes).  The peer-mask ranking has one shape.
constexpr int64_t CS_SOLO_KEYS = 8192;

// Launches the one-launch small sort with KPT keys per thread if n fits (else *done stays false).  The
// cluster is the next power of two of CTAs; more than 8 where the device schedules such clusters.
template <class U, int KIND, class V, int MODE, int KPT>
int launch_cluster_sort(hpcs_ctx* ctx, U* keys, uint32_t* vals, int64_t n, cudaStream_t s, bool* done) {
  using L = ClusterSmem<U, V, KPT, MODE>;
  static_assert(L::BYTES <= MAX_DYN_SMEM, "a slice fits");
  auto k = cluster_sort_kernel<U, KIND, V, KPT, MODE>;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.blockDim = dim3(CS_NT, 1, 1);
  cfg.dynamicSmemBytes = L::BYTES;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  static int max_ctas_by_dev[64] = {0};
  int& max_ctas = max_ctas_by_dev[ctx->device & 63];
  if (!max_ctas) {
    HPCS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(L::BYTES)));
    HPCS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    attr.val.clusterDim.x = CS_MAX_CTAS;
    cfg.gridDim = dim3(CS_MAX_CTAS, 1, 1);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess) cudaGetLastError();
    max_ctas = clusters > 0 ? CS_MAX_CTAS : 8;
  }
  int ctas = 1;
  while (int64_t(ctas) * L::SLICE < n) ctas *= 2;
  if (ctas > max_ctas) return HPCS_OK;
  attr.val.clusterDim.x = unsigned(ctas);
  cfg.gridDim = dim3(unsigned(ctas), 1, 1);
  KernelTimer kt(ctx, s, HPCS_K_LOOKBACK);
  HPCS_CUDA(cudaLaunchKernelEx(&cfg, k, keys, vals, uint32_t(n), int(ctx->cfg.skip_trivial_passes), device_error_word(ctx)));
  *done = true;
  return HPCS_OK;
}

// Keys per thread of the one-launch small sort of n keys, 0 where n takes the large-array kernels.
template <class U, class V, int MODE>
inline int cluster_kpt(int64_t n) {
  constexpr bool ONE = MODE == RANK_PEER_MASK;
  constexpr int LARGEST = !ONE && sizeof(U) == 4 && std::is_same<V, NoValue>::value ? 32 : 16;
  const int64_t per = n <= CS_SOLO_KEYS ? n : (n + CS_MAX_CTAS - 1) / CS_MAX_CTAS;  // keys a slice must hold
  if (per > CS_NT * LARGEST) return 0;
  if (ONE) return 16;
  if (per <= CS_NT * 4 && n <= CS_SOLO_KEYS) return 4;
  return per <= CS_NT * 8 ? 8 : per <= CS_NT * 16 ? 16 : LARGEST;
}

// A small sort in one cluster launch if n fits (else *done stays false).
template <class U, int KIND, class V, int MODE>
int enqueue_cluster_sort(hpcs_ctx* ctx, U* keys, uint32_t* vals, int64_t n, cudaStream_t s, bool* done) {
  constexpr bool ONE = MODE == RANK_PEER_MASK;
  constexpr int LARGEST = !ONE && sizeof(U) == 4 && std::is_same<V, NoValue>::value ? 32 : 16;
  switch (cluster_kpt<U, V, MODE>(n)) {
    case 0: return HPCS_OK;
    case 4: return launch_cluster_sort<U, KIND, V, MODE, ONE ? 16 : 4>(ctx, keys, vals, n, s, done);
    case 8: return launch_cluster_sort<U, KIND, V, MODE, ONE ? 16 : 8>(ctx, keys, vals, n, s, done);
    case 16: return launch_cluster_sort<U, KIND, V, MODE, 16>(ctx, keys, vals, n, s, done);
    default: return launch_cluster_sort<U, KIND, V, MODE, LARGEST>(ctx, keys, vals, n, s, done);
  }
}

// Whether the sort's rows (and its plan) fit the context's budget, or the slices it was lent.
inline bool rows_fit(const hpcs_ctx* ctx, size_t row_bytes0, size_t row_bytes1) {
  const DevBuf* bufs[3] = {&ctx->status0, &ctx->status1, &ctx->plan};
  const size_t want[3] = {row_bytes0, row_bytes1, sizeof(SortPlan)};
  size_t held = ctx->held_bytes;
  for (int i = 0; i < 3; i++) {
    if (bufs[i]->bytes >= want[i]) continue;
    if (bufs[i]->borrowed) return false;
    held += std::max(want[i], size_t(256)) - bufs[i]->bytes;
  }
  return ctx->cfg.pool_bytes <= 0 || held <= size_t(ctx->cfg.pool_bytes);
}

// Enqueue a full LSD sort of n keys (and optional 4-byte items) in device memory.
// keys/vals are sorted in place (with scratch B owned by the context).
template <class U, int KIND, class V>
int enqueue_sort(hpcs_ctx* ctx, U* keys, uint32_t* vals, int64_t n, cudaStream_t s) {
  using CA = SortConfig<U, V, RANK_ORDERED_ATOMIC>;
  using CP = SortConfig<U, V, RANK_PEER_MASK>;
  constexpr bool PAIRS = !std::is_same<V, NoValue>::value;
  if (n <= 1) return HPCS_OK;
  if (n > MAX_KEYS_PER_SORT) return fail(HPCS_ERR_RANGE, "n exceeds HPCS_MAX_KEYS");
  if (ctx->cfg.pass_scheme == HPCS_PASSES_LOOKBACK && n > MAX_KEYS_LOOKBACK)
    return fail(HPCS_ERR_RANGE, "look-back passes take at most 2^30 - 1 keys when forced");
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  HPCS_CUDA(cudaStreamIsCapturing(s, &cap));
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  const bool ordered = ctx->rank_mode == RANK_ORDERED_ATOMIC;
  int rc;
  // small sorts: one cluster launch (not when a pass scheme is forced)
  if (ctx->cfg.pass_scheme == HPCS_PASSES_AUTO) {
    bool done = false;
    rc = ordered ? enqueue_cluster_sort<U, KIND, V, RANK_ORDERED_ATOMIC>(ctx, keys, vals, n, s, &done)
                 : enqueue_cluster_sort<U, KIND, V, RANK_PEER_MASK>(ctx, keys, vals, n, s, &done);
    if (rc != HPCS_OK || done) return rc;
  }
  if ((rc = ensure(ctx, ctx->keys_b, size_t(n) * sizeof(U))) != HPCS_OK) return rc;
  if (PAIRS && (rc = ensure(ctx, ctx->vals_b, size_t(n) * 4)) != HPCS_OK) return rc;

  // 16-byte alignment is required by the bulk copies; unaligned callers go through A'.
  U* a = keys;
  uint32_t* va = vals;
  const bool keys_unaligned = (reinterpret_cast<uintptr_t>(keys) & 15) != 0;
  const bool vals_unaligned = PAIRS && (reinterpret_cast<uintptr_t>(vals) & 15) != 0;
  if (keys_unaligned) {
    if ((rc = ensure(ctx, ctx->keys_a, size_t(n) * sizeof(U))) != HPCS_OK) return rc;
    a = static_cast<U*>(ctx->keys_a.ptr);
    HPCS_CUDA(cudaMemcpyAsync(a, keys, size_t(n) * sizeof(U), cudaMemcpyDeviceToDevice, s));
  }
  if (vals_unaligned) {
    if ((rc = ensure(ctx, ctx->vals_a, size_t(n) * 4)) != HPCS_OK) return rc;
    va = static_cast<uint32_t*>(ctx->vals_a.ptr);
    HPCS_CUDA(cudaMemcpyAsync(va, vals, size_t(n) * 4, cudaMemcpyDeviceToDevice, s));
  }
  constexpr int P = int(sizeof(U));
  // The passes: look-back with the tile for n, look-back with the large tile, chunked (unless a scheme is
  // forced); the first whose rows fit.  The later ones are slower and take less scratch: 2^28 u32 keys 26 MiB
  // of look-back rows, 1 MiB of count tables; 1 Mi keys 128 Ki + 128 Ki of rows, with the large tile 52 + 52.
  const int tile_kpt[2] = {ordered ? lookback_kpt<U, V, RANK_ORDERED_ATOMIC>(n, ctx->sms) : CP::KPT, ordered ? CA::KPT : CP::KPT};
  ChunkGeometry geo{0, 0, 0};
  int64_t num_tiles = 0;
  int kpt = 0;  // 0: chunked passes
  const int first = ctx->cfg.pass_scheme == HPCS_PASSES_CHUNKED ? 2 : 0, last = ctx->cfg.pass_scheme == HPCS_PASSES_LOOKBACK ? 1 : 2;
  for (int option = first; option <= last; option++) {
    kpt = option < 2 ? tile_kpt[option] : 0;
    size_t rows[2];
    if (kpt) {
      const int64_t unit = int64_t(ordered ? CA::NT : CP::NT) * kpt;
      num_tiles = (n + unit - 1) / unit;
      rows[0] = rows[1] = size_t(num_tiles) * RADIX * 4;
    } else {
      using SA = ChunkShape<U, V, RANK_ORDERED_ATOMIC>;
      using SP = ChunkShape<U, V, RANK_PEER_MASK>;
      const int cap = ordered ? SA::MAX_RANGES : SP::MAX_RANGES;
      geo = chunk_geometry(n, ordered ? SA::TILE : SP::TILE, ctx->sms < cap ? ctx->sms : cap);
      num_tiles = 0;
      rows[0] = size_t(geo.chunks) * (P + 3) * RADIX * 4;
      rows[1] = 0;
    }
    if (option < last && !rows_fit(ctx, rows[0], rows[1])) continue;
    rc = ensure(ctx, ctx->status0, rows[0]);
    if (rc == HPCS_OK && rows[1]) rc = ensure(ctx, ctx->status1, rows[1]);
    if (rc == HPCS_OK) rc = ensure(ctx, ctx->plan, sizeof(SortPlan));
    if (rc != HPCS_ERR_OOM) break;  // (the device itself may be full)
  }
  if (rc != HPCS_OK) return rc;
  const bool lookback = kpt != 0;
  // the look-back launches are chained: each pass's CTAs start as the last pass's finish (u32 sorts,
  // us, plain / chained launches: 150 Ki keys 69 / 51, 1 Mi 75 / 61, 10 M 181 / 167)
  const bool chained = lookback && !capturing;

  SortArgs args{};
  args.keys_a = a;
  args.keys_b = ctx->keys_b.ptr;
  args.vals_a = va;
  args.vals_b = PAIRS ? ctx->vals_b.ptr : nullptr;
  args.n = n;
  args.plan = static_cast<SortPlan*>(ctx->plan.ptr);
  args.status[0] = static_cast<uint32_t*>(ctx->status0.ptr);
  args.status[1] = static_cast<uint32_t*>(ctx->status1.ptr);
  args.num_tiles = int(num_tiles);
  args.skip_trivial = ctx->cfg.skip_trivial_passes;
  args.poison_tile = ctx->cfg.poison_tile;
  args.spin_limit_ns = uint64_t(ctx->cfg.spin_limit_ns);
  args.trace = ctx->trace;
  args.trace_pass = ctx->trace_pass;
  args.trace_capacity = ctx->trace_capacity;
  if (!lookback) {
    // status0 holds [chunks][P][256] per-range input counts, then [3][chunks][256] tables
    args.chunk_hist = static_cast<uint32_t*>(ctx->status0.ptr);
    args.ctab = args.chunk_hist + size_t(geo.chunks) * P * RADIX;
    args.chunks = geo.chunks;
    args.chunk_keys = geo.chunk_keys;
    args.chunk_magic = geo.magic;
  }
  HPCS_CUDA(cudaMemsetAsync(args.plan, 0, sizeof(SortPlan), s));

  // K1: fused histogram + plan
  {
    KernelTimer kt(ctx, s, HPCS_K_HISTOGRAM);
    if ((rc = launch_histogram<U, KIND>(ctx, a, n, &args.plan->hist[0][0], args, 1, s)) != HPCS_OK) return rc;
  }
  // K3: one launch per digit
  if (!lookback)
    rc = ordered ? launch_chunk_passes<U, KIND, V, RANK_ORDERED_ATOMIC>(ctx, args, s)
                 : launch_chunk_passes<U, KIND, V, RANK_PEER_MASK>(ctx, args, s);
  else
    rc = ordered ? launch_lookback_passes<U, KIND, V, RANK_ORDERED_ATOMIC>(ctx, args, kpt, chained, s)
                 : launch_lookback_passes<U, KIND, V, RANK_PEER_MASK>(ctx, args, kpt, chained, s);
  if (rc != HPCS_OK) return rc;
  // finalize: result back into the caller's buffer if it ended in B; collect errors
  {
    int64_t want = (n + 255) / 256;
    int grid = int(want > int64_t(ctx->sms) * 8 ? int64_t(ctx->sms) * 8 : want);
    KernelTimer kt(ctx, s, HPCS_K_FINALIZE);
    HPCS_CUDA(launch_chained(chained, finalize_kernel<U>, grid, 256, 0, s, args, PAIRS ? 1 : 0, device_error_word(ctx)));
  }
  if (keys_unaligned)
    HPCS_CUDA(cudaMemcpyAsync(keys, a, size_t(n) * sizeof(U), cudaMemcpyDeviceToDevice, s));
  if (vals_unaligned) HPCS_CUDA(cudaMemcpyAsync(vals, va, size_t(n) * 4, cudaMemcpyDeviceToDevice, s));
  return HPCS_OK;
}

// Instantiated once each (sort_u32.cu, sort_u64.cu, pairs_u32.cu, pairs_u64.cu).
#ifndef HPCS_INSTANTIATE_SORTS
#define HPCS_EXTERN_SORT(U, KIND)                                                               \
  extern template int enqueue_sort<U, KIND, NoValue>(hpcs_ctx*, U*, uint32_t*, int64_t, cudaStream_t); \
  extern template int enqueue_sort<U, KIND, uint32_t>(hpcs_ctx*, U*, uint32_t*, int64_t, cudaStream_t);
HPCS_EXTERN_SORT(uint32_t, KIND_UNSIGNED)
HPCS_EXTERN_SORT(uint32_t, KIND_SIGNED)
HPCS_EXTERN_SORT(uint32_t, KIND_FLOAT)
HPCS_EXTERN_SORT(uint64_t, KIND_UNSIGNED)
HPCS_EXTERN_SORT(uint64_t, KIND_SIGNED)
HPCS_EXTERN_SORT(uint64_t, KIND_FLOAT)
#undef HPCS_EXTERN_SORT
#endif

}  // namespace hpcs
