// LSD radix sort kernels for sm_100a.
//
// Restates HPCsharp's LSD hot path (RadixSortLsd.cs, RadixSortLsdParallel.cs,
// Histogram.cs, HistogramParallel.cs) as three kernels per sort:
//
//   K1 hist_all_digits  One 128-bit vectorised read of every key builds the byte histogram
//                       of every digit at once (HistogramByteComponents[Par],
//                       Histogram.cs:261-296, HistogramParallel.cs:163-222).  The last CTA
//                       to finish turns the counts into the per-digit exclusive starts
//                       (ComputeStartOfBins, RadixSortLsd.cs:112-125), marks digit passes
//                       whose keys all share one digit value as skippable (the idea of
//                       RadixSortLsd.cs:2093-2117), and assigns ping-pong buffers.
//   K3 digit passes     One launch per 8-bit digit: a single sweep whose tiles' offsets one CTA
//                       scans (lookback_pass.cuh) or per-range passes without inter-CTA waiting
//                       (chunk_pass.cuh).  Ranking is stable (input order within a digit), so a
//                       pass equals the reference's stable scatter (RadixSortLsdParallel.cs:96-135
//                       with the bin-major / quantum-minor offsets of :49-94).
//   finalize            Copies the result back to the caller's buffer when an odd number of
//                       passes ran (only possible when passes were skipped).
#pragma once
#include <cstdint>
#include <type_traits>

#include "common.cuh"

namespace hpcs {

constexpr int RADIX = 256;
constexpr int MAX_PASSES = 8;

constexpr int64_t MAX_KEYS_PER_SORT = (int64_t(1) << 31) - 1;     // positions below 2^31
// A forced look-back scheme has always refused more (its former passes had 30-bit prefixes); the present
// ones have no such limit, and the default scheme runs them for every size.
constexpr int64_t MAX_KEYS_LOOKBACK = (int64_t(1) << 30) - 1;
struct NoValue {};

// Per-sort control block in device memory (zeroed before K1).
struct SortPlan {
  uint32_t hist[MAX_PASSES][RADIX];       // raw digit counts
  uint32_t bin_start[MAX_PASSES][RADIX];  // exclusive scan per digit
  int32_t src_sel[MAX_PASSES];            // 0: A->B, 1: B->A, -1: pass skipped
  uint32_t tile_counter[MAX_PASSES];
  int32_t final_sel;                      // buffer holding the result (0 = A)
  uint32_t done_blocks;
  uint32_t error;                         // DeviceError bits
  uint32_t idle_flag;                     // never written: the wait-timeout test hook spins on it
  int32_t exec_idx[MAX_PASSES];           // 0, 1, 2, ... over the executed passes
  int32_t next_shift[MAX_PASSES];         // bit shift of the next executed pass's digit, -1 if none
  int32_t heavy[MAX_PASSES];              // the most frequent value of each digit (lowest on ties)
  int32_t skewed[MAX_PASSES];             // 1 when that value holds more than 1/32 of the keys
  int32_t heavy2[MAX_PASSES];             // the second most frequent value
  int32_t grouped[MAX_PASSES];            // 1 when the first holds more than 5/16 of the keys
};

struct SortArgs {
  void* keys_a;
  void* keys_b;
  void* vals_a;
  void* vals_b;
  int64_t n;
  SortPlan* plan;
  uint32_t* status[2];    // look-back passes: [tiles][256] totals and bases (lookback_pass.cuh)
  int num_tiles;
  int pass;
  int skip_trivial;
  int poison_tile;        // test hook: this tile never publishes (-1 = off)
  uint64_t spin_limit_ns; // bound on every device-side wait
  // Tile trace (debug): when non-null, thread 0 writes TRACE_WORDS stamps per tile of
  // pass `trace_pass`: tile id, SM id, then %globaltimer at start, data ready, ranked,
  // look-back done (digit 0), end of scatter.
  uint64_t* trace;
  int trace_pass;
  int trace_capacity;  // tiles
  // Chunked passes (chunk_hist != null): the keys are cut into `chunks` ranges of
  // chunk_keys keys (a whole number of tiles); CTA j of every kernel owns range j.
  uint32_t* chunk_hist;   // [chunks][P][256] digit counts of each input range (K1)
  uint32_t* ctab;         // [3][chunks][256] per-range counts of the next executed digit
  int chunks;
  uint32_t chunk_keys;
  uint32_t chunk_magic;   // ceil(2^32 / chunk_keys): range of position p = umulhi(p, magic) (-1)
};
constexpr int TRACE_WORDS = 7;

__device__ __forceinline__ uint32_t sm_id() {
  uint32_t v;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(v));
  return v;
}

// =====================================================================================
// K1: fused all-digit histogram (+ plan in the last CTA)
// =====================================================================================
// Counters are privatised per lane: bin b of digit d for lane l lives at word
// (d*256 + b)*COPIES + l % COPIES, so the 32 shared atomics of one warp instruction fall in
// (nearly) distinct banks whatever the key values -- one shared-memory wavefront each
// instead of ~3.3 for random bins.  32-bit keys: 32 copies (4 x 256 x 32 words = 128 KiB);
// 64-bit keys: 16 copies (8 x 256 x 16 words = 128 KiB).
template <class U>
struct HistSmem {
  static constexpr int P = int(sizeof(U));
  static constexpr int COPIES = P == 4 ? 32 : 16;
  static constexpr size_t BYTES = size_t(P) * RADIX * COPIES * 4;
};

// 16-byte vectors in flight per thread in the histogram's read (8 x 16 B x 1024 threads = 128 KiB
// per SM).
#ifndef HPCS_HIST_VIF
#define HPCS_HIST_VIF 8
#endif

// cta / ncta: this CTA's index and the CTA count of this array's histogram (the grid of a
// single-array launch; the array's ranges in the batched sort's grid-level launch).
template <class U, int KIND, int NT>
__device__ __forceinline__ void hist_all_digits_body(const U* __restrict__ keys, int64_t n,
                                                     uint32_t* __restrict__ hist_out, const SortArgs& args,
                                                     int make_plan, const int cta, const int ncta) {
  constexpr int P = HistSmem<U>::P;
  constexpr int COPIES = HistSmem<U>::COPIES;
  constexpr int VEC = 16 / int(sizeof(U));
  using KO = KeyOrder<U, KIND>;
  extern __shared__ __align__(16) uint32_t sh[];  // [P][256][COPIES]
  __shared__ uint32_t s_last;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int copy = lane & (COPIES - 1);
  for (int i = tid; i < P * RADIX * COPIES; i += NT) sh[i] = 0;
  __syncthreads();

  auto count_key = [&](U k) {
    const U o = KO::to_ordered(k);
#pragma unroll
    for (int d = 0; d < P; d++) {
      const uint32_t dg = uint32_t(o >> (8 * d)) & 0xFFu;
      atomicAdd(&sh[(d * RADIX + dg) * COPIES + copy], 1u);
    }
  };

  // Grid-stride over all vectors, or (chunked) CTA j over the vectors of key range j.
  const bool chunked = args.chunk_hist != nullptr;
  const int64_t nvec = n / VEC;
  const uint4* vkeys = reinterpret_cast<const uint4*>(keys);
  int64_t vend = nvec, stride = int64_t(ncta) * NT;
  int64_t i = int64_t(cta) * NT + tid;
  bool owns_tail = cta == 0;
  if (chunked) {
    const int64_t lo = int64_t(cta) * args.chunk_keys;  // a multiple of VEC
    const int64_t hi = lo + args.chunk_keys < n ? lo + args.chunk_keys : n;
    i = lo / VEC + tid;
    vend = hi / VEC;
    stride = NT;
    owns_tail = hi == n;
  }
  // HPCS_HIST_VIF vectors in flight per thread per iteration
  for (; i + (HPCS_HIST_VIF - 1) * stride < vend; i += HPCS_HIST_VIF * stride) {
    uint4 v[HPCS_HIST_VIF];
#pragma unroll
    for (int u = 0; u < HPCS_HIST_VIF; u++) v[u] = ldg_stream_v4(vkeys + i + u * stride);
#pragma unroll
    for (int u = 0; u < HPCS_HIST_VIF; u++) {
      const U* e = reinterpret_cast<const U*>(&v[u]);
#pragma unroll
      for (int j = 0; j < VEC; j++) count_key(e[j]);
    }
  }
  for (; i < vend; i += stride) {
    const uint4 v = ldg_stream_v4(vkeys + i);
    const U* e = reinterpret_cast<const U*>(&v);
#pragma unroll
    for (int j = 0; j < VEC; j++) count_key(e[j]);
  }
  // ragged tail (fewer than VEC keys)
  if (owns_tail && tid < VEC) {
    const int64_t t = nvec * VEC + tid;
    if (t < n) count_key(keys[t]);
  }
  __syncthreads();
  // fold the copies (rotated start so a warp's reads hit distinct banks) into the output,
  // and (chunked) into this range's row of per-range counts
  uint32_t* crow = chunked ? args.chunk_hist + int64_t(cta) * P * RADIX : nullptr;
  for (int j = tid; j < P * RADIX; j += NT) {
    uint32_t c = 0;
#pragma unroll 8
    for (int q = 0; q < COPIES; q++) c += sh[j * COPIES + ((q + lane) & (COPIES - 1))];
    if (c) atomicAdd(hist_out + j, c);
    if (chunked) crow[j] = c;
  }

  if (!make_plan) return;

  if (chunked) {
    // the first executed pass adds its next-digit counts into table 1
    uint32_t* t1 = args.ctab + (int64_t(args.chunks) + cta) * RADIX;
    for (int j = tid; j < RADIX; j += NT) t1[j] = 0;
  } else {
    // Clear the tile rows of the look-back passes (totals and bases).
    const int64_t words = int64_t(args.num_tiles) * RADIX;
    const int64_t gstride = int64_t(ncta) * NT;
    for (int64_t w = int64_t(cta) * NT + tid; w < words; w += gstride) {
      args.status[0][w] = 0;
      args.status[1][w] = 0;
    }
  }
  // Last-block-done: the final CTA builds the plan.
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = (atomicAdd(&args.plan->done_blocks, 1u) == uint32_t(ncta) - 1u) ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  SortPlan* plan = args.plan;
  // 256 threads per digit, NT / 256 digits at a time
  constexpr int GROUPS = NT / RADIX;
  static_assert(P % GROUPS == 0 || GROUPS % P == 0, "whole rounds of digits");
  __shared__ uint32_t s_trivial[P];
  __shared__ uint32_t s_wsum[NT / 32];
  __shared__ unsigned long long s_heavy[P];
  __shared__ unsigned long long s_heavy2[P];
  if (tid < P) {
    s_trivial[tid] = 0;
    s_heavy[tid] = 0ull;
    s_heavy2[tid] = 0ull;
  }
  __syncthreads();
  const int grp = tid / RADIX, bin = tid % RADIX;
  for (int d0 = 0; d0 < P; d0 += GROUPS) {
    const int d = d0 + grp;
    const bool on = d < P;
    const uint32_t c = on ? ld_volatile(&hist_out[d * RADIX + bin]) : 0u;
    // most frequent value: max of (count, 255 - value); then the most frequent of the others
    const unsigned long long packed = (static_cast<unsigned long long>(c) << 8) | uint32_t(255 - bin);
    unsigned long long best = packed;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xFFFFFFFFu, best, o);
      best = y > best ? y : best;
    }
    if (on && lane == 0 && (best >> 8)) atomicMax(&s_heavy[d], best);
    if (on && int64_t(c) == n) s_trivial[d] = 1;
    // exclusive scan of the digit's 256 counts (8 warps)
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_wsum[tid >> 5] = incl;
    __syncthreads();
    unsigned long long next = on && c && packed != s_heavy[d] ? packed : 0ull;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xFFFFFFFFu, next, o);
      next = y > next ? y : next;
    }
    if (on && lane == 0 && next) atomicMax(&s_heavy2[d], next);
    uint32_t base = 0;
    for (int w = grp * (RADIX / 32); w < (tid >> 5); w++) base += s_wsum[w];
    if (on) plan->bin_start[d][bin] = base + incl - c;
    __syncthreads();
  }
  if (tid == 0) {
    int sel = 0, executed = 0, prev = -1;
    for (int d = 0; d < MAX_PASSES; d++) {
      plan->tile_counter[d] = 0;
      plan->exec_idx[d] = -1;
      plan->next_shift[d] = -1;
      plan->heavy[d] = d < P ? int(255u - uint32_t(s_heavy[d] & 255ull)) : 0;
      plan->skewed[d] = d < P && int64_t(s_heavy[d] >> 8) > n / 32 ? 1 : 0;
      plan->heavy2[d] = d < P && s_heavy2[d] ? int(255u - uint32_t(s_heavy2[d] & 255ull)) : plan->heavy[d];
      plan->grouped[d] = d < P && int64_t(s_heavy[d] >> 8) > n / 16 * 5 ? 1 : 0;
      if (d >= P) {
        plan->src_sel[d] = -1;
        continue;
      }
      bool skip = args.skip_trivial && s_trivial[d];
      if (skip) {
        plan->src_sel[d] = -1;
      } else {
        plan->src_sel[d] = sel;
        plan->exec_idx[d] = executed;
        if (prev >= 0) plan->next_shift[prev] = 8 * d;
        prev = d;
        sel ^= 1;
        executed++;
      }
    }
    plan->final_sel = sel;
    __threadfence();
  }
}

template <class U, int KIND, int NT>
__global__ void __launch_bounds__(NT, 1) hist_all_digits_kernel(const U* __restrict__ keys, int64_t n,
                                                                 uint32_t* __restrict__ hist_out,
                                                                 SortArgs args, int make_plan) {
  chain_release();
  hist_all_digits_body<U, KIND, NT>(keys, n, hist_out, args, make_plan, int(blockIdx.x), int(gridDim.x));
}

// The fused histogram (and plan) of many arrays in one launch (the batched sort's grid-level
// path): CTA c counts range map[c].y of array map[c].x, whose sort arguments are args[map[c].x].
template <class U, int KIND, int NT>
__global__ void __launch_bounds__(NT, 1) seg_hist_all_digits_kernel(const SortArgs* __restrict__ args,
                                                                    const int2* __restrict__ map) {
  const int2 m = map[blockIdx.x];
  const SortArgs a = args[m.x];
  hist_all_digits_body<U, KIND, NT>(static_cast<const U*>(a.keys_a), a.n, &a.plan->hist[0][0], a, 1, m.y, a.chunks);
}

// =====================================================================================
// K3: shared parts of the 8-bit digit passes
// =====================================================================================
//
// In-warp stable ranking.  Keys sit warp-striped (key i of lane l is tile position
// w*32*KPT + i*32 + l), so a warp's keys in (i, lane) order are in input order.  Each warp
// owns 256 digit counters in shared memory; the rank of a key among the warp's earlier
// keys with the same digit is
//   RANK_ORDERED_ATOMIC  the value returned by one shared-memory atomicAdd per key.  This
//                        relies on the hardware resolving same-address atomics of one warp
//                        instruction in ascending lane order.  PTX leaves that order
//                        undefined, so every context verifies it first with
//                        rank_probe_kernel (the same code path) and otherwise uses:
//   RANK_PEER_MASK       fully defined: each lane ORs its lane bit into a per-(warp, digit)
//                        mask; after __syncwarp the mask is the set of same-digit lanes
//                        (the peers), the rank is counter + popc(peers below me), and the
//                        lowest peer advances the counter and clears the mask.
// Both give identical ranks.  (__match_any_sync / ballots would also be defined but
// run 10-20x slower than one shared atomic on this part.)
enum RankMode : int { RANK_ORDERED_ATOMIC = 0, RANK_PEER_MASK = 1 };

template <int MODE>
__device__ __forceinline__ uint32_t rank_in_warp(uint32_t* cnt, uint32_t* msk, uint32_t d, bool valid, int parity,
                                                 int lane) {
  if (MODE == RANK_ORDERED_ATOMIC) {
    return valid ? atomicAdd(&cnt[d], 1u) : 0u;
  } else {
    uint32_t* m = msk + parity * RADIX + (valid ? d : 0u);
    if (valid) atomicOr(m, 1u << lane);
    __syncwarp();
    const uint32_t peers = valid ? *reinterpret_cast<volatile uint32_t*>(m) : 0u;
    const uint32_t before = valid ? cnt[d] : 0u;
    const uint32_t lt = peers & lanemask_lt();
    __syncwarp();
    if (valid && lt == 0u) {
      cnt[d] = before + __popc(peers);
      *m = 0u;
    }
    return before + __popc(lt);
  }
}

// Ordered-atomic ranking for a pass whose two most frequent digit values h1, h2 hold much of the keys:
// their lanes would serialise on two counters.  A value's keys in a warp are counted in a register
// instead (every lane holds the same count) and rank by that count and a popcount of the vote, without
// touching shared memory; the other lanes rank with their own atomic.  Same ranks as
// rank_in_warp<RANK_ORDERED_ATOMIC>.  All lanes call rank() once per row of keys, then close() once.
// The votes are worth it from h1 ~ 0.3 of the keys on, whether h2 is as frequent or rare (us per look-back
// pass, atomics / votes, one value of share 0.25, 0.35, 0.5, 1: 32 Mi u32 keys 113 / 124, 126 / 125,
// 141 / 123, 190 / 104; 16 Mi u64 pairs 111 / 113, 115 / 112, 123 / 111, 138 / 98; two values of together
// 0.5, 0.7, 1: u32 keys 119 / 121, 129 / 118, 140 / 109).
struct FrequentRanks {
  uint32_t h1, h2;  // h2 == RADIX: there is no second value
  uint32_t c1 = 0u, c2 = 0u;
  __device__ __forceinline__ FrequentRanks(uint32_t a, uint32_t b) : h1(a), h2(b != a ? b : uint32_t(RADIX)) {}
  __device__ __forceinline__ uint32_t rank(uint32_t* cnt, uint32_t d, bool valid) {
    const bool is1 = valid && d == h1, is2 = valid && d == h2;
    const uint32_t m1 = __ballot_sync(0xFFFFFFFFu, is1), m2 = __ballot_sync(0xFFFFFFFFu, is2);
    uint32_t r = 0u;
    if (valid && !is1 && !is2) r = atomicAdd(&cnt[d], 1u);
    if (is1 || is2) r = (is1 ? c1 : c2) + uint32_t(__popc((is1 ? m1 : m2) & lanemask_lt()));
    c1 += uint32_t(__popc(m1));
    c2 += uint32_t(__popc(m2));
    return r;
  }
  // the two counters, which no atomic touched
  __device__ __forceinline__ void close(uint32_t* cnt, int lane) const {
    if (lane == 0) cnt[h1] = c1;
    if (lane == 1 && h2 < uint32_t(RADIX)) cnt[h2] = c2;
  }
};

// Issue the bulk copy of tile t (keys, then items, at dst) with mbar as its barrier (called by one
// thread).  The 16-byte-aligned body is copied by the TMA engine; the ragged tail (< 16 bytes) is
// read with plain loads by the consumers.  A tile past the end arrives with zero bytes.
template <class U, bool PAIRS, int TILE>
__device__ __forceinline__ void stage_tile(unsigned char* dst, size_t keys_bytes, uint64_t* mbar, const U* kin,
                                           const uint32_t* vin, int64_t n, int64_t t) {
  const int64_t base = t * TILE;
  int64_t cnt = n - base;
  cnt = cnt < 0 ? 0 : (cnt < TILE ? cnt : TILE);
  const uint32_t kbytes = uint32_t((cnt * int64_t(sizeof(U))) & ~int64_t(15));
  const uint32_t vbytes = PAIRS ? uint32_t((cnt * 4) & ~int64_t(15)) : 0u;
  fence_proxy_async_smem();
  mbar_arrive_expect_tx(mbar, kbytes + vbytes);
  if (kbytes) bulk_copy_g2s(dst, kin + base, kbytes, mbar);
  if (PAIRS && vbytes) bulk_copy_g2s(dst + keys_bytes, vin + base, vbytes, mbar);
}

// Verifies, on this GPU, that the ordered-atomic ranking gives lane-ordered (stable) ranks:
// every warp ranks KPT x 32 digits with exactly the passes' code and compares each rank
// with a brute-force count of earlier equal digits.  Patterns: uniform bytes, 4 values,
// one value, and partial last rows.  Mismatches are added to *bad.
template <int NT, int KPT>
__global__ void __launch_bounds__(NT) rank_probe_kernel(uint32_t* bad, uint32_t seed) {
  constexpr int NW = NT / 32;
  __shared__ uint32_t cnt[NW][RADIX];
  __shared__ uint16_t dig[NW][32 * KPT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t mism = 0;
  for (int pattern = 0; pattern < 4; pattern++) {
    for (int i = lane; i < RADIX; i += 32) cnt[warp][i] = 0u;
    const int valid_n = pattern == 3 ? (32 * KPT - 37) : 32 * KPT;
    __syncwarp();
    uint32_t x = seed ^ (blockIdx.x * 0x9E3779B9u) ^ (threadIdx.x * 0x85EBCA6Bu) ^ (pattern * 0xC2B2AE35u);
    uint32_t d[KPT], r[KPT];
#pragma unroll
    for (int i = 0; i < KPT; i++) {
      x ^= x << 13;
      x ^= x >> 17;
      x ^= x << 5;
      d[i] = pattern == 0 ? (x & 255u) : pattern == 1 ? (x & 3u) : pattern == 2 ? 9u : ((x >> 3) & 7u);
      dig[warp][i * 32 + lane] = uint16_t(d[i]);
    }
#pragma unroll
    for (int i = 0; i < KPT; i++) {
      const bool valid = i * 32 + lane < valid_n;
      r[i] = rank_in_warp<RANK_ORDERED_ATOMIC>(cnt[warp], nullptr, d[i], valid, i & 1, lane);
    }
    __syncwarp();
    for (int i = 0; i < KPT; i++) {
      const int pos = i * 32 + lane;
      if (pos >= valid_n) continue;
      uint32_t want = 0;
      for (int q = 0; q < pos; q++) want += (dig[warp][q] == d[i]) ? 1u : 0u;
      if (want != r[i]) mism++;
    }
    __syncwarp();
  }
  if (mism) atomicAdd(bad, mism);
}

// Copy B -> A when the result ended in the scratch buffer, and fold this sort's device
// error bits into the context's accumulator.
template <class U>
__global__ void finalize_kernel(SortArgs args, int has_vals, uint32_t* err_accum) {
  chain_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    uint32_t e = ld_volatile(&args.plan->error);
    if (e) atomicOr(err_accum, e);
  }
  if (args.plan->final_sel != 1) return;
  const int64_t n = args.n;
  const U* src = static_cast<const U*>(args.keys_b);
  U* dst = static_cast<U*>(args.keys_a);
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = src[i];
  if (has_vals) {
    const uint32_t* vs = static_cast<const uint32_t*>(args.vals_b);
    uint32_t* vd = static_cast<uint32_t*>(args.vals_a);
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) vd[i] = vs[i];
  }
}

// The batched sort's grid-level path: CTA c copies range map[c].y of array map[c].x back into
// the caller's buffer when that array's result ended in its scratch buffer (an odd number of
// passes ran), and the array's first CTA folds its device error bits into the context's word.
template <class U>
__global__ void seg_finalize_kernel(const SortArgs* __restrict__ args, const int2* __restrict__ map,
                                    uint32_t* err_accum) {
  const int2 m = map[blockIdx.x];
  const SortArgs a = args[m.x];
  if (m.y == 0 && threadIdx.x == 0) {
    const uint32_t e = ld_volatile(&a.plan->error);
    if (e) atomicOr(err_accum, e);
  }
  if (a.plan->final_sel != 1) return;
  const int64_t lo = int64_t(m.y) * a.chunk_keys;
  const int64_t hi = lo + a.chunk_keys < a.n ? lo + a.chunk_keys : a.n;
  const U* src = static_cast<const U*>(a.keys_b);
  U* dst = static_cast<U*>(a.keys_a);
  for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) dst[i] = src[i];
}

}  // namespace hpcs
