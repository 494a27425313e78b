// Radix selection / top-k on the GPU.
//
// Restates the observable contract of HPCsharp's SelectTopK(this uint[] a, int k)
// (SelectionTopKRadix.cs:142-171): afterwards a[k] is the k-th smallest key (0-based) and
// a[k..n-1] holds exactly the multiset of the n-k largest.  The reference gets there with an
// in-place MSD radix select of 16-bit digits (RadixSelectionTopKWordInner, :96-133) whose
// movers clobber the prefix; here the prefix is defined too: a[0..k-1] holds the k smallest.
//
// Selection: an MSD radix select over the order-transformed key (the same transforms as the
// sort), 8 bits per level.  A strided sample of the keys first bounds where the selected key
// lies: a window around its rank (for the k largest, the window is open at the top).  One read of
// all keys keeps the keys inside (the candidates) and counts those below; the levels then
// histogram only candidates that match the prefix chosen so far, and the last CTA of each level
// picks the bin and advances the device-side SelectState.  When the sample misled (the rank falls
// outside the candidates), the levels run over all keys instead: level 0 histograms all n keys and
// the keys of the chosen bin are compacted into the candidate buffer.  The choice is made on the
// device, so nothing returns to the host between levels, and the launches are chained.
//
// Rearrangement: a stable three-way partition (keys < v, == v, > v around the selected key v).  The
// candidates of a tile lie together, so the tiles' class counts come from the window read's counts
// and the candidates, without another read of the keys; a scan of them; a stable per-tile scatter.
// The k largest ("top-k" of a serving request) are the keys > v among the candidates plus
// copies of v up to k, sorted ascending (in one CTA for up to 256 keys, else with the LSD
// sort) so the output bytes are deterministic.
#pragma once
#include <cstdint>

#include "cluster_sort.cuh"
#include "common.cuh"

namespace hpcs {

struct SelectState {
  uint64_t prefix;     // ordered-key bits chosen so far
  uint64_t mask;       // which bits of the prefix are fixed
  int64_t rank;        // rank still to find among keys matching the prefix
  int64_t less;        // keys strictly below the prefix range
  int64_t eq;          // keys equal to the selected key (valid after the last level)
  int64_t cand_count;  // candidates compacted after level 0
  unsigned long long gathered;  // keys > v written to the top-k output so far
  int64_t n_total;     // keys selected among
  uint64_t threshold;           // the window's lower end
  uint64_t threshold_hi;        // the window's upper end (inclusive)
  unsigned long long below;     // keys below the window
  int32_t mode;        // where the levels look (SelMode)
  uint32_t ticket;     // CTAs of the current level that are through
  uint32_t hist[256];
};
// Where the levels look: the window's candidates (CAND), the candidates of the top-byte bin that level 0
// chose among all keys (FULL), those strictly between the window's ends (INSIDE), or nowhere, since the
// selected key is one of the ends (DONE).  All but CAND are the shift of the first level that the finish runs.
template <class U>
struct SelMode {
  static constexpr int32_t TOP = int32_t(sizeof(U) * 8) - 8;
  static constexpr int32_t CAND = 255, FULL = TOP - 8, INSIDE = TOP, DONE = -1;
};

constexpr int SEL_NT = 512;
constexpr int SEL_COPIES = 32;
constexpr int SEL_VPT = 4;  // 16-byte vectors in flight per thread
constexpr int SEL_CTAS_PER_SM = 4;

// Per-warp staging of appended keys in shared memory: a warp scan places each lane's keys in
// the warp's CAP-key buffer, and a buffer that would overflow goes to dst with one atomic on
// the global counter, so a sparse compaction takes one atomic per CAP keys instead of one per
// warp and vector row.  Every lane of the warp makes the same calls; count is the same in all
// lanes.  Positions at or beyond `cap` are not written.
template <class U, int E, int CAP>
struct WarpStage {
  U* buf;
  uint32_t count;
  U* dst;
  unsigned long long* counter;
  int64_t cap;

  __device__ __forceinline__ void flush() {
    if (count == 0u) return;
    const int lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(counter, (unsigned long long)count);
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    for (uint32_t j = lane; j < count; j += 32)
      if (int64_t(base + j) < cap) dst[base + j] = buf[j];
    __syncwarp();
    count = 0u;
  }

  __device__ __forceinline__ void add(const U* k, uint32_t take) {
    static_assert(32 * E <= CAP, "one call must fit an empty buffer");
    if (__ballot_sync(0xFFFFFFFFu, take != 0u) == 0u) return;  // nothing kept by the warp
    const int lane = threadIdx.x & 31;
    const uint32_t c = __popc(take);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (total == 0u) return;  // uniform over the warp
    if (count + total > uint32_t(CAP)) flush();
    uint32_t pos = count + incl - c;
#pragma unroll
    for (int e = 0; e < E; e++)
      if ((take >> e) & 1u) buf[pos++] = k[e];
    count += total;
    __syncwarp();  // the keys are in the buffer before any lane flushes it
  }
};

// One level: histogram of the digit at `shift` over the keys whose ordered bits match (prefix,
// mask); the last CTA through chooses the bin that holds st->rank, advances the prefix and clears the
// histogram.  Level 0 (shift = bits - 8) first decides between the candidates and all n keys: the
// rank must fall among the candidates.  CTAs beyond what the keys can use return at once, so the
// grid can be large enough for all keys.  (Separate decide, histogram and pick launches took ~55 us
// of a 285 us top-k call.)
// FINISH: select_finish_kernel takes the candidates, so level 0 has work only where the rank is not
// among them, or where they are more than `limit`.  So many more than expected are copies of the window's
// ends (a value between them that filled as much would have filled the sample too): level 0 counts the
// copies, and the rank falls on an end (DONE) or strictly between, where the expected few keys lie
// (INSIDE: compacted anew).  The cluster of the finish would read them all once per level: the 1000
// largest of 2^27 u32 keys, half of them the largest value, 2590 -> 467 us, all keys equal 4950 -> 743.
template <class U, int KIND, bool FINISH>
__global__ void __launch_bounds__(SEL_NT, SEL_CTAS_PER_SM) select_level_kernel(const U* keys, int64_t n,
                                                                              const U* cand, int64_t rank,
                                                                              SelectState* st, int shift, int open_top,
                                                                              int64_t limit) {
  using KO = KeyOrder<U, KIND>;
  constexpr int E = int(16 / sizeof(U));
  constexpr int TOP_SHIFT = int(sizeof(U) * 8) - 8;
  __shared__ uint32_t sh[256 * SEL_COPIES];
  __shared__ uint32_t s_last;
  __shared__ int64_t s_w[8];
  __shared__ int s_bin;
  __shared__ int64_t s_excl, s_cnt;
  chain_wait();
  chain_release();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the window is open at the top for the k largest: the other keys lie below it
  const int64_t c = st->cand_count, below = open_top ? n - c : int64_t(st->below);
  const bool first = shift == TOP_SHIFT;
  const bool among = first ? below <= rank && rank < below + c : true;  // rank among the candidates
  bool wide = false;
  if (FINISH && among) {
    if (c <= limit) return;
    wide = st->threshold != st->threshold_hi;  // (equal ends: the finish reads no candidate)
    if (!wide) return;
  }
  const U* src = among ? cand : keys;
  const int64_t m = among ? c : n;
  const int64_t per_cta = int64_t(SEL_NT) * SEL_VPT * E;
  // (the whole grid where the last CTA resets cand_count: no CTA may read it after that)
  const int64_t want = ((wide ? n : m) + per_cta - 1) / per_cta;
  const uint32_t active = want < 1 ? 1u : (want < int64_t(gridDim.x) ? uint32_t(want) : gridDim.x);
  if (blockIdx.x >= active) return;
  const U prefix = first ? U(0) : U(st->prefix), mask = first ? U(0) : U(st->mask);
  for (int i = tid; i < 256 * SEL_COPIES; i += SEL_NT) sh[i] = 0;
  __syncthreads();
  if (FINISH && wide) {  // bins 0 and 1: the copies of the window's ends
    const U lo = U(st->threshold), hi = U(st->threshold_hi);
    uint32_t nlo = 0u, nhi = 0u;
    visit_keys<U, SEL_VPT>(src, m, active, [&](const U* k, int nv) {
#pragma unroll
      for (int e = 0; e < E; e++) {
        const U o = KO::to_ordered(k[e]);
        nlo += e < nv && o == lo ? 1u : 0u;
        nhi += e < nv && o == hi ? 1u : 0u;
      }
    });
    nlo = __reduce_add_sync(0xFFFFFFFFu, nlo);
    nhi = __reduce_add_sync(0xFFFFFFFFu, nhi);
    if (lane == 0) {
      atomicAdd(&sh[0], nlo);
      atomicAdd(&sh[SEL_COPIES], nhi);
    }
  } else {
    visit_keys<U, SEL_VPT>(src, m, active, [&](const U* k, int nv) {
#pragma unroll
      for (int e = 0; e < E; e++) {
        const U o = KO::to_ordered(k[e]);
        if (e < nv && (o & mask) == prefix) atomicAdd(&sh[((uint32_t(o >> shift) & 0xFFu) * SEL_COPIES) + lane], 1u);
      }
    });
  }
  __syncthreads();
  for (int b = tid; b < 256; b += SEL_NT) {
    uint32_t h = 0;
    for (int q = 0; q < SEL_COPIES; q++) h += sh[b * SEL_COPIES + ((q + lane) & (SEL_COPIES - 1))];
    if (h) atomicAdd(&st->hist[b], h);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&st->ticket, 1u) == active - 1u ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();

  if (FINISH && wide) {
    if (tid == 0) {
      const U lo = U(st->threshold), hi = U(st->threshold_hi);
      const int64_t nlo = ld_volatile(&st->hist[0]), nhi = ld_volatile(&st->hist[1]);
      const int64_t r = rank - below;
      const bool at_lo = r < nlo, at_hi = !at_lo && r >= c - nhi;
      st->mode = at_lo || at_hi ? SelMode<U>::DONE : SelMode<U>::INSIDE;
      st->less = below + (at_lo ? 0 : at_hi ? c - nhi : nlo);
      st->eq = at_lo ? nlo : at_hi ? nhi : 0;
      st->rank = at_lo ? r : at_hi ? r - (c - nhi) : r - nlo;
      st->prefix = at_lo ? uint64_t(lo) : at_hi ? uint64_t(hi) : 0ull;
      st->mask = at_lo || at_hi ? uint64_t(U(~U(0))) : 0ull;
      st->cand_count = 0;  // INSIDE: rebuilt by the compaction
      st->hist[0] = 0;
      st->hist[1] = 0;
      st->ticket = 0;
    }
    return;
  }
  // the last CTA: a scan of the 256 counts, the thread whose bin spans the rank records it
  const int64_t r = first ? (among ? rank - below : rank) : st->rank;
  const int64_t h = tid < 256 ? int64_t(ld_volatile(&st->hist[tid])) : 0;
  int64_t incl = h;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31 && warp < 8) s_w[warp] = incl;
  if (tid == 0) {
    s_bin = 255;
    s_excl = 0;
    s_cnt = 0;
  }
  __syncthreads();
  int64_t excl = incl - h;
  for (int w = 0; w < warp && w < 8; w++) excl += s_w[w];
  // the bins' ranges [excl, excl + h) are disjoint: at most one thread matches; a rank past
  // every key (not reachable through the entry points) falls to bin 255
  if (tid < 256 && ((h > 0 && r >= excl && r < excl + h) || (tid == 255 && r >= excl + h))) {
    s_bin = tid;
    s_excl = excl;
    s_cnt = h;
  }
  __syncthreads();
  if (tid < 256) st->hist[tid] = 0;
  if (tid == 0) {
    st->ticket = 0;
    if (first) {
      st->mode = among ? SelMode<U>::CAND : SelMode<U>::FULL;
      st->less = among ? below : 0;
      if (!among) st->cand_count = 0;  // rebuilt by the compaction
    }
    st->prefix = uint64_t(prefix) | uint64_t(s_bin) << shift;
    st->mask = uint64_t(mask) | uint64_t(0xFF) << shift;
    st->rank = r - s_excl;
    st->less += s_excl;
    if (shift == 0) st->eq = s_cnt;
  }
}

// Level 0 looked beyond the candidates: copies the keys of its choice (the bin of the ordered top byte, or
// the keys strictly between the window's ends) into `cand`.  With `out` (top-k): the keys above those, all
// among the k largest, go to out[0..) through st->gathered at once (fewer than k of them: the selected
// rank lies below them).
template <class U, int KIND>
__global__ void __launch_bounds__(SEL_NT, SEL_CTAS_PER_SM) select_compact_kernel(const U* keys, int64_t n,
                                                                U* cand, SelectState* st,
                                                                U* out, int64_t k_out) {
  using KO = KeyOrder<U, KIND>;
  constexpr int E = int(16 / sizeof(U));
  constexpr int CAP = 1024 / int(sizeof(U));  // 1 KiB per warp and buffer
  __shared__ U s_buf[2][SEL_NT / 32][CAP];
  chain_wait();
  chain_release();
  const int32_t mode = st->mode;
  if (mode == SelMode<U>::CAND) return;  // the rank lies among the candidates
  // DONE: only the keys above the selected one are wanted
  if (mode == SelMode<U>::DONE && (!out || st->less + st->eq == n)) return;
  const int warp = threadIdx.x >> 5;
  // [first, last]: the keys for `cand`; none when DONE (first above last: some key lies above last)
  const U prefix = U(st->prefix);
  const U first = mode == SelMode<U>::FULL ? prefix : U((mode == SelMode<U>::INSIDE ? U(st->threshold) : prefix) + 1);
  const U last = mode == SelMode<U>::FULL ? U(prefix | U(~U(st->mask))) : mode == SelMode<U>::INSIDE ? U(U(st->threshold_hi) - 1) : prefix;
  WarpStage<U, E, CAP> to_cand{s_buf[0][warp], 0u, cand, reinterpret_cast<unsigned long long*>(&st->cand_count),
                               INT64_MAX};
  WarpStage<U, E, CAP> to_out{s_buf[1][warp], 0u, out, &st->gathered, k_out};
  visit_keys<U, SEL_VPT>(keys, n, gridDim.x, [&](const U* k, int nv) {
    uint32_t take = 0u, above = 0u;
#pragma unroll
    for (int e = 0; e < E; e++) {
      const U o = KO::to_ordered(k[e]);
      if (e < nv && o >= first && o <= last) take |= 1u << e;
      if (e < nv && o > last) above |= 1u << e;
    }
    to_cand.add(k, take);
    if (out) to_out.add(k, above);
  });
  to_cand.flush();
  if (out) to_out.flush();
}

// The remaining levels in one cluster of CTAs, for up to half a million candidates: all but those
// that the window's two ends share or, when level 0 ran over all keys, the levels below it (none when
// level 0 found the selected key).  Up to 16
// 32-bit candidates per thread stay in registers from level to level.  Per level every CTA
// histograms its share, the 256 totals go to every CTA (distributed shared memory), one cluster
// barrier, and every CTA picks the bin for itself.  With `out` (the k largest): then the candidates
// above the selected key are appended to out and copies of it fill the rest.  (Four level launches of
// ~8.5 us each and a gather of 6 before: 1.1 M candidates in 137 CTAs, bound by the launches' chains of
// latency.)
constexpr int FIN_NT = 1024;
constexpr int64_t FIN_MAX_CANDIDATES = int64_t(1) << 19;  // expected; more share the work of all SMs
struct FinishSmem {
  uint32_t hist[256 * 32];
  uint32_t tot[2][CS_MAX_CTAS][256];  // by the level's parity
};

template <class U, int KIND>
__global__ void __launch_bounds__(FIN_NT, 1) select_finish_kernel(const U* cand, int64_t n, int64_t rank,
                                                                 SelectState* st, int open_top, U* out,
                                                                 int64_t k) {
  using KO = KeyOrder<U, KIND>;
  constexpr int E = int(16 / sizeof(U));
  extern __shared__ __align__(128) unsigned char smem[];
  FinishSmem& sm = *reinterpret_cast<FinishSmem*>(smem);
  __shared__ uint32_t s_w[8];
  __shared__ uint32_t s_pick[3];
  cluster_arrive();  // waited for before the first store to another CTA
  chain_wait();
  chain_release();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t ctas = gridDim.x, cta = blockIdx.x;  // the grid is one cluster
  const int64_t c = st->cand_count;
  const bool window = st->mode == SelMode<U>::CAND;
  const int64_t below = open_top ? n - c : int64_t(st->below);
  U prefix = window ? U(0) : U(st->prefix), mask = window ? U(0) : U(st->mask);
  uint32_t r = uint32_t(window ? rank - below : st->rank);
  int64_t less = window ? below : st->less;
  uint32_t eq = uint32_t(st->eq);  // (0 unless DONE)
  int shift = window ? int(sizeof(U) * 8) - 8 : st->mode;
  if (window) {  // the digits that lo and hi share are every candidate's
    const U lo = U(st->threshold), hi = U(st->threshold_hi);
    while (shift >= 0 && (lo >> shift) == (hi >> shift)) {
      prefix = (lo >> shift) << shift;
      mask |= U(0xFF) << shift;
      shift -= 8;
    }
    if (shift < 0) eq = uint32_t(c);  // lo == hi
  }
  constexpr int V = 4;
  const int64_t gtid = int64_t(cta) * FIN_NT + tid;
  const bool held = c <= int64_t(ctas) * FIN_NT * V * E;  // uniform over the cluster
  U keep[V * E];
  uint32_t valid = 0u;
  if (held) {
#pragma unroll
    for (int j = 0; j < V; j++) {
      const int64_t at = (int64_t(j) * ctas * FIN_NT + gtid) * E;
      if (at + E <= c) {
        const uint4 v = ld_stream_v4(cand + at);
#pragma unroll
        for (int e = 0; e < E; e++) keep[j * E + e] = KO::to_ordered(reinterpret_cast<const U*>(&v)[e]);
        valid |= ((1u << E) - 1u) << (j * E);
      } else {
#pragma unroll
        for (int e = 0; e < E; e++) {
          keep[j * E + e] = at + e < c ? KO::to_ordered(cand[at + e]) : U(0);
          valid |= (at + e < c ? 1u : 0u) << (j * E + e);
        }
      }
    }
  }
  for (int i = tid; i < 256 * 32; i += FIN_NT) sm.hist[i] = 0u;
  cluster_wait();  // every CTA has started
  for (int parity = 0; shift >= 0; shift -= 8, parity ^= 1) {
    __syncthreads();  // the histogram is clear
    auto count = [&](U o) {
      if ((o & mask) == prefix) atomicAdd(&sm.hist[((uint32_t(o >> shift) & 0xFFu) * 32) + lane], 1u);
    };
    if (held) {
#pragma unroll
      for (int i = 0; i < V * E; i++)
        if ((valid >> i) & 1u) count(keep[i]);
    } else {
      visit_keys<U, V>(cand, c, ctas, [&](const U* kk, int nv) {
#pragma unroll
        for (int e = 0; e < E; e++)
          if (e < nv) count(KO::to_ordered(kk[e]));
      });
    }
    __syncthreads();
    // four threads per bin fold its 32 copies and clear them; each stores to a quarter of the CTAs
    {
      const int bin = tid >> 2, q = tid & 3;
      uint32_t h = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        uint32_t* p = &sm.hist[bin * 32 + ((q * 8 + i + bin) & 31)];  // rotated: fewer bank conflicts
        h += *p;
        *p = 0u;
      }
      h += __shfl_xor_sync(0xFFFFFFFFu, h, 1);
      h += __shfl_xor_sync(0xFFFFFFFFu, h, 2);
      const uint32_t slot = smem_u32(&sm.tot[parity][cta][bin]);
      for (uint32_t d = uint32_t(q); d < ctas; d += 4u) cluster_store(cluster_addr(slot, d), h);
    }
    cluster_arrive();
    cluster_wait();  // every CTA's totals of this level are here
    uint32_t h = 0, incl = 0;
    if (tid < 256) {
#pragma unroll
      for (uint32_t d = 0; d < uint32_t(CS_MAX_CTAS); d++) h += d < ctas ? sm.tot[parity][d][tid] : 0u;
      incl = h;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) s_w[warp] = incl;
    }
    __syncthreads();
    if (tid < 256) {
      uint32_t excl = incl - h;
      for (int w = 0; w < warp; w++) excl += s_w[w];
      // the bins' ranges [excl, excl + h) are disjoint: exactly one thread matches
      if (h > 0u && r >= excl && r < excl + h) {
        s_pick[0] = uint32_t(tid);
        s_pick[1] = excl;
        s_pick[2] = h;
      }
    }
    __syncthreads();
    prefix |= U(s_pick[0]) << shift;
    mask |= U(0xFF) << shift;
    r -= s_pick[1];
    less += s_pick[1];
    eq = s_pick[2];
  }
  if (cta == 0 && tid == 0) {
    st->prefix = uint64_t(prefix);
    st->mask = uint64_t(mask);
    st->rank = r;
    st->less = less;
    st->eq = eq;
  }
  if (!out) return;
  const int64_t above = n - less - int64_t(eq);
  if (above == 0) {
    // the selected key is the largest of all: nothing to append
  } else if (held) {
    uint32_t take = 0u;
#pragma unroll
    for (int i = 0; i < V * E; i++) {
      take |= (((valid >> i) & 1u) != 0u && keep[i] > prefix ? 1u : 0u) << i;
      keep[i] = KO::from_ordered(keep[i]);
    }
    warp_append<U, V * E>(keep, take, out, &st->gathered, k);
  } else {
    visit_keys<U, V>(cand, c, ctas, [&](const U* kk, int nv) {
      uint32_t take = 0u;
#pragma unroll
      for (int e = 0; e < E; e++)
        if (e < nv && KO::to_ordered(kk[e]) > prefix) take |= 1u << e;
      warp_append<U, E>(kk, take, out, &st->gathered, k);
    });
  }
  const U vraw = KO::from_ordered(prefix);
  for (int64_t j = above + int64_t(cta) * FIN_NT + tid; j < k; j += int64_t(ctas) * FIN_NT) out[j] = vraw;
}

// ---- the sampled window ---------------------------------------------------------------
// Keys at stride n / S give two values lo <= hi: the sample values of ranks rlo and rhi, which the
// host places m sampled keys below and above the expected sample rank of the selected key (for the k
// largest, hi is open).  One read of all keys then counts the keys below lo and keeps the keys in
// [lo, hi].  The window's width shrinks as 1/sqrt(S): 32-bit keys take 32 Ki samples, 64-bit keys 8 Ki
// (16 per thread would spill registers in the one-CTA select).
template <class U>
__host__ __device__ constexpr int select_sample_size() {
  return sizeof(U) == 4 ? 32768 : 8192;
}
constexpr int SAMPLE_NT = 1024;

// The ordered sample into samp[], one key per thread (a CTA gathering all of it waited ~30 us for cold
// sectors), and the state set up.  Inputs under 4 S keys are not sampled.
template <class U, int KIND>
__global__ void __launch_bounds__(512) select_gather_kernel(const U* __restrict__ keys, int64_t n, U* __restrict__ samp,
                                                            SelectState* st) {
  constexpr int S = select_sample_size<U>();
  chain_release();
  const int i = int(blockIdx.x) * 512 + threadIdx.x;
  if (i == 0) {
    st->n_total = n;
    st->prefix = 0;
    st->mask = 0;
    st->less = 0;
    st->eq = 0;
    st->cand_count = 0;
    st->gathered = 0;
    st->below = 0;
    st->mode = SelMode<U>::CAND;
    st->ticket = 0;
    st->threshold = 0;
    st->threshold_hi = uint64_t(U(~U(0)));
  }
  if (i < 256) st->hist[i] = 0;
  if (n >= int64_t(4) * S && i < S) samp[i] = KeyOrder<U, KIND>::to_ordered(keys[int64_t(i) * (n / S)]);
}

// One CTA: the sample values of ranks rlo and rhi (below 0: the lowest value, at or above S: the
// highest) by two MSD radix selects side by side; per level a histogram of the samples matching each
// prefix and a scan of its 256 bins by 8 warps.
template <class U>
__global__ void __launch_bounds__(SAMPLE_NT) select_sample_kernel(const U* samp, int64_t rlo, int64_t rhi,
                                                                 SelectState* st) {
  constexpr int S = select_sample_size<U>();
  constexpr int PER = S / SAMPLE_NT;
  constexpr int BITS = int(sizeof(U) * 8);
  __shared__ uint32_t hist[2][256];
  __shared__ uint32_t s_wsum[2][8];
  __shared__ uint32_t s_pick[2][2];
  chain_wait();
  chain_release();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  U o[PER];
#pragma unroll
  for (int q = 0; q < PER; q++) o[q] = samp[tid + q * SAMPLE_NT];
  U prefix[2] = {0, 0}, mask = 0;
  // an open end needs no select: the other end's rank serves both
  uint32_t rank[2] = {uint32_t(rlo <= 0 ? rhi : rlo), uint32_t(rhi >= S - 1 ? rlo : rhi)};
  if (rlo <= 0 && rhi >= S - 1) rank[0] = rank[1] = 0u;
  const int which = (tid >> 8) & 1, bin = tid & 255;  // the bin this thread scans (threads < 512)
  for (int shift = BITS - 8; shift >= 0; shift -= 8) {
    const bool same = prefix[0] == prefix[1];  // one histogram serves both (uniform)
    if (tid < 512) hist[which][bin] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < PER; q++) {
      const uint32_t d = uint32_t(o[q] >> shift) & 0xFFu;
      if ((o[q] & mask) == prefix[0]) atomicAdd(&hist[0][d], 1u);
      if (!same && (o[q] & mask) == prefix[1]) atomicAdd(&hist[1][d], 1u);
    }
    __syncthreads();
    uint32_t c = 0, incl = 0;
    if (tid < 512) {
      c = hist[same ? 0 : which][bin];
      incl = c;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if (lane >= off) incl += y;
      }
      if (lane == 31) s_wsum[which][warp & 7] = incl;
    }
    __syncthreads();
    if (tid < 512) {
      uint32_t excl = incl - c;
      for (int w = 0; w < (warp & 7); w++) excl += s_wsum[which][w];
      const uint32_t r = which ? rank[1] : rank[0];
      // the bins' ranges [excl, excl + c) are disjoint: exactly one thread matches
      if (c > 0u && r >= excl && r < excl + c) {
        s_pick[which][0] = uint32_t(bin);
        s_pick[which][1] = excl;
      }
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 2; w++) {
      prefix[w] |= U(s_pick[w][0]) << shift;
      rank[w] -= s_pick[w][1];
    }
    mask |= U(0xFF) << shift;
    __syncthreads();
  }
  if (tid == 0) {
    st->threshold = rlo <= 0 ? 0ull : uint64_t(prefix[0]);
    st->threshold_hi = rhi >= S - 1 ? uint64_t(U(~U(0))) : uint64_t(prefix[1]);
  }
}

// A tile of the window read and of the partition: WIN_NT threads with four 16-byte vectors each.
constexpr int WIN_NT = 512;
template <class U>
__host__ __device__ constexpr int win_tile() {
  return WIN_NT * 64 / int(sizeof(U));
}
// Per tile: its candidates lie at cand[base .. base + count), `below` of its keys below the window.
struct WinTile {
  uint32_t base, count, below;
};

// One read of the keys: keys in [lo, hi] go to `cand`, keys below lo are counted.
//   TILES  (the select) one tile per CTA; each tile's candidates lie together and are recorded with its
//          count of keys below; a key's slot comes from one shared atomic per thread that has any
//          (their order does not matter);
//   !TILES (the k largest, a candidate per warp or fewer expected) `steps` consecutive tiles per CTA; a
//          warp gathers its candidates in shared memory, and the CTA takes one range of the global
//          counter at the end: one barrier and at most one global atomic per CTA (an atomic per warp
//          with candidates cost 2 ns each: 2^27 u64 keys 490 us);
//   COPY   the keys also go to `copy`, so that the partition can write back into the array they came
//          from.
// Short-lived CTAs read faster than persistent ones (2^28 u32 keys, 199 us as a persistent kernel
// that staged kept keys per warp, 5.4 TB/s; a bare read takes 150).
template <class U, int KIND, bool COPY, bool TILES>
__global__ void __launch_bounds__(WIN_NT, TILES || sizeof(U) == 8 ? 3 : 4) select_window_kernel(const U* keys, int64_t n,
                                                               U* cand, SelectState* st,
                                                               U* copy, WinTile* tiles,
                                                               int steps) {
  using KO = KeyOrder<U, KIND>;
  constexpr int E = int(16 / sizeof(U)), V = 4, T = win_tile<U>(), NW = WIN_NT / 32;
  constexpr int CAP = 512 / int(sizeof(U));  // a warp's gathered candidates
  __shared__ uint32_t s_count, s_below;
  __shared__ unsigned long long s_base;
  __shared__ uint32_t s_n[NW];
  __shared__ U s_k[TILES ? 1 : NW][TILES ? 1 : CAP];
  chain_wait();
  chain_release();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (TILES && tid == 0) {
    s_count = 0u;
    s_below = 0u;
  }
  const U lo = U(st->threshold), hi = U(st->threshold_hi);
  const bool aligned = ((reinterpret_cast<uintptr_t>(keys) | (COPY ? reinterpret_cast<uintptr_t>(copy) : 0)) & 15u) == 0;
  unsigned long long* counter = reinterpret_cast<unsigned long long*>(&st->cand_count);
  union Vec {
    uint4 v;
    U k[E];
  } r[V];
  uint32_t take = 0u, below = 0u;  // bit j * E + e: key e of vector j
  // loads the keys at t0 and classifies them
  auto read_tile = [&](int64_t t0) {
    const int tn = int(n - t0 < T ? n - t0 : T);
    uint32_t valid = 0xFFFFFFFFu;
    if (aligned && tn == T) {  // uniform over the CTA
      const uint4* p = reinterpret_cast<const uint4*>(keys + t0);
#pragma unroll
      for (int j = 0; j < V; j++) r[j].v = ld_stream_v4(p + j * WIN_NT + tid);
      if (COPY) {
        uint4* q = reinterpret_cast<uint4*>(copy + t0);
#pragma unroll
        for (int j = 0; j < V; j++) q[j * WIN_NT + tid] = r[j].v;
      }
    } else {
      valid = 0u;
#pragma unroll
      for (int j = 0; j < V; j++) {
#pragma unroll
        for (int e = 0; e < E; e++) {
          const int i = (j * E + e) * WIN_NT + tid;
          r[j].k[e] = i < tn ? keys[t0 + i] : U(0);
          if (i < tn) {
            valid |= 1u << (j * E + e);
            if (COPY) copy[t0 + i] = r[j].k[e];
          }
        }
      }
    }
    take = below = 0u;
#pragma unroll
    for (int j = 0; j < V; j++) {
#pragma unroll
      for (int e = 0; e < E; e++) {
        const U o = KO::to_ordered(r[j].k[e]);
        take |= (o >= lo && o <= hi ? 1u : 0u) << (j * E + e);
        if (TILES) below |= (o < lo ? 1u : 0u) << (j * E + e);
      }
    }
    take &= valid;
    below &= valid;
  };
  auto append = [&](U* out) {
#pragma unroll
    for (int j = 0; j < V; j++) {
#pragma unroll
      for (int e = 0; e < E; e++)
        if ((take >> (j * E + e)) & 1u) *out++ = r[j].k[e];
    }
  };
  if (!TILES) {
    uint32_t have = 0u;  // gathered by the warp
    for (int q = 0; q < steps; q++) {
      const int64_t t0 = (int64_t(blockIdx.x) * steps + q) * T;
      if (t0 >= n) break;  // uniform over the CTA
      read_tile(t0);
      if (!__any_sync(0xFFFFFFFFu, take != 0u)) continue;
      const uint32_t c = uint32_t(__popc(take));
      uint32_t incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
      }
      const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
      if (have + total <= uint32_t(CAP)) {
        append(&s_k[warp][have + incl - c]);
        have += total;
      } else {  // more than the buffer holds: these go to the global range at once
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(counter, (unsigned long long)total);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        append(cand + base + (incl - c));
      }
    }
    if (lane == 0) s_n[warp] = have;
    if (!__syncthreads_or(have != 0u)) return;
    const uint32_t all = __reduce_add_sync(0xFFFFFFFFu, lane < NW ? s_n[lane] : 0u);
    const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? s_n[lane] : 0u);
    if (tid == 0) s_base = atomicAdd(counter, (unsigned long long)all);
    __syncthreads();
    U* out = cand + s_base + before;
    for (uint32_t i = uint32_t(lane); i < have; i += 32) out[i] = s_k[warp][i];
    return;
  }
  read_tile(int64_t(blockIdx.x) * T);
  __syncthreads();  // the counters are zero
  uint32_t slot = 0u;
  if (take) slot = atomicAdd(&s_count, uint32_t(__popc(take)));
  const uint32_t b = __reduce_add_sync(0xFFFFFFFFu, uint32_t(__popc(below)));
  if (lane == 0 && b) atomicAdd(&s_below, b);
  __syncthreads();
  const uint32_t count = s_count;
  if (tid == 0) {
    unsigned long long base = 0;
    if (count) base = atomicAdd(counter, (unsigned long long)count);
    s_base = base;
    if (tiles) tiles[blockIdx.x] = {uint32_t(base), count, s_below};
    if (s_below) atomicAdd(&st->below, (unsigned long long)s_below);
  }
  if (count == 0u) return;  // uniform over the CTA
  __syncthreads();
  append(cand + s_base + slot);
}

// ---- stable three-way partition around the selected key -----------------------------
// Three launches over the window read's tiles: the tiles' class counts, one CTA's scan of them into
// output starts, and the scatter.
constexpr int PART_NT = WIN_NT;

template <class U, int KIND>
__device__ __forceinline__ int part_class(U k, U v_ordered) {
  const U o = KeyOrder<U, KIND>::to_ordered(k);
  return o < v_ordered ? 0 : (o == v_ordered ? 1 : 2);
}

// A warp per tile: counts[tile] = {keys < v, keys == v}, from the keys below the window and the tile's
// candidates (a few percent of the keys), or from the keys themselves when the window missed.
template <class U, int KIND>
__global__ void __launch_bounds__(256) partition_count_kernel(const U* keys, int64_t n,
                                                              const U* cand, const SelectState* st,
                                                              const WinTile* tiles, int64_t ntiles,
                                                              uint2* counts) {
  constexpr int T = win_tile<U>();
  chain_wait();
  chain_release();
  const U v = U(st->prefix);
  const int lane = threadIdx.x & 31;
  const int64_t t = (int64_t(blockIdx.x) * 256 + threadIdx.x) >> 5;
  if (t >= ntiles) return;  // warp-uniform
  const bool among = st->mode == SelMode<U>::CAND;
  const WinTile w = tiles[t];
  const U* src = among ? cand + w.base : keys + t * T;
  const int m = among ? int(w.count) : int(n - t * T < T ? n - t * T : T);
  uint32_t l = 0, e = 0;
#pragma unroll 4
  for (int i = lane; i < m; i += 32) {
    const int cl = part_class<U, KIND>(src[i], v);
    l += cl == 0;
    e += cl == 1;
  }
  l = __reduce_add_sync(0xFFFFFFFFu, l);
  e = __reduce_add_sync(0xFFFFFFFFu, e);
  if (lane == 0) counts[t] = make_uint2(l + (among ? w.below : 0u), e);
}

// One CTA: counts[] into exclusive starts, each thread a run of consecutive tiles.
static __global__ void __launch_bounds__(1024) partition_scan_kernel(uint2* counts, int64_t ntiles) {
  __shared__ uint32_t s_w[2][32];
  chain_wait();
  chain_release();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t per = (ntiles + 1023) / 1024;
  const int64_t t0 = tid * per, t1 = t0 + per < ntiles ? t0 + per : ntiles;
  uint32_t sum[2] = {0u, 0u};
#pragma unroll 8
  for (int64_t t = t0; t < t1; t++) {
    const uint2 c = counts[t];
    sum[0] += c.x;
    sum[1] += c.y;
  }
  uint32_t incl[2] = {sum[0], sum[1]};
#pragma unroll
  for (int q = 0; q < 2; q++) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl[q], o);
      if (lane >= o) incl[q] += y;
    }
    if (lane == 31) s_w[q][warp] = incl[q];
  }
  __syncthreads();
  uint32_t run[2];
#pragma unroll
  for (int q = 0; q < 2; q++) run[q] = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? s_w[q][lane] : 0u) + incl[q] - sum[q];
#pragma unroll 8
  for (int64_t t = t0; t < t1; t++) {
    const uint2 c = counts[t];
    counts[t] = make_uint2(run[0], run[1]);
    run[0] += c.x;
    run[1] += c.y;
  }
}

// A tile per CTA, a row of 32 consecutive keys per warp load: warp w holds keys [w * 32 * KPT, ...) of
// the tile, row j at + j * 32.  A key's stable slot among its class comes from the class ballots of its
// row, the rows before it and the warps before it.  Rows are written straight from the registers: a row
// is at most three runs, and the sectors that neighbouring rows share meet in L2.  (Staging a warp's
// keys in class order in shared memory first took more instructions than the fewer sectors saved: 33 M
// f32 keys 70 us.)
template <class U, int KIND>
__global__ void __launch_bounds__(PART_NT, 3) partition_scatter_kernel(const U* keys, int64_t n,
                                                                    const SelectState* st,
                                                                    const uint2* starts,
                                                                    U* out) {
  constexpr int T = win_tile<U>(), KPT = T / PART_NT, SUB = 32 * KPT, NW = PART_NT / 32;
  __shared__ uint32_t s_c[2][NW];
  chain_wait();
  chain_release();
  const U v = U(st->prefix);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tile = blockIdx.x;
  const int64_t base = tile * T + warp * SUB;
  const int sub_n = int(n - base < SUB ? (n - base < 0 ? 0 : n - base) : SUB);
  const U* kin = keys + base;
  U k[KPT];
  uint32_t cls = 0u;  // two bits per key
  uint32_t c0 = 0, c1 = 0;
  if (sub_n == SUB) {  // warp-uniform: full rows need no bounds
#pragma unroll
    for (int j = 0; j < KPT; j++) k[j] = kin[j * 32 + lane];
#pragma unroll
    for (int j = 0; j < KPT; j++) cls |= uint32_t(part_class<U, KIND>(k[j], v)) << (2 * j);
  } else {
#pragma unroll
    for (int j = 0; j < KPT; j++) {
      const int i = j * 32 + lane;
      k[j] = i < sub_n ? kin[i] : U(0);
      cls |= (i < sub_n ? uint32_t(part_class<U, KIND>(k[j], v)) : 3u) << (2 * j);
    }
  }
  // two bits per key: 00 below v, 01 equal, 10 above, 11 none
  c0 = __reduce_add_sync(0xFFFFFFFFu, uint32_t(__popc(~(cls | (cls >> 1)) & (0x55555555u >> (32 - 2 * KPT)))));
  c1 = __reduce_add_sync(0xFFFFFFFFu, uint32_t(__popc(cls & ~(cls >> 1) & 0x55555555u)));
  if (lane == 0) {
    s_c[0][warp] = c0;
    s_c[1][warp] = c1;
  }
  const uint2 start = starts[tile];
  __syncthreads();
  // keys of class 0 and 1 in the warps before
  const uint32_t b0 = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? s_c[0][lane] : 0u);
  const uint32_t b1 = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? s_c[1][lane] : 0u);
  // the next output position of each class (uniform over the warp); positions fit 32 bits (n < 2^31).
  // Class 2 starts behind the others and, of the keys before this warp, behind none but its own.
  const uint32_t less = uint32_t(st->less), eq = uint32_t(st->eq);
  const uint32_t before = uint32_t(tile) * uint32_t(T) + uint32_t(warp * SUB);  // keys before this warp's
  uint32_t p0 = start.x + b0, p1 = start.y + b1;
  uint32_t p2 = less + eq + (before - p0 - p1);
  p1 += less;
  const uint32_t lt = lanemask_lt();
  const uint32_t n32 = uint32_t(n);
#pragma unroll
  for (int j = 0; j < KPT; j++) {
    const uint32_t c = (cls >> (2 * j)) & 3u;
    const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, c == 0u);
    const uint32_t m1 = __ballot_sync(0xFFFFFFFFu, c == 1u);
    const uint32_t m2 = __ballot_sync(0xFFFFFFFFu, c == 2u);
    const uint32_t mine = c == 0u ? m0 : (c == 1u ? m1 : m2);
    const uint32_t pos = (c == 0u ? p0 : (c == 1u ? p1 : p2)) + __popc(mine & lt);
    if (c < 3u && pos < n32) out[pos] = k[j];
    p0 += __popc(m0);
    p1 += __popc(m1);
    p2 += __popc(m2);
  }
}

// ---- the k largest: keys > v compacted, then copies of v ------------------------------
// The keys above the level-0 bin are already in out (select_compact_kernel); this appends the
// candidates > v (the level-0 bin's keys) and fills the rest with copies of v.
template <class U, int KIND>
__global__ void __launch_bounds__(SEL_NT, SEL_CTAS_PER_SM) topk_gather_kernel(const U* cand, int64_t k,
                                                             SelectState* st, U* out) {
  using KO = KeyOrder<U, KIND>;
  constexpr int E = int(16 / sizeof(U));
  chain_wait();
  chain_release();
  const U v = U(st->prefix);
  const int64_t n = st->n_total;
  int64_t greater = n - st->less - st->eq;
  greater = greater < 0 ? 0 : greater;  // never index below out[0]
  visit_keys<U, SEL_VPT>(cand, st->cand_count, gridDim.x, [&](const U* kk, int nv) {
    uint32_t take = 0u;
#pragma unroll
    for (int e = 0; e < E; e++)
      if (e < nv && KO::to_ordered(kk[e]) > v) take |= 1u << e;
    warp_append<U, E>(kk, take, out, &st->gathered, k);
  });
  // copies of the selected key fill the rest (greater <= k by construction)
  const U vraw = KO::from_ordered(v);
  const int64_t stride = int64_t(gridDim.x) * SEL_NT;
  const int64_t gtid = int64_t(blockIdx.x) * SEL_NT + threadIdx.x;
  for (int64_t j = greater + gtid; j < k; j += stride) out[j] = vraw;
}

// ---- sort of a small top-k output in one CTA ------------------------------------------
// The k <= topk_small_sort_max<U>() outputs are sorted ascending by their ordered value in shared
// memory (a bitonic network over the next power of two, padded with the largest ordered value,
// so the padding sorts behind every key and only the first k slots are written back; longer outputs
// go through the one-launch small sort, which takes 7.3 us for 1000 keys, this network 10.8).  Keys
// with equal ordered values have equal bits, so the bytes equal the LSD sort's.
template <class U>
__host__ __device__ constexpr int topk_small_sort_max() {
  return 256;
}
constexpr int TOPK_SMALL_SORT_NT = 128;

template <class U, int KIND>
__global__ void __launch_bounds__(TOPK_SMALL_SORT_NT) topk_small_sort_kernel(U* out, int k) {
  using KO = KeyOrder<U, KIND>;
  __shared__ U s[topk_small_sort_max<U>()];
  chain_wait();
  if (k <= 1) return;
  int N = 2;
  while (N < k) N <<= 1;
  for (int i = threadIdx.x; i < N; i += TOPK_SMALL_SORT_NT) s[i] = i < k ? KO::to_ordered(out[i]) : U(~U(0));
  __syncthreads();
  for (int size = 2; size <= N; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int p = threadIdx.x; p < (N >> 1); p += TOPK_SMALL_SORT_NT) {
        const int i = ((p & ~(stride - 1)) << 1) | (p & (stride - 1));  // lower element of the pair
        const int j = i + stride;
        const bool up = (i & size) == 0;
        const U a = s[i], b = s[j];
        if ((a > b) == up) {
          s[i] = b;
          s[j] = a;
        }
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < k; i += TOPK_SMALL_SORT_NT) out[i] = KO::from_ordered(s[i]);
}

}  // namespace hpcs
