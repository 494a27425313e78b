// One LSD digit pass in a single sweep over the keys (sm_100a).
//
// Persistent CTAs take tiles of TILE = NT x KPT keys in order from a counter; the first ticket makes
// its CTA the scanner, ticket t + 1 is tile t.  Per tile t a sorting CTA
//   rank     loads the staged keys (and items) into registers, warp-striped, and ranks each key
//            among its warp's keys of the same digit (one ordered shared atomic per key, or the
//            peer-mask ranking): stable within the warp;
//   scan     turns the per-warp digit counters into tile offsets and publishes the tile's digit
//            totals in its row of totals[];
//   reorder  stores the keys (and items) into shared memory in (digit, input order) order;
//   scatter  writes tile t - 1, reordered one iteration ago, as coalesced per-digit runs, its global
//            bases read from its row of bases[].
// The scanner follows the rows of totals[] as they are published, one thread per digit, and
// publishes every tile's global base per digit: the bin start plus the totals of all tiles before,
// the bin-major / quantum-minor offsets of RadixSortLsdParallel.cs:49-94 with one quantum per tile.
//
// Why this shape.  A key costs three random shared-memory accesses (the ranking atomic, the offset
// lookup, the reorder store; ~4 clocks per warp instruction each), so the shared-memory pipe bounds
// a pass near 0.5 ms per 2^28 4-byte keys.  A decoupled look-back, where every tile adds up its
// predecessors' totals itself, reads ~40 rows per tile at 148 tiles in flight and its chain kept the
// CTAs waiting (27 clocks per 32 keys); one scanner reads each row once, 32 rows in flight, and its
// ~2 us of latency pass while the tile is reordered and the next one ranked.  Tiles are taken in
// order by CTAs that run, and the scanner is the first CTA to run, so every wait is for a running
// CTA, whatever part of the grid is resident (a lone scanner waits for the others to be scheduled).
//
// Row words.  totals[]: the tag of the executed pass (1, 2, ...) in the upper half, the count (at most
// TILE) below; bases[]: the base (n < 2^31) under a flag bit that alternates between executed passes.
// Both are zero before the first pass, so no pass clears them.
#pragma once
#include "radix_kernels.cuh"

namespace hpcs {

// Rows of totals per scanner step.
#ifndef HPCS_LB_ROWS
#define HPCS_LB_ROWS 32
#endif
constexpr int LB_ROWS = HPCS_LB_ROWS;
static_assert(LB_ROWS <= 32, "a mask of rows");
// A scanner without any tile to wait for gives up after this many wait limits.
constexpr uint64_t LB_IDLE_LIMITS = 64;

template <class U, class V, int NT, int KPT, int MODE>
struct LookbackSmem {
  static constexpr bool PAIRS = !std::is_same<V, NoValue>::value;
  static constexpr int TILE = NT * KPT;
  static constexpr int NW = NT / 32;
  static constexpr int G = NT / RADIX;        // threads per digit in the digit scan
  static constexpr int NWG = NW / G;          // warps summed by each of them
  static constexpr int RS = RADIX + 32 / NW;  // warp-counter row stride: conflict-free scan
  static constexpr size_t KEYS_BYTES = size_t(TILE) * sizeof(U);
  static constexpr size_t VALS_BYTES = PAIRS ? size_t(TILE) * 4 : 0;
  static constexpr size_t BUF_BYTES = KEYS_BYTES + VALS_BYTES;
  static constexpr size_t OFF_STAGE = 0;  // bulk-copy stage
  static constexpr size_t OFF_REORDER = OFF_STAGE + BUF_BYTES;
  static constexpr size_t OFF_CNT = OFF_REORDER + BUF_BYTES;  // [NW][RS]
  // the offsets looked up in the reorder, 16 bits each: two digits share a word, which costs a
  // random warp access fewer bank conflicts than 32-bit offsets; row stride as for the counters
  static constexpr int OS = RADIX + 2;
  static constexpr size_t OFF_OFFSETS = OFF_CNT + size_t(NW) * RS * 4;  // [NW][OS]
  static constexpr size_t OFF_MSK = (OFF_OFFSETS + size_t(NW) * OS * 2 + 15) / 16 * 16;
  static constexpr size_t MSK_BYTES = MODE == RANK_PEER_MASK ? size_t(NW) * 2 * RADIX * 4 : 0;
  static constexpr size_t OFF_GBASE = (OFF_MSK + MSK_BYTES + 15) / 16 * 16;  // [256] global base - local start
  static constexpr size_t OFF_WSUM = OFF_GBASE + RADIX * 4;
  static constexpr size_t OFF_TILE = OFF_WSUM + 32 * 4;  // tile id of the next iteration
  static constexpr size_t OFF_MBAR = (OFF_TILE + 4 + 7) / 8 * 8;
  static constexpr size_t BYTES = OFF_MBAR + 8;
  static_assert(G >= 1 && (G & (G - 1)) == 0 && NW % G == 0 && 32 % NW == 0, "digit-scan geometry");
  static_assert(TILE < 65536, "tile counts and positions are kept in 16 bits");
};

// The scanner: thread d < 256 of the CTA for digit d, each warp at its own pace.
template <class Dummy = void>
__device__ __forceinline__ void scan_totals(const SortArgs& args, SortPlan* plan, int x) {
  const int d = threadIdx.x, lane = d & 31;
  if (d >= RADIX) return;
  const int rows = args.num_tiles;
  const uint32_t tag = uint32_t(x + 1) << 16;
  const uint32_t flag = (x & 1) ? 0u : 0x80000000u;
  const uint32_t* tin = args.status[0] + d;
  uint32_t* bout = args.status[1] + d;
  uint32_t base = plan->bin_start[args.pass][d] | flag;  // (the sums stay below 2^31)
  auto load = [&](uint32_t(&v)[LB_ROWS], int row) {
    const uint32_t* p = tin + int64_t(row) * RADIX;
    if (row + LB_ROWS <= rows) {
#pragma unroll
      for (int i = 0; i < LB_ROWS; i++) v[i] = ld_relaxed_gpu(p + i * RADIX);
    } else {
#pragma unroll
      for (int i = 0; i < LB_ROWS; i++) v[i] = row + i < rows ? ld_relaxed_gpu(p + i * RADIX) : 0u;
    }
  };
  // publishes the bases of the rows from `row` whose totals are there; their number
  auto consume = [&](const uint32_t(&v)[LB_ROWS], int row) -> int {
    uint32_t* p = bout + int64_t(row) * RADIX;
    uint32_t miss = 0u;
#pragma unroll
    for (int i = 0; i < LB_ROWS; i++) miss |= v[i] ^ tag;
    if (__all_sync(0xFFFFFFFFu, (miss >> 16) == 0u)) {
#pragma unroll
      for (int i = 0; i < LB_ROWS; i++) {
        st_relaxed_gpu(p + i * RADIX, base);
        base += v[i] - tag;
      }
      return LB_ROWS;
    }
    uint32_t there = 0u;
#pragma unroll
    for (int i = 0; i < LB_ROWS; i++) there |= ((v[i] ^ tag) < 0x10000u ? 1u : 0u) << i;
    const int c = __ffs(~__reduce_and_sync(0xFFFFFFFFu, there)) - 1;  // (some row is missing)
#pragma unroll
    for (int i = 0; i < LB_ROWS; i++) {
      if (i < c) {
        st_relaxed_gpu(p + i * RADIX, base);
        base += v[i] - tag;
      }
    }
    return c;
  };
  // nothing new at `row`: false once the wait ran out.  The limit counts while some tile is out;
  // before that the other CTAs are not scheduled yet.
  uint64_t idle_since = 0, since = 0;
  auto keep_waiting = [&](int row) -> bool {
    bool go = true;
    if (lane == 0) {
      const uint64_t now = global_timer_ns();
      if (idle_since == 0) idle_since = now;
      if (int(ld_volatile(&plan->tile_counter[args.pass])) - 1 <= row) since = 0;
      else if (since == 0) since = now;
      const bool late = (since != 0 && now - since > args.spin_limit_ns) ||
                        now - idle_since > LB_IDLE_LIMITS * args.spin_limit_ns;
      if (late) atomicOr(&plan->error, uint32_t(DERR_LOOKBACK_TIMEOUT));
      go = !late && ld_volatile(&plan->error) == 0u;
    }
    return __any_sync(0xFFFFFFFFu, lane == 0 && go);
  };
  // One step of rows at a time where the totals just come in; two steps in flight while the scanner
  // is behind (whole steps are there at once).
  uint32_t a[LB_ROWS], b[LB_ROWS];
  int row = 0;
  uint32_t idle = 0;                    // reads without anything new
  bool loaded = false, behind = false;  // a[] holds the rows from `row`; the last step was whole
  for (;;) {
    if (!loaded) load(a, row);
    if (behind) load(b, row + LB_ROWS);
    int c = consume(a, row);
    row += c;
    bool whole = c == LB_ROWS;
    loaded = false;
    if (whole && behind) {
      load(a, row + LB_ROWS);
      c = consume(b, row);
      row += c;
      loaded = whole = c == LB_ROWS;
    }
    behind = whole;
    if (row >= rows) return;
    if (c > 0) {
      idle_since = since = 0;
      idle = 0;
    } else if (++idle % 32u == 0u && !keep_waiting(row)) {
      return;
    }
  }
}

template <class U, int KIND, class V, int NT, int KPT, int MODE, int BATCH>
__global__ void __launch_bounds__(NT, 1) lookback_pass_kernel(SortArgs args) {
  using L = LookbackSmem<U, V, NT, KPT, MODE>;
  constexpr bool PAIRS = L::PAIRS;
  constexpr int TILE = L::TILE;
  constexpr int G = L::G, NWG = L::NWG, RS = L::RS;

  chain_wait();
  chain_release();
  SortPlan* plan = args.plan;
  const int pass = args.pass;
  const int sel = plan->src_sel[pass];
  if (sel < 0) return;  // every key has the same digit here: the pass is the identity (uniform)
  const int shift = 8 * pass;
  const int x = plan->exec_idx[pass];
  const uint32_t tag = uint32_t(x + 1) << 16;
  const uint32_t flag = (x & 1) ? 0u : 0x80000000u;
  uint32_t* err = &plan->error;
  const int64_t n = args.n;
  const int num_tiles = args.num_tiles;

  extern __shared__ __align__(128) unsigned char smem[];
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + L::OFF_CNT);
  uint32_t* s_gbase = reinterpret_cast<uint32_t*>(smem + L::OFF_GBASE);
  uint32_t* s_wsum = reinterpret_cast<uint32_t*>(smem + L::OFF_WSUM);
  volatile int* s_tile = reinterpret_cast<volatile int*>(smem + L::OFF_TILE);
  uint64_t* s_mbar = reinterpret_cast<uint64_t*>(smem + L::OFF_MBAR);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const U* kin = static_cast<const U*>(sel ? args.keys_b : args.keys_a);
  U* kout = static_cast<U*>(sel ? args.keys_a : args.keys_b);
  const uint32_t* vin = static_cast<const uint32_t*>(sel ? args.vals_b : args.vals_a);
  uint32_t* vout = static_cast<uint32_t*>(sel ? args.vals_a : args.vals_b);

  // tickets: a grid of one CTA has one tile and needs no scanner
  const int first = gridDim.x > 1 ? 1 : 0;
  uint32_t ticket = 0u;  // thread 0: taken one iteration before its tile's copy is issued
  // thread 0: the ticket's tile becomes the next iteration's and is copied into the stage buffer
  auto feed = [&]() {
    const int t = int(ticket) - first;
    *s_tile = t;
    if (t >= 0 && t < num_tiles) {
      stage_tile<U, PAIRS, TILE>(smem + L::OFF_STAGE, L::KEYS_BYTES, s_mbar, kin, vin, n, t);
      ticket = atomicAdd(&plan->tile_counter[pass], 1u);  // (first used an iteration from now)
    }
  };
  if (tid == 0) {
    mbar_init(s_mbar, 1);
    fence_mbar_init();
    ticket = atomicAdd(&plan->tile_counter[pass], 1u);
    feed();
  }
  __syncthreads();
  int u = *s_tile;
  if (u < 0) {
    scan_totals(args, plan, x);
    return;
  }

  uint32_t* cnt_w = s_cnt + warp * RS;
  uint16_t* s_off = reinterpret_cast<uint16_t*>(smem + L::OFF_OFFSETS);
  const uint16_t* off_w = s_off + warp * L::OS;
  uint32_t* msk_w = reinterpret_cast<uint32_t*>(smem + L::OFF_MSK) + warp * 2 * RADIX;
  if (MODE == RANK_PEER_MASK)
    for (int i = lane; i < 2 * RADIX; i += 32) msk_w[i] = 0u;
  const uint32_t n32 = uint32_t(n);
  const Digit<U, KIND> dig(shift);
  // This pass's two most frequent values hold much of the keys: they rank by votes (ordered-atomic
  // mode only).
  const bool grouped = MODE == RANK_ORDERED_ATOMIC && plan->grouped[pass] != 0;
  const uint32_t heavy = uint32_t(plan->heavy[pass]), heavy2 = uint32_t(plan->heavy2[pass]);
  const int sd = tid / G, sq = tid % G;  // the digit and warp group this thread scans
  const int wbase = warp * 32 * KPT;
  bool out_of_range = false;

  auto trace_row = [&](int t) -> uint64_t* {
    return args.trace && pass == args.trace_pass && tid == 0 && t < args.trace_capacity
               ? args.trace + int64_t(t) * TRACE_WORDS
               : nullptr;
  };
  // The base of digit sd in tile t (threads with sq == 0): requested early, waited for (bounded) when
  // needed.
  const uint32_t* bases = args.status[1];
  auto request_base = [&](int t) -> uint32_t {
    if (sq != 0) return 0u;
    return first ? ld_relaxed_gpu(bases + int64_t(t) * RADIX + sd) : (plan->bin_start[pass][sd] | flag);
  };
  auto await_base = [&](int t, uint32_t w) -> uint32_t {
    if (sq != 0) return 0u;
    uint64_t t0 = 0;
    for (uint32_t polls = 0; (w & 0x80000000u) != flag; polls++) {
      w = atomicOr(args.status[1] + int64_t(t) * RADIX + sd, 0u);
      if (polls % 32u != 31u) continue;  // the error word and the time are looked at now and then
      const uint64_t now = global_timer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > args.spin_limit_ns) atomicOr(err, uint32_t(DERR_LOOKBACK_TIMEOUT));
      if (ld_volatile(err) != 0u) break;
    }
    return w & 0x7FFFFFFFu;
  };

  U* rk = reinterpret_cast<U*>(smem + L::OFF_REORDER);  // the reordered tile
  uint32_t* rv = reinterpret_cast<uint32_t*>(smem + L::OFF_REORDER + L::KEYS_BYTES);

  // Writes the reordered tile t.  In batches: all of a batch's
  // keys, then all of its bases, then the writes, so that BATCH shared loads are in flight (the
  // compiler may not move a load above a store that could alias it).  Every destination is checked
  // against n: after a wait that ran out the bases are not trusted, and a bad one is recorded.
  auto scatter = [&](auto full_tag, int t) {
    constexpr bool FULL = decltype(full_tag)::value;
    const int tile_n = FULL ? TILE : int(n - int64_t(t) * TILE);
#pragma unroll
    for (int b = 0; b < KPT; b += BATCH) {
      U k[BATCH];
      uint32_t v[PAIRS ? BATCH : 1], pos[BATCH];
#pragma unroll
      for (int i = 0; i < BATCH && b + i < KPT; i++) {
        const int s = (b + i) * NT + tid;
        k[i] = FULL || s < tile_n ? rk[s] : U(0);
        if (PAIRS) v[PAIRS ? i : 0] = FULL || s < tile_n ? rv[s] : 0u;
      }
#pragma unroll
      for (int i = 0; i < BATCH && b + i < KPT; i++) pos[i] = s_gbase[dig(k[i])] + uint32_t((b + i) * NT + tid);
#pragma unroll
      for (int i = 0; i < BATCH && b + i < KPT; i++) {
        if (FULL || (b + i) * NT + tid < tile_n) {
          if (pos[i] < n32) {
            kout[pos[i]] = k[i];
            if (PAIRS) vout[pos[i]] = v[PAIRS ? i : 0];
          } else {
            out_of_range = true;
          }
        }
      }
    }
    if (uint64_t* tr = trace_row(t)) tr[6] = global_timer_ns();
  };

  uint32_t prev_local = 0;  // tile-local start of digit sd in the tile before (sq == 0)

  // Ranks, scans and reorders tile t of iteration it, and writes the tile before it.
  auto tile_body = [&](auto full_tag, int t, int it, int prev) {
    constexpr bool FULL = decltype(full_tag)::value;
    const int64_t tile_base = int64_t(t) * TILE;
    const int tile_n = FULL ? TILE : int(n - tile_base);
    const int bulk_keys = FULL ? TILE : int((int64_t(tile_n) * int64_t(sizeof(U))) & ~int64_t(15)) / int(sizeof(U));
    const int bulk_vals = FULL ? TILE : (PAIRS ? int((int64_t(tile_n) * 4) & ~int64_t(15)) / 4 : 0);
    uint64_t* tr = trace_row(t);
    if (tr) {
      tr[0] = uint64_t(t);
      tr[1] = sm_id();
      tr[2] = global_timer_ns();
    }
    const uint32_t base_word = prev >= 0 ? request_base(prev) : 0u;
    __syncwarp();  // every lane has looked its offsets of the last tile up
    for (int i = lane; i < RADIX; i += 32) cnt_w[i] = 0u;
    if (!mbar_wait_bounded(s_mbar, uint32_t(it & 1), args.spin_limit_ns) && lane == 0)
      atomicOr(err, uint32_t(DERR_TMA_TIMEOUT));
    __syncwarp();
    if (tr) tr[3] = global_timer_ns();

    // ---- load (warp-striped) and rank within the warp --------------------------------
    const U* sk = reinterpret_cast<const U*>(smem + L::OFF_STAGE);
    const uint32_t* sv = reinterpret_cast<const uint32_t*>(smem + L::OFF_STAGE + L::KEYS_BYTES);
    U key[KPT];
    uint32_t val[PAIRS ? KPT : 1];
    uint32_t rank[(KPT + 1) / 2];  // two 16-bit ranks per word
#pragma unroll
    for (int i = 0; i < KPT; i++) {
      const int idx = wbase + i * 32 + lane;
      U k = U(0);
      if (FULL || idx < bulk_keys) k = sk[idx];
      else if (idx < tile_n) k = kin[tile_base + idx];
      key[i] = k;
      if (PAIRS) {
        uint32_t v = 0u;
        if (FULL || idx < bulk_vals) v = sv[idx];
        else if (idx < tile_n) v = vin[tile_base + idx];
        val[PAIRS ? i : 0] = v;
      }
    }
#pragma unroll
    for (int i = 0; i < (KPT + 1) / 2; i++) rank[i] = 0u;
    if (grouped) {
      FrequentRanks fr(heavy, heavy2);
#pragma unroll
      for (int i = 0; i < KPT; i++) {
        const int idx = wbase + i * 32 + lane;
        rank[i / 2] |= fr.rank(cnt_w, dig(key[i]), FULL || idx < tile_n) << (16 * (i & 1));
      }
      fr.close(cnt_w, lane);
    } else {
#pragma unroll
      for (int i = 0; i < KPT; i++) {
        const int idx = wbase + i * 32 + lane;
        rank[i / 2] |= rank_in_warp<MODE>(cnt_w, msk_w, dig(key[i]), FULL || idx < tile_n, i & 1, lane) << (16 * (i & 1));
      }
    }
    fence_proxy_async_smem();  // the stage buffer was read; the next bulk copy overwrites it
    __syncthreads();  // (A) warp counts complete; the stage buffer is free
    if (tid == 0) feed();
    if (tr) tr[4] = global_timer_ns();

    // ---- scan over (digit, warp): tile offsets per warp; publish the digit totals ----
    uint32_t local;
    {
      uint32_t c[NWG];
      uint32_t gsum = 0;
#pragma unroll
      for (int m = 0; m < NWG; m++) {
        c[m] = s_cnt[(sq * NWG + m) * RS + sd];
        gsum += c[m];
      }
      uint32_t qi = gsum;  // inclusive over the digit's warp groups
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, qi, o, G);
        if (sq >= o) qi += y;
      }
      const uint32_t total = __shfl_sync(0xFFFFFFFFu, qi, lane | (G - 1));
      if (sq == 0 && t != args.poison_tile) st_relaxed_gpu(args.status[0] + int64_t(t) * RADIX + sd, tag | total);
      uint32_t di = total;  // inclusive over this warp's digits (lanes G apart)
#pragma unroll
      for (int o = G; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, di, o);
        if (lane >= o) di += y;
      }
      if (lane == 31) s_wsum[warp] = di;
      // only now, with this tile's totals published: no CTA's totals may wait for another's bases
      if (prev >= 0) {
        const uint32_t base = await_base(prev, base_word);
        if (sq == 0) s_gbase[sd] = base - prev_local;
      }
      __syncthreads();  // (B) the warps' digit sums; the bases of `prev`
      local = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? s_wsum[lane] : 0u) + di - total;
      uint32_t run = local + qi - gsum;
#pragma unroll
      for (int m = 0; m < NWG; m++) {
        s_off[(sq * NWG + m) * L::OS + sd] = uint16_t(run);
        run += c[m];
      }
    }
    // tile `prev` was reordered before this iteration's first barrier; it is a full tile (only the
    // last tile of all is short, and the CTA that has it has none after it)
    if (prev >= 0) {
      if (uint64_t* trp = trace_row(prev)) trp[5] = global_timer_ns();
      scatter(std::true_type(), prev);
    }
    __syncthreads();  // (C) offsets ready; `prev` is written

    // ---- reorder the tile in shared memory by digit (a batch's lookups before its stores) ----
#pragma unroll
    for (int b = 0; b < KPT; b += BATCH) {
      uint32_t pos[BATCH];
#pragma unroll
      for (int i = b; i < b + BATCH && i < KPT; i++)
        pos[i - b] = uint32_t(off_w[dig(key[i])]) + ((rank[i / 2] >> (16 * (i & 1))) & 0xFFFFu);
#pragma unroll
      for (int i = b; i < b + BATCH && i < KPT; i++) {
        if (FULL || wbase + i * 32 + lane < tile_n) {
          rk[pos[i - b]] = key[i];
          if (PAIRS) rv[pos[i - b]] = val[PAIRS ? i : 0];
        }
      }
    }
    prev_local = local;
  };

  int prev = -1, it = 0;
  for (; u < num_tiles; it++) {
    if (n - int64_t(u) * TILE >= TILE) tile_body(std::true_type(), u, it, prev);
    else tile_body(std::false_type(), u, it, prev);
    prev = u;
    u = *s_tile;  // written after this iteration's barrier (A), not before the next one's
  }
  if (prev >= 0) {
    const uint32_t base = await_base(prev, request_base(prev));
    if (sq == 0) s_gbase[sd] = base - prev_local;
    __syncthreads();  // bases and the last tile's reordered keys ready
    if (uint64_t* trp = trace_row(prev)) trp[5] = global_timer_ns();
    if (n - int64_t(prev) * TILE >= TILE) scatter(std::true_type(), prev);
    else scatter(std::false_type(), prev);
  }
  if (out_of_range) atomicOr(err, uint32_t(DERR_BOUNDS));
}

}  // namespace hpcs
