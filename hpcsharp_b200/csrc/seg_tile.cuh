// Tiled block-level kernel of the batched segmented sort: one CTA sorts one array that is too long for
// its variant's in-shared-memory kernel, in tiles of NT x KPT keys.
//
// The array is read once to histogram every digit (digit counts do not depend on the order of the
// keys), then each pass runs its tiles in order with running per-digit offsets, ping-pong with the
// array's scratch: one read and one write a pass, mostly in L2.  The next tile is staged by a bulk copy
// while this one is scanned, reordered and written.
//
// What bounds it: the shared-memory pipe, as in the look-back pass (three random accesses per key and
// pass), and the latency of a tile's barriers.  Two shapes: 256 threads x 32 4-byte keys, two CTAs per SM
// hiding each other's barriers (arrays of 8-64 Ki keys: 68 Gkeys/s, 24 with 8-byte keys; the other shape
// 47 and 23), and 512 x 46, one per SM, whose fewer arrays at a time stay in L2 (arrays of 64 Ki-1 Mi
// keys: 64 and 27; the other shape 52 and 21).  The tiled kernels it replaces (serial lookups and stores,
// histogram on shared counters): 48 and 22, 49 and 25.  The histogram's counters are private to groups
// of lanes (1-2 wavefronts per warp atomic instead of ~3.5) and lie in the tile buffers, which are free
// at that time.
#pragma once
#include <cstdint>

#include "radix_kernels.cuh"
#include "segmented.cuh"

namespace hpcs {

template <int NT, int KPT4, int MODE>
struct SegTileSmem {
  static constexpr int NW = NT / 32;
  static constexpr int G = NT / RADIX;
  static constexpr int NWG = NW / G;
  static constexpr int RS = RADIX + 32 / NW;
  static constexpr int OS = RADIX + 2;
  static constexpr size_t BUF_BYTES = size_t(NT) * KPT4 * 4;
  static constexpr size_t OFF_STAGE = 0;
  static constexpr size_t OFF_REORDER = OFF_STAGE + BUF_BYTES;
  static constexpr size_t OFF_CNT = OFF_REORDER + BUF_BYTES;              // [NW][RS]
  static constexpr size_t OFF_OFFSETS = OFF_CNT + size_t(NW) * RS * 4;    // [NW][OS], 16-bit
  static constexpr size_t OFF_MSK = (OFF_OFFSETS + size_t(NW) * OS * 2 + 15) / 16 * 16;
  static constexpr size_t MSK_BYTES = MODE == RANK_PEER_MASK ? size_t(NW) * 2 * RADIX * 4 : 0;
  static constexpr size_t OFF_HIST = OFF_MSK + MSK_BYTES;                 // [8][256]
  static constexpr size_t OFF_RUN = OFF_HIST + 8 * RADIX * 4;             // running start per digit
  static constexpr size_t OFF_GBASE = OFF_RUN + RADIX * 4;
  static constexpr size_t OFF_WSUM = OFF_GBASE + RADIX * 4;
  static constexpr size_t OFF_SEG = OFF_WSUM + 32 * 4;
  static constexpr size_t OFF_MBAR = (OFF_SEG + 4 + 7) / 8 * 8;
  static constexpr size_t BYTES = OFF_MBAR + 8;
  static_assert(NT * KPT4 < 65536, "offsets are kept in 16 bits");
};

// Digit of one pass for a key order known at run time (but for u64 in the wide shape the three orders of one
// key width share their code: an SM runs arrays of several types at once, and six copies of the unrolled loops missed the
// instruction cache, 2 of ~10 stall cycles per instruction).  x ^ top ^ (sign & flip): unsigned keys
// change nothing, signed keys the sign bit, floats the sign bit or, when negative, every bit.
template <class U>
struct RunDigit {
  uint32_t sel, top, flip;
  bool hi_word;
  __device__ __forceinline__ RunDigit(int kind, int shift)
      : sel(0x4440u | uint32_t((shift >> 3) & 3)), hi_word(sizeof(U) == 4 || shift >= 32) {
    top = kind != KIND_UNSIGNED && hi_word ? 0x80000000u : 0u;
    flip = kind == KIND_FLOAT ? (hi_word ? 0x7FFFFFFFu : 0xFFFFFFFFu) : 0u;
  }
  __device__ __forceinline__ uint32_t operator()(U x) const {
    const uint32_t hi = uint32_t(uint64_t(x) >> (sizeof(U) == 8 ? 32 : 0));
    const uint32_t w = hi_word ? hi : uint32_t(x);
    return __byte_perm(w ^ top ^ (uint32_t(int32_t(hi) >> 31) & flip), 0u, sel);
  }
};

// Ranks the tile's keys (key[], warp-striped) by `dig`, scans the counters and stores the keys into the
// reorder buffer in (digit, input order) order; advances the digits' running starts and sets their global
// bases; stages tile `next` (if not negative) of src once this one is in registers.
template <class U, int NT, int KPT4, int MODE>
__device__ __forceinline__ void seg_tile_reorder(const U (&key)[KPT4 * 4 / int(sizeof(U))], int tile_n, const RunDigit<U>& dig,
                                                 unsigned char* smem, const U* src, int64_t n, int next) {
  using L = SegTileSmem<NT, KPT4, MODE>;
  constexpr int KPT = KPT4 * 4 / int(sizeof(U)), TILE = NT * KPT, G = L::G, NWG = L::NWG, RS = L::RS, BATCH = 8;
  U* buf = reinterpret_cast<U*>(smem + L::OFF_REORDER);
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + L::OFF_CNT);
  uint16_t* s_off = reinterpret_cast<uint16_t*>(smem + L::OFF_OFFSETS);
  uint32_t* s_run = reinterpret_cast<uint32_t*>(smem + L::OFF_RUN);
  uint32_t* s_gbase = reinterpret_cast<uint32_t*>(smem + L::OFF_GBASE);
  uint32_t* s_wsum = reinterpret_cast<uint32_t*>(smem + L::OFF_WSUM);
  uint64_t* s_mbar = reinterpret_cast<uint64_t*>(smem + L::OFF_MBAR);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* cnt_w = s_cnt + warp * RS;
  uint32_t* msk_w = reinterpret_cast<uint32_t*>(smem + L::OFF_MSK) + warp * 2 * RADIX;
  const uint16_t* off_w = s_off + warp * L::OS;
  const int sd = tid / G, sq = tid % G;  // the digit and warp group this thread scans
  const int wbase = warp * 32 * KPT;
  uint32_t total, local;
  uint32_t rank[(KPT + 1) / 2];  // two 16-bit ranks per word
#pragma unroll
  for (int i = 0; i < (KPT + 1) / 2; i++) rank[i] = 0u;
#pragma unroll
  for (int i = 0; i < KPT; i++)
    rank[i / 2] |= rank_in_warp<MODE>(cnt_w, msk_w, dig(key[i]), wbase + i * 32 + lane < tile_n, i & 1, lane) << (16 * (i & 1));
  __syncthreads();  // warp counts complete; the tile is in registers
  if (next >= 0 && tid == 0) stage_tile<U, false, TILE>(smem + L::OFF_STAGE, 0, s_mbar, src, nullptr, n, next);
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
    total = __shfl_sync(0xFFFFFFFFu, qi, lane | (G - 1));
    uint32_t di = total;  // inclusive over this warp's digits (lanes G apart)
#pragma unroll
    for (int o = G; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, di, o);
      if (lane >= o) di += y;
    }
    if (lane == 31) s_wsum[warp] = di;
    __syncthreads();
    local = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? s_wsum[lane] : 0u) + di - total;
    uint32_t run = local + qi - gsum;
#pragma unroll
    for (int m = 0; m < NWG; m++) {
      s_off[(sq * NWG + m) * L::OS + sd] = uint16_t(run);
      run += c[m];
    }
    if (sq == 0) {
      const uint32_t r = s_run[sd];
      s_gbase[sd] = r - local;
      s_run[sd] = r + total;
    }
  }
  __syncthreads();  // offsets (and bases) ready; the counters are read
#pragma unroll
  for (int b = 0; b < KPT; b += BATCH) {
    uint32_t pos[BATCH];
#pragma unroll
    for (int i = b; i < b + BATCH && i < KPT; i++)
      pos[i - b] = uint32_t(off_w[dig(key[i])]) + ((rank[i / 2] >> (16 * (i & 1))) & 0xFFFFu);
#pragma unroll
    for (int i = b; i < b + BATCH && i < KPT; i++)
      if (wbase + i * 32 + lane < tile_n) buf[pos[i - b]] = key[i];
  }
  __syncwarp();
  for (int i = lane; i < RADIX; i += 32) cnt_w[i] = 0u;  // for the next tile or pass
  __syncthreads();  // the reordered tile is in place
}

// One array.  `phase` is the stage barrier's expected parity, carried from
// array to array.
template <class U, int NT, int KPT4, int MODE>
__device__ __forceinline__ void seg_tile_sort(U* keys, U* scratch, int64_t n, int kind, unsigned char* smem,
                                              uint32_t* err, uint64_t spin_limit_ns, uint32_t& phase) {
  using L = SegTileSmem<NT, KPT4, MODE>;
  constexpr int KPT = KPT4 * 4 / int(sizeof(U)), TILE = NT * KPT, P = int(sizeof(U));
  constexpr int BATCH = 8;
  U* stage = reinterpret_cast<U*>(smem + L::OFF_STAGE);
  U* buf = reinterpret_cast<U*>(smem + L::OFF_REORDER);
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + L::OFF_CNT);
  uint32_t* s_hist = reinterpret_cast<uint32_t*>(smem + L::OFF_HIST);
  uint32_t* s_run = reinterpret_cast<uint32_t*>(smem + L::OFF_RUN);
  uint32_t* s_gbase = reinterpret_cast<uint32_t*>(smem + L::OFF_GBASE);
  uint32_t* s_wsum = reinterpret_cast<uint32_t*>(smem + L::OFF_WSUM);
  uint64_t* s_mbar = reinterpret_cast<uint64_t*>(smem + L::OFF_MBAR);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* cnt_w = s_cnt + warp * L::RS;
  const int wbase = warp * 32 * KPT;

  for (int i = lane; i < RADIX; i += 32) cnt_w[i] = 0u;
  __syncwarp();

  // ---- all digits' histograms, lane-private counters in the tile buffers -----------------
  constexpr int FIT = int(2 * L::BUF_BYTES / (size_t(P) * RADIX * 4));
  constexpr int COPIES = FIT >= 32 ? 32 : FIT >= 16 ? 16 : 8;
  static_assert(FIT >= 8, "the private histograms fit the tile buffers");
  uint32_t* priv = reinterpret_cast<uint32_t*>(smem + L::OFF_STAGE);  // [P][256][COPIES]
  for (int i = tid; i < P * RADIX * COPIES; i += NT) priv[i] = 0u;
  __syncthreads();
  const bool aligned = (reinterpret_cast<uintptr_t>(keys) & 15) == 0;
  {
    const int copy = lane & (COPIES - 1);
    // the ordered bits at once: x ^ top ^ (sign & flip), as in RunDigit
    const U top = kind != KIND_UNSIGNED ? U(1) << (8 * P - 1) : U(0);
    const U flip = kind == KIND_FLOAT ? U(~U(0)) >> 1 : U(0);
    auto count = [&](U x) {
      const U o = x ^ top ^ ((U(0) - (x >> (8 * P - 1))) & flip);
#pragma unroll
      for (int d = 0; d < P; d++) atomicAdd(&priv[(d * RADIX + (uint32_t(o >> (8 * d)) & 0xFFu)) * COPIES + copy], 1u);
    };
    constexpr int E = 16 / P, VIF = 4;  // 16-byte vectors in flight per thread
    int64_t done = 0;
    if (aligned) {
      const int64_t nvec = n / E;
      const uint4* v = reinterpret_cast<const uint4*>(keys);
      for (int64_t b = 0; b < nvec; b += VIF * NT) {
        union {
          uint4 v;
          U k[E];
        } r[VIF];
#pragma unroll
        for (int j = 0; j < VIF; j++) {
          const int64_t i = b + j * NT + tid;
          if (i < nvec) r[j].v = v[i];
        }
#pragma unroll
        for (int j = 0; j < VIF; j++) {
          if (b + j * NT + tid < nvec) {
#pragma unroll
            for (int e = 0; e < E; e++) count(r[j].k[e]);
          }
        }
      }
      done = nvec * E;
    }
#pragma unroll 1
    for (int64_t i = done + tid; i < n; i += NT) count(keys[i]);
  }
  __syncthreads();
  for (int j = tid; j < P * RADIX; j += NT) {
    uint32_t c = 0;
#pragma unroll 8
    for (int q = 0; q < COPIES; q++) c += priv[j * COPIES + ((q + lane) & (COPIES - 1))];
    s_hist[j] = c;
  }
  fence_proxy_async_smem();  // the stage buffer was used through the generic proxy
  __syncthreads();

  const int ntiles = int((n + TILE - 1) / TILE);
  U* src = keys;
  U* dst = scratch;
  const uint32_t n32 = uint32_t(n);
  bool bad = false;
  for (int p = 0; p < P; p++) {
    // digit starts; a pass whose keys all share one digit is the identity
    uint32_t c = 0, incl = 0;
    if (tid < RADIX) {
      c = s_hist[p * RADIX + tid];
      incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) s_wsum[warp] = incl;
    }
    const bool trivial = __syncthreads_or(tid < RADIX && int64_t(c) == n) != 0;
    if (trivial) continue;
    if (tid < RADIX) s_run[tid] = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? s_wsum[lane] : 0u) + incl - c;
    const RunDigit<U> dig(kind, 8 * p);
    const bool staged = aligned || src == scratch;  // (scratch is aligned)
    // In the wide shape, alone on its SM, a pass's first tile is loaded directly, the second staged meanwhile;
    // the narrow shape's other CTA covers that wait (whole batches 0.4% faster staged).
    constexpr int FIRST = NT == 512 ? 1 : 0;  // the first tile that is staged
    if (staged && ntiles > FIRST && tid == 0) stage_tile<U, false, TILE>(smem + L::OFF_STAGE, 0, s_mbar, src, nullptr, n, FIRST);
    __syncthreads();  // running starts ready; s_wsum may be rewritten
    for (int t = 0; t < ntiles; t++) {
      const int64_t tb = int64_t(t) * TILE;
      const int tile_n = int(n - tb < TILE ? n - tb : TILE);
      U key[KPT];
      const bool bulked = staged && t >= FIRST;
      if (bulked) {
        if (!mbar_wait_bounded(s_mbar, phase, spin_limit_ns) && lane == 0) atomicOr(err, uint32_t(DERR_TMA_TIMEOUT));
        phase ^= 1u;
      }
      const int bulk = bulked ? int((int64_t(tile_n) * int64_t(sizeof(U))) & ~int64_t(15)) / int(sizeof(U)) : 0;
#pragma unroll
      for (int i = 0; i < KPT; i++) {
        const int idx = wbase + i * 32 + lane;
        key[i] = idx < bulk ? stage[idx] : (idx < tile_n ? src[tb + idx] : U(0));
      }
      fence_proxy_async_smem();  // the stage buffer was read; the next bulk copy overwrites it
      seg_tile_reorder<U, NT, KPT4, MODE>(key, tile_n, dig, smem, src, n, bulked && t + 1 < ntiles ? t + 1 : -1);
      // ---- coalesced per-digit runs; every destination is checked against n ------------------
#pragma unroll
      for (int b = 0; b < KPT; b += BATCH) {
        U k[BATCH];
        uint32_t pos[BATCH];
#pragma unroll
        for (int i = 0; i < BATCH && b + i < KPT; i++) {
          const int s = (b + i) * NT + tid;
          k[i] = s < tile_n ? buf[s] : U(0);
        }
#pragma unroll
        for (int i = 0; i < BATCH && b + i < KPT; i++) pos[i] = s_gbase[dig(k[i])] + uint32_t((b + i) * NT + tid);
#pragma unroll
        for (int i = 0; i < BATCH && b + i < KPT; i++) {
          if ((b + i) * NT + tid < tile_n) {
            if (pos[i] < n32) dst[pos[i]] = k[i];
            else bad = true;
          }
        }
      }
      // (no barrier: the next tile's bases and reorder come after two of its own)
    }
    // the next pass's bulk copies read what this pass wrote through the generic proxy
    asm volatile("fence.proxy.async.global;" ::: "memory");
    __syncthreads();
    U* tmp = src;
    src = dst;
    dst = tmp;
  }
  if (bad) atomicOr(err, uint32_t(DERR_BOUNDS));
  // an odd number of executed passes leaves the result in scratch
  if (src != keys)
    for (int64_t i = tid; i < n; i += NT) keys[i] = src[i];
  __syncthreads();
}

template <int NT, int KPT4, int MODE>
__global__ void __launch_bounds__(NT, 512 / NT) seg_tile_kernel(SegParams prm) {
  using L = SegTileSmem<NT, KPT4, MODE>;
  extern __shared__ __align__(128) unsigned char smem[];
  int* s_seg = reinterpret_cast<int*>(smem + L::OFF_SEG);
  if (MODE == RANK_PEER_MASK) {
    uint32_t* s_msk = reinterpret_cast<uint32_t*>(smem + L::OFF_MSK);
    for (int i = threadIdx.x; i < L::NW * 2 * RADIX; i += NT) s_msk[i] = 0u;
  }
  if (threadIdx.x == 0) {
    mbar_init(reinterpret_cast<uint64_t*>(smem + L::OFF_MBAR), 1);
    fence_mbar_init();
  }
  uint32_t phase = 0;
  for (;;) {
    if (threadIdx.x == 0) *s_seg = int(atomicAdd(prm.queue, 1u));
    __syncthreads();
    const int sidx = *s_seg;
    __syncthreads();
    if (sidx >= prm.nsegs) break;
    const SegDesc sd = prm.segs[sidx];
    if (sd.n <= 1) continue;
    const int kind = sd.dtype % 3;  // u32, i32, f32, u64, i64, f64: unsigned, signed, float
    // The wide shape, one array at a time on its SM, has a copy for unsigned 8-byte keys without the order
    // transform, which every digit of theirs paid: one array of 13,000 keys 94 -> 86 us, 148 of 50,000 323 ->
    // 300 (u32 arrays, whose code shares the registers, 0-3% slower).  Two arrays per SM share their code.
    if (NT == 512 && sd.dtype == 3)
      seg_tile_sort<uint64_t, NT, KPT4, MODE>(static_cast<uint64_t*>(sd.keys), static_cast<uint64_t*>(sd.scratch), sd.n, KIND_UNSIGNED, smem,
                                    prm.err, prm.spin_limit_ns, phase);
    else if (sd.dtype >= 3)
      seg_tile_sort<uint64_t, NT, KPT4, MODE>(static_cast<uint64_t*>(sd.keys), static_cast<uint64_t*>(sd.scratch), sd.n, kind, smem,
                                    prm.err, prm.spin_limit_ns, phase);
    else
      seg_tile_sort<uint32_t, NT, KPT4, MODE>(static_cast<uint32_t*>(sd.keys), static_cast<uint32_t*>(sd.scratch), sd.n, kind, smem,
                                    prm.err, prm.spin_limit_ns, phase);
  }
}

}  // namespace hpcs
