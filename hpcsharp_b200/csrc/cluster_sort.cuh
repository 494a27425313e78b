// LSD sort of a small array (keys, or keys with a 32-bit item each), in place, in one launch of one
// thread-block cluster.
//
// A sort of ~10^5 keys through the large-array kernels is a chain of launches with little to do in
// each, and a cooperative launch with a grid barrier through L2 per exchange took ~9 us a pass (42 us
// for 100 Ki u32 keys, 22 us for 1000).  Here CTA c of the cluster owns the keys at positions [c *
// SLICE, (c + 1) * SLICE).  Per pass:
//   rank     the slice's keys, warp-striped in registers, by the sort's per-warp ranking; stable;
//   totals   the slice's digit totals go to every CTA of the cluster (distributed shared memory), the
//            slice is reordered by digit in shared memory, and a cluster barrier follows;
//   bases    every CTA adds up the totals: digit starts over all slices + the totals of the slices
//            before its own (the bin-major / quantum-minor offsets of RadixSortLsdParallel.cs:49-94 with
//            one quantum per CTA);
//   scatter  coalesced per-digit runs into the array itself (every slice is in registers by now), and
//            a second cluster barrier, after which the next pass reads its slice through L2.
// Writing the runs into the owners' shared memory instead (two buffers per CTA) cost more: remote
// stores of ~32-key runs moved 5.6 bytes per clock and CTA (131072 u32 keys: 5800 of 13800 clocks a
// pass).  An array of one slice never leaves its CTA: the reordered slice is the next pass's input,
// and no cluster barrier is taken.
// A pass whose keys all share one digit moves nothing.  The largest shape, whose sizes the look-back
// passes sorted before with such passes left out, does not rank them either: its first pass finds the bits
// that vary over all keys (the differences from the first key travel with the totals).  262,144 equal u32
// keys: 56 us a call with four ranked passes, 19.5 so; smaller shapes would pay ~2 us of 30 for it.  The barriers are the cluster's hardware barrier
// and every CTA takes the same ones, so no wait depends on data.
#pragma once
#include <cstdint>

#include "radix_kernels.cuh"

namespace hpcs {

constexpr int CS_NT = 512;
constexpr int CS_MAX_CTAS = 16;  // beyond 8 CTAs a cluster is non-portable: asked for at launch

template <class U, class V, int KPT, int MODE>
struct ClusterSmem {
  static constexpr bool PAIRS = !std::is_same<V, NoValue>::value;
  static constexpr int SLICE = CS_NT * KPT;
  static constexpr int NW = CS_NT / 32;
  static constexpr int G = CS_NT / RADIX;     // threads per digit in the digit scan
  static constexpr int NWG = NW / G;          // warps summed by each of them
  static constexpr int RS = RADIX + 32 / NW;  // warp-counter row stride: conflict-free scan
  static constexpr int OS = RADIX + 2;        // offset row stride (16-bit)
  static constexpr size_t KEYS_BYTES = size_t(SLICE) * sizeof(U);
  static constexpr size_t BUF_BYTES = KEYS_BYTES + (PAIRS ? size_t(SLICE) * 4 : 0);
  static constexpr size_t OFF_BUF = 0;  // the reordered slice
  static constexpr size_t OFF_CNT = OFF_BUF + BUF_BYTES;                          // [NW][RS]
  static constexpr size_t OFF_OFFSETS = OFF_CNT + size_t(NW) * RS * 4;                // [NW][OS], 16-bit
  static constexpr size_t OFF_MSK = (OFF_OFFSETS + size_t(NW) * OS * 2 + 15) / 16 * 16;
  static constexpr size_t MSK_BYTES = MODE == RANK_PEER_MASK ? size_t(NW) * 2 * RADIX * 4 : 0;
  static constexpr size_t OFF_TOT = OFF_MSK + MSK_BYTES;                              // [CTAS][256] totals
  static constexpr size_t OFF_GBASE = OFF_TOT + size_t(CS_MAX_CTAS) * RADIX * 4;      // global base - local
  static constexpr size_t OFF_WSUM = OFF_GBASE + RADIX * 4;
  static constexpr bool LOOK = KPT >= 32;  // leaves passes on constant digits out
  static constexpr size_t OFF_WBITS = OFF_WSUM + 32 * 4;                        // [NW] varying bits of a warp's keys
  static constexpr size_t OFF_CBITS = OFF_WBITS + size_t(NW) * sizeof(U);       // [CTAS] of a CTA's
  static constexpr size_t BYTES = LOOK ? OFF_CBITS + size_t(CS_MAX_CTAS) * sizeof(U) : OFF_WBITS;
  static_assert(SLICE < 65536, "offsets are kept in 16 bits");
};

__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();  // (.aligned: the warp arrives as one)
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of this CTA's shared-memory address `a` in CTA `rank` of the cluster, and stores to it.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_store(uint32_t a, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t a, uint64_t v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
// OR over a warp's values.
__device__ __forceinline__ uint32_t warp_or(uint32_t v) { return __reduce_or_sync(0xFFFFFFFFu, v); }
__device__ __forceinline__ uint64_t warp_or(uint64_t v) {
  return uint64_t(warp_or(uint32_t(v >> 32))) << 32 | warp_or(uint32_t(v));
}
// Keys that other CTAs wrote: through L2, never from a stale L1 line.
__device__ __forceinline__ uint32_t ld_cg(const uint32_t* p) { return __ldcg(p); }
__device__ __forceinline__ uint64_t ld_cg(const uint64_t* p) {
  return __ldcg(reinterpret_cast<const unsigned long long*>(p));
}

template <class U, int KIND, class V, int KPT, int MODE>
__global__ void __launch_bounds__(CS_NT, 1) cluster_sort_kernel(U* keys, uint32_t* vals, uint32_t n, int skip_trivial,
                                                               uint32_t* err) {
  using L = ClusterSmem<U, V, KPT, MODE>;
  constexpr bool PAIRS = L::PAIRS;
  constexpr int P = int(sizeof(U));
  constexpr int NT = CS_NT, G = L::G, NWG = L::NWG, RS = L::RS;
  constexpr int BATCH = KPT < 8 ? KPT : 8;
  extern __shared__ __align__(128) unsigned char smem[];
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + L::OFF_CNT);
  uint16_t* s_off = reinterpret_cast<uint16_t*>(smem + L::OFF_OFFSETS);
  uint32_t* s_tot = reinterpret_cast<uint32_t*>(smem + L::OFF_TOT);
  uint32_t* s_gbase = reinterpret_cast<uint32_t*>(smem + L::OFF_GBASE);
  uint32_t* s_wsum = reinterpret_cast<uint32_t*>(smem + L::OFF_WSUM);
  U* s_wbits = reinterpret_cast<U*>(smem + L::OFF_WBITS);
  U* s_cbits = reinterpret_cast<U*>(smem + L::OFF_CBITS);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* cnt_w = s_cnt + warp * RS;
  const uint16_t* off_w = s_off + warp * L::OS;
  uint32_t* msk_w = reinterpret_cast<uint32_t*>(smem + L::OFF_MSK) + warp * 2 * RADIX;
  const uint32_t ctas = gridDim.x, cta = blockIdx.x;  // the grid is one cluster
  const uint32_t lo = cta * uint32_t(L::SLICE);
  const int cnt = n > lo ? int(n - lo < uint32_t(L::SLICE) ? n - lo : uint32_t(L::SLICE)) : 0;
  const int sd = tid / G, sq = tid % G;  // the digit and warp group this thread scans
  const int wbase = warp * 32 * KPT;
  bool out_of_range = false;

  const bool solo = ctas == 1u;
  if (!solo) cluster_arrive();  // waited for before the first store to another CTA: that CTA has started
  if (MODE == RANK_PEER_MASK)
    for (int i = lane; i < 2 * RADIX; i += 32) msk_w[i] = 0u;
  U* buf = reinterpret_cast<U*>(smem + L::OFF_BUF);
  uint32_t* vbuf = reinterpret_cast<uint32_t*>(smem + L::OFF_BUF + L::KEYS_BYTES);
  for (int i = lane; i < RADIX; i += 32) cnt_w[i] = 0u;
  const bool look = L::LOOK && skip_trivial;
  U varies = U(~U(0));  // the bits that differ among the keys (every bit until the first pass has looked)
  for (int p = 0; p < P; p++) {
    if (L::LOOK && (uint32_t(varies >> (8 * p)) & 0xFFu) == 0u) continue;  // uniform over the cluster
    const Digit<U, KIND> dig(8 * p);
    bool last = p == P - 1;
    __syncwarp();

    // ---- load (warp-striped) and rank within the warp --------------------------------
    U key[KPT];
    uint32_t val[PAIRS ? KPT : 1];
    uint32_t rank[(KPT + 1) / 2];  // two 16-bit ranks per word
    if (solo && p > 0) {
#pragma unroll
      for (int i = 0; i < KPT; i++) {
        const int idx = wbase + i * 32 + lane;
        key[i] = idx < cnt ? buf[idx] : U(0);
        if (PAIRS) val[PAIRS ? i : 0] = idx < cnt ? vbuf[idx] : 0u;
      }
    } else {
#pragma unroll
      for (int i = 0; i < KPT; i++) {
        const int idx = wbase + i * 32 + lane;
        key[i] = idx < cnt ? ld_cg(keys + lo + idx) : U(0);
        if (PAIRS) val[PAIRS ? i : 0] = idx < cnt ? ld_cg(vals + lo + idx) : 0u;
      }
    }
    if (look && p == 0) {
      const U first = ld_cg(keys);
      U diff = U(0);
#pragma unroll
      for (int i = 0; i < KPT; i++)
        if (wbase + i * 32 + lane < cnt) diff |= key[i] ^ first;
      diff = warp_or(diff);
      if (lane == 0) s_wbits[warp] = diff;
    }
#pragma unroll
    for (int i = 0; i < (KPT + 1) / 2; i++) rank[i] = 0u;
#pragma unroll
    for (int i = 0; i < KPT; i++) {
      const bool valid = wbase + i * 32 + lane < cnt;
      rank[i / 2] |= rank_in_warp<MODE>(cnt_w, msk_w, dig(key[i]), valid, i & 1, lane) << (16 * (i & 1));
    }
    __syncthreads();  // warp counts complete; the slice is in registers

    // ---- scan over (digit, warp): slice offsets per warp; the digit totals go to every CTA ----
    uint32_t total, local;
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
      if (!solo) {
        if (p == 0) cluster_wait();  // every CTA has started
        // the digit's threads share the stores to the CTAs
        const uint32_t slot = smem_u32(s_tot + cta * RADIX + sd);
        for (uint32_t r = uint32_t(sq); r < ctas; r += uint32_t(G)) cluster_store(cluster_addr(slot, r), total);
        __syncwarp();
        if (look && p == 0 && warp == L::NW - 1) {
          const U diff = warp_or(lane < L::NW ? s_wbits[lane] : U(0));
          if (lane < int(ctas)) cluster_store(cluster_addr(smem_u32(s_cbits + cta), uint32_t(lane)), diff);
          __syncwarp();
        }
      }
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
    }
    __syncthreads();  // offsets ready; the counters are read

    // ---- reorder the slice by digit (a batch's lookups before its stores) --------------
#pragma unroll
    for (int b = 0; b < KPT; b += BATCH) {
      uint32_t pos[BATCH];
#pragma unroll
      for (int i = b; i < b + BATCH && i < KPT; i++)
        pos[i - b] = uint32_t(off_w[dig(key[i])]) + ((rank[i / 2] >> (16 * (i & 1))) & 0xFFFFu);
#pragma unroll
      for (int i = b; i < b + BATCH && i < KPT; i++) {
        if (wbase + i * 32 + lane < cnt) {
          buf[pos[i - b]] = key[i];
          if (PAIRS) vbuf[pos[i - b]] = val[PAIRS ? i : 0];
        }
      }
    }
    for (int i = lane; i < RADIX; i += 32) cnt_w[i] = 0u;  // for the next pass
    if (solo) {
      __syncthreads();  // the reordered slice is in place
      if (last) {
#pragma unroll
        for (int i = 0; i < KPT; i++) {
          const int s = i * NT + tid;
          if (s < cnt) {
            keys[s] = buf[s];
            if (PAIRS) vals[s] = vbuf[s];
          }
        }
      }
      continue;
    }
    cluster_arrive();  // (the totals have long arrived: the release does not wait for them)
    cluster_wait();    // every CTA's totals are here, and every CTA's keys are in registers
    if (look) {
      if (p == 0) {
        varies = warp_or(lane < int(ctas) ? s_cbits[lane] : U(0));
        // floats of both signs: the order flips every bit of the negative ones
        if (KIND == KIND_FLOAT && (varies >> (8 * P - 1)) != 0) varies = U(~U(0));
      }
      last = last || U(varies >> (8 * (p < P - 1 ? p + 1 : 0))) == 0;
    }

    // ---- global bases: digit starts over all slices + the slices before this one -------
    uint32_t all = 0, pre = 0;
    for (uint32_t r = uint32_t(sq); r < ctas; r += uint32_t(G)) {
      const uint32_t v = s_tot[r * RADIX + sd];
      all += v;
      pre += r < cta ? v : 0u;
    }
    __syncwarp();
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      all += __shfl_xor_sync(0xFFFFFFFFu, all, o);
      pre += __shfl_xor_sync(0xFFFFFFFFu, pre, o);
    }
    uint32_t di = all;  // inclusive over this warp's digits
#pragma unroll
    for (int o = G; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, di, o);
      if (lane >= o) di += y;
    }
    if (lane == 31) s_wsum[warp] = di;
    // (a pass with one digit value leaves the array as it is)
    const bool identity = __syncthreads_or(all == n) != 0 && skip_trivial;
    const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? s_wsum[lane] : 0u);
    if (sq == 0) s_gbase[sd] = before + di - all + pre - local;
    __syncthreads();  // bases and the reordered slice ready

    // ---- scatter: per-digit runs ---------------------------------------------------------
    if (!identity) {
#pragma unroll
      for (int b = 0; b < KPT; b += BATCH) {
        U k[BATCH];
        uint32_t v[PAIRS ? BATCH : 1], pos[BATCH];
#pragma unroll
        for (int i = 0; i < BATCH && b + i < KPT; i++) {
          const int s = (b + i) * NT + tid;
          k[i] = s < cnt ? buf[s] : U(0);
          if (PAIRS) v[PAIRS ? i : 0] = s < cnt ? vbuf[s] : 0u;
        }
#pragma unroll
        for (int i = 0; i < BATCH && b + i < KPT; i++) pos[i] = s_gbase[dig(k[i])] + uint32_t((b + i) * NT + tid);
#pragma unroll
        for (int i = 0; i < BATCH && b + i < KPT; i++) {
          if ((b + i) * NT + tid >= cnt) continue;
          if (pos[i] < n) {
            keys[pos[i]] = k[i];
            if (PAIRS) vals[pos[i]] = v[PAIRS ? i : 0];
          } else {
            out_of_range = true;
          }
        }
      }
    }
    if (!last) {
      cluster_arrive();  // the array holds this pass's order, and the totals are read
      cluster_wait();
    }
  }
  if (out_of_range) atomicOr(err, uint32_t(DERR_BOUNDS));
}

}  // namespace hpcs
