// probe.cuh -- batch_contains as one pass: probe + ordered match compaction.
//
// Contract (blocked_bloomfilter_batch_dispatch.hpp:29-69, filter_base.hpp:34-45):
// write i + match_offset (32-bit wrap) for every matching key index i, in
// ascending order, and return the count.
//
// Shape: CTAs of 256 or 1024 threads pull tiles of 1024 or 4096 keys
// (fused_shape) from a device counter (so a tile is only ever taken after all earlier tiles were
// taken by running CTAs: the waits below cannot deadlock).  Inside a tile,
// thread t owns 1 or 4 consecutive keys of each round (4: loaded as one
// 16-byte vector); matches are ranked with warp ballots and a CTA scan, and
// the tile's global offset comes from the per-tile status words, summed at
// once or by a decoupled look-back.  Every wait is bounded: on timeout the
// kernel raises the error word and carries on with a short prefix, so it
// always terminates.
#pragma once

#include <cstdint>

#include "common.cuh"

namespace dtlg {

struct ProbeArgs {
  const void* filter;           // Bloom words / cuckoo table (+ victim record)
  const uint32_t* keys_al;      // keys rounded down to a 16-byte boundary
  uint64_t n_phys;              // pre + key_cnt
  uint32_t pre;                 // keys_al[0 .. pre) precede the first key
  uint32_t match_offset;
  uint32_t* out;                // match positions
  unsigned long long* count_out;  // device: total match count
  unsigned long long* status;   // per-tile look-back words (zeroed)
  unsigned int* tile_ctr;       // tile queue head (zeroed)
  unsigned int* err;            // error word (zeroed); bit 0 = wait timed out
  uint32_t n_tiles;
  // Fused plan, blocking calls (result != null): the CTA that finishes last
  // clears the words above for the slot's next call and writes the outcome to
  // host memory (see result_word).
  unsigned int* done;           // CTAs finished (zeroed)
  unsigned long long* result;
  uint32_t ticket;
  Addr addr;
  uint64_t victim_word;         // cuckoo: 32-bit word index of the victim record
  // Block-range pass (two-pass probe only; all zero = off): a key whose block
  // (bucket) lies outside [blk_lo, blk_hi) is not probed in this pass.
  uint32_t range_on, blk_lo, blk_hi;
  // 1 when the filter base is 32-byte aligned: blocks of >= 32 bytes are then
  // read with 256-bit loads.
  uint32_t vec32;
  // 1: a Bloom filter's 256-bit block loads do not allocate in L1 (bitmask
  // plan, filters that cannot live in L1; set by the planner)
  uint32_t l1na;
  // 1: the bitmask kernel tests several keys at once where the kind can
  // (Ops::contains_n; set by the planner)
  uint32_t together;
  // blocked cuckoo filter: log2(buckets per block), and the shift that turns
  // the block hash into the bucket hash (32: the bucket hash is key * C[0])
  uint32_t bcf_bucket_bits, bcf_hash_shift;
  // classic Bloom filter: bits per key, and the bit index (h >> shift) & mask
  uint32_t cbf_k, cbf_bit_shift, cbf_bit_mask;
};

// The outcome of a blocking fused probe in one 64-bit word, so that the host
// sees all of it or nothing: ticket of the call | error bit | match count
// (below 2^31 for every batch of the one-round shapes).
constexpr uint32_t kResultErr = 1u << 31;
__host__ __device__ constexpr unsigned long long result_word(uint32_t ticket, bool err, uint32_t count) {
  return static_cast<unsigned long long>(ticket) << 32 | (err ? kResultErr : 0u) | count;
}

constexpr int kProbeThreads = 256;
constexpr unsigned long long kFlagAgg = 1ull << 62;
constexpr unsigned long long kFlagPrefix = 2ull << 62;
constexpr uint32_t kSpinLimit = 1u << 22;  // ~ seconds with the backoff below

#ifdef __CUDACC__

__device__ __forceinline__ unsigned long long ld_volatile(const unsigned long long* p) {
  return *reinterpret_cast<const volatile unsigned long long*>(p);
}
__device__ __forceinline__ void st_volatile(unsigned long long* p, unsigned long long v) {
  *reinterpret_cast<volatile unsigned long long*>(p) = v;
}

// Exclusive prefix of this tile from the predecessors' status words (warp 0).
// A wait that spins `limit` times sets bit 0 of *a.err and returns what it has.
__device__ __forceinline__ uint32_t look_back(const ProbeArgs& a, uint32_t tile, uint32_t lane,
                                              uint32_t limit = kSpinLimit) {
  uint32_t excl = 0;
  int64_t pred = static_cast<int64_t>(tile) - 1;
  uint32_t spins = 0;
  while (pred >= 0) {
    const int64_t idx = pred - static_cast<int64_t>(lane);
    const unsigned long long st = idx >= 0 ? ld_volatile(a.status + idx) : kFlagPrefix;
    const unsigned long long flag = st & (3ull << 62);
    const uint32_t not_ready = __ballot_sync(0xffffffffu, flag == 0);
    const uint32_t prefix = __ballot_sync(0xffffffffu, flag == kFlagPrefix);
    // lanes 0..fp (nearest predecessors first) must all be ready
    const uint32_t need = prefix ? ((prefix & (0u - prefix)) << 1) - 1u : 0xffffffffu;
    if (not_ready & need) {
      if (++spins > limit) {
        if (lane == 0) atomicOr(a.err, 1u);
        break;
      }
      __nanosleep(64);
      continue;
    }
    uint32_t v = (need >> lane) & 1u ? static_cast<uint32_t>(st) : 0u;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    excl += v;
    if (prefix) break;
    pred -= 32;
  }
  return excl;
}

// Exclusive prefix of this tile as the sum of every earlier tile's aggregate,
// one status word per thread and step (all threads of the CTA; s_sum: one word
// per warp).  For grids whose tiles all run at once: their aggregates appear
// at the same time, so a look-back by 32 would walk the whole list window by
// window, one L2 round trip each, where this takes one round trip in all.
// The waits are bounded as in look_back.
__device__ __forceinline__ uint32_t sum_predecessors(const ProbeArgs& a, uint32_t tile, uint32_t* s_sum) {
  uint32_t sum = 0, spins = 0;
  for (uint32_t p = threadIdx.x; p < tile;) {
    const unsigned long long st = ld_volatile(a.status + p);
    if (st == 0) {
      if (++spins > kSpinLimit) {
        atomicOr(a.err, 1u);
        break;
      }
      __nanosleep(20);
      continue;
    }
    sum += static_cast<uint32_t>(st);
    p += blockDim.x;
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if ((threadIdx.x & 31u) == 0) s_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  uint32_t total = 0;
  for (uint32_t w = 0; w < (blockDim.x >> 5); w++) total += s_sum[w];
  return total;
}

// Shape of the fused probe for a batch of n_phys keys: keys per thread and
// round, rounds per tile, threads per CTA.
struct FusedShape {
  uint32_t kpt, rounds, threads, n_tiles;
};

// Up to kFusedOneKey keys a thread tests one key, so that no thread waits for
// four gathers one after the other, in CTAs of 1024 threads, at most one per
// SM: few tiles to hand out and sum (blocking calls of 60 000 keys: 16.8 us,
// with 256-thread CTAs 20.5; 300 000 keys 23.4 against 20.8).  Up to
// kFusedOneRound keys a thread tests four (tiles of 1024); beyond, tiles of
// 4096 keys, whose fewer status words and tickets count more.  Kernel times
// against tiles of 4096 keys throughout, offsets by look-back: 60001 keys
// (zoned u32 w=16 z=4, 225 KiB) 12.7 -> 9 us, 900001 keys (u64 w=8 s=8 k=8, 8
// MiB) 22.7 -> 13.3 us, 1024 keys 4.2 + 1.5 (the zeroing) -> 3.4 us.
constexpr uint32_t kMaxRounds = 4;
constexpr uint64_t kFusedOneKey = 148ull << 10;
constexpr uint64_t kFusedOneRound = 2ull << 20;
constexpr uint32_t kFusedSumTiles = 2048;  // offsets by sum_predecessors up to this many tiles

__host__ __device__ inline FusedShape fused_shape(uint64_t n_phys) {
  FusedShape s{};
  s.kpt = n_phys <= kFusedOneKey ? 1u : 4u;
  s.threads = s.kpt == 1 ? 1024u : static_cast<uint32_t>(kProbeThreads);
  s.rounds = n_phys <= kFusedOneRound ? 1u : kMaxRounds;
  const uint32_t tile = s.threads * s.kpt * s.rounds;
  s.n_tiles = static_cast<uint32_t>((n_phys + tile - 1) / tile);
  return s;
}

// Ops::contains(const ProbeArgs&, uint32_t key) -> bool, safe for any key
// value (block / bucket indexes are always inside the filter).  KPT keys per
// thread and round, ROUNDS rounds per tile.
template <class Ops, int KPT, int ROUNDS, int THREADS>
__global__ void __launch_bounds__(THREADS)
probe_kernel(const __grid_constant__ ProbeArgs a) {
  constexpr uint32_t kRoundKeys = THREADS * KPT;
  constexpr uint32_t kWarps = THREADS / 32;
  static_assert(ROUNDS * kWarps <= 32, "one warp scans the warp totals");
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_wtot[ROUNDS * kWarps];
  __shared__ uint32_t s_excl;
  __shared__ uint32_t s_sum[kWarps];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const bool by_sum = a.n_tiles <= kFusedSumTiles;

  for (;;) {
    uint32_t tile = 0;
    if (a.n_tiles > 1) {
      if (threadIdx.x == 0) s_tile = atomicAdd(a.tile_ctr, 1u);
      __syncthreads();
      tile = s_tile;
      if (tile >= a.n_tiles) break;
    }
    const uint64_t tbase = static_cast<uint64_t>(tile) * (kRoundKeys * ROUNDS);

    uint32_t flags[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
      const uint64_t p0 = tbase + r * kRoundKeys + threadIdx.x * KPT;
      uint32_t f = 0;
      if (p0 < a.n_phys) {
        uint32_t k[KPT];
        if constexpr (KPT == 4) {
          const uint4 kv = __ldcs(reinterpret_cast<const uint4*>(a.keys_al) + (p0 >> 2));
          k[0] = kv.x; k[1] = kv.y; k[2] = kv.z; k[3] = kv.w;
        } else {
          k[0] = __ldcs(a.keys_al + p0);
        }
#pragma unroll
        for (int q = 0; q < KPT; q++) f |= (Ops::contains(a, k[q]) ? 1u : 0u) << q;
        // drop lanes before the first key and past the last one
#pragma unroll
        for (int q = 0; q < KPT; q++) {
          const uint64_t p = p0 + q;
          if (p < a.pre || p >= a.n_phys) f &= ~(1u << q);
        }
      }
      flags[r] = f;
      const uint32_t tot = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(__popc(f)));
      if (lane == 0) s_wtot[r * kWarps + warp] = tot;
    }
    __syncthreads();

    uint32_t agg = 0;
    if (warp == 0) {
      // exclusive scan of the warp totals in key order (round-major)
      const uint32_t v = lane < ROUNDS * kWarps ? s_wtot[lane] : 0u;
      uint32_t incl = v;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= static_cast<uint32_t>(d)) incl += t;
      }
      agg = __shfl_sync(0xffffffffu, incl, 31);
      if (lane == 0 && a.n_tiles > 1)
        st_volatile(a.status + tile, ((tile == 0 || by_sum) ? kFlagPrefix : kFlagAgg) | agg);
      if (lane < ROUNDS * kWarps) s_wtot[lane] = incl - v;
      if (!by_sum) {
        uint32_t excl = 0;
        if (tile > 0) {
          excl = look_back(a, tile, lane);
          if (lane == 0) st_volatile(a.status + tile, kFlagPrefix | static_cast<uint32_t>(excl + agg));
        }
        if (lane == 0) s_excl = excl;
      }
    }
    uint32_t excl;
    if (by_sum) {
      excl = sum_predecessors(a, tile, s_sum);  // its barrier also publishes s_wtot
    } else {
      __syncthreads();
      excl = s_excl;
    }
    if (threadIdx.x == 0 && tile == a.n_tiles - 1) {
      if (a.n_tiles == 1) *a.err = 0u;  // the workspace is not zeroed for one tile
      const bool failed = *reinterpret_cast<volatile unsigned int*>(a.err) != 0u;
      *a.count_out = failed ? ~0ull : static_cast<unsigned long long>(excl) + agg;
    }

#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
      uint32_t f = flags[r];
      // rank of this thread's matches among the warp's
      uint32_t rank = 0;
#pragma unroll
      for (int q = 0; q < KPT; q++) rank += __popc(__ballot_sync(0xffffffffu, (f >> q) & 1u) & lt_mask);
      uint32_t pos = excl + s_wtot[r * kWarps + warp] + rank;
      const uint64_t p0 = tbase + r * kRoundKeys + threadIdx.x * KPT;
      const uint32_t logical0 = static_cast<uint32_t>(p0 - a.pre);
      while (f) {
        const int q = __ffs(f) - 1;
        f &= f - 1;
        __stcs(a.out + pos, logical0 + static_cast<uint32_t>(q) + a.match_offset);
        pos++;
      }
    }
    if (a.n_tiles <= gridDim.x) break;  // one tile per CTA
    __syncthreads();
  }
  if constexpr (ROUNDS == 1) {
    if (a.result == nullptr) return;
    __shared__ bool s_last;
    __syncthreads();  // the CTA's positions are written
    if (threadIdx.x == 0) {
      __threadfence();
      s_last = a.n_tiles == 1 || atomicAdd(a.done, 1u) == a.n_tiles - 1;
    }
    __syncthreads();
    if (!s_last) return;
    // every other CTA has finished with the status words
    if (a.n_tiles > 1)
      for (uint32_t i = threadIdx.x; i < a.n_tiles; i += blockDim.x) a.status[i] = 0ull;
    __syncthreads();
    if (threadIdx.x == 0) {
      const bool failed = *reinterpret_cast<volatile unsigned int*>(a.err) != 0u;
      const unsigned long long n = ld_volatile(a.count_out);
      *a.tile_ctr = 0u;
      *a.done = 0u;
      *a.err = 0u;
      __threadfence_system();
      st_volatile(a.result, result_word(a.ticket, failed, static_cast<uint32_t>(n) & ~kResultErr));
    }
  }
}

#endif  // __CUDACC__

}  // namespace dtlg
