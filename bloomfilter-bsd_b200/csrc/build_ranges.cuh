// build_ranges.cuh -- batch_insert of a blocked Bloom filter range by range in
// shared memory.
//
// Global atomic ORs are bounded by the L2's atomic requests (two 32-byte
// sectors per key of a 64-byte block).  Here the filter is cut into ranges of
// at most kBuildRangeBytes that fit in shared memory, and two kernels build it:
//
//   1. key_scatter_kernel          sorts each tile of keys by range in shared
//                                  memory and appends its runs to the ranges'
//                                  buckets (4 bytes per key)
//   2. bloom_build_ranges_kernel   one CTA per range: its bucket's keys are
//                                  ORed into zeroed shared memory with
//                                  shared-memory atomics, the words that have
//                                  bits ORed into the filter with coalesced
//                                  global atomics (a 32-byte sector each)
//
// The filter's words are never read and stored back, so builds may overlap
// other inserts into the same words, as those of the other plans.
//
// Measured (u64 w=8 s=8 k=8): 2^27 keys into 256 MiB, 2034 us with the coarse
// partition and global atomics, 1056 so: the scatter 496 (270 Gkeys/s; 0.67
// LSU wavefronts per key, the pipe 63 % busy, barriers and shared-memory
// latency the rest), the range build the rest (8 shared atomics of 3.5 bank
// cycles per warp and key, and the atomics on the words).
//
// A bucket holds its expected share of the keys and some slack; the keys of a
// run that does not fit are ORed into the words by the scatter itself, before
// the second kernel reads them, so any key distribution gives the same words.
#pragma once

#include <cstdint>

#include "bloom.cuh"
#include "common.cuh"

namespace dtlg {

constexpr uint32_t kBuildRangeBytes = 128u << 10;  // largest range (dynamic shared memory of its CTA)
constexpr uint32_t kBuildMaxRanges = 4096;
constexpr int kScatterThreads = 1024;
constexpr int kScatterKeysPerThread = 16;
constexpr uint32_t kScatterTile = kScatterThreads * kScatterKeysPerThread;

struct RangeArgs {
  const uint32_t* keys_al;  // 16-byte aligned key base (see ProbeArgs)
  uint64_t n_phys;
  uint32_t pre;
  Addr addr;
  uint32_t range_log2;      // a range is 2^range_log2 consecutive blocks
  uint32_t range_shift;     // POW2: range = block hash >> range_shift (two ranges or more)
  uint32_t n_ranges;
  uint32_t n_tiles;
  uint32_t cap;             // keys per bucket, a multiple of 4; n_ranges * cap < 2^32
  uint32_t* buckets;        // n_ranges x cap
  unsigned int* fill;       // per range: keys sent to its bucket, may exceed cap (zeroed)
  uint32_t prefetch;        // the range build hints its range + prefetch into L2 (0: none)
  void* filter;
  // the layout, for the keys that find their bucket full
  uint32_t word_bytes, w;
  Schedule sched;
};

#ifdef __CUDACC__

// Hints `bytes` (a multiple of 16) from a 16-byte aligned address into L2.
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(bytes) : "memory");
}

// BloomOps::insert for a layout known at run time, one 32-bit atomic per bit.
static __device__ __noinline__ void insert_any(const RangeArgs& a, uint32_t key) {
  const uint32_t per = a.word_bytes / 4;
  unsigned int* base = static_cast<unsigned int*>(a.filter) +
                       static_cast<uint64_t>(block_index(key * mul_const(0), a.addr)) * a.w * per;
  for (uint32_t g = 0; g < a.sched.ng; g++) {
    const Group& gr = a.sched.g[g];
    auto draw = [&](uint32_t sel, uint32_t shift, uint32_t bits) {
      return sel == kSelZero ? 0u : (key * mul_const(static_cast<int>(sel)) >> shift) & ((1u << bits) - 1u);
    };
    const uint32_t word = gr.wconst + (gr.wbits ? draw(gr.wsel, gr.wshift, gr.wbits) : 0u);
    for (uint32_t j = 0; j < gr.nbit; j++) {
      const uint32_t b = draw(gr.bit[j].sel, gr.bit[j].shift, gr.bit[j].bits) + gr.bit[j].off;
      atomicOr(base + word * per + (b >> 5), 1u << (b & 31u));
    }
  }
}

// The range of a key: the top bits of its block hash under POW2 addressing.
template <bool MAGIC>
__device__ __forceinline__ uint32_t build_range_of(uint32_t key, const RangeArgs& a) {
  const uint32_t h = key * mul_const(0);
  if constexpr (MAGIC) return block_index_of<true>(h, a.addr) >> a.range_log2;
  return h >> a.range_shift;
}

// Shared memory of a scatter CTA (dynamic): the tile's keys sorted by range,
// the ranges' counts (then run starts), the ranges' destinations.
struct KeyScatter {
  static constexpr uint32_t THREADS = kScatterThreads, kTile = kScatterTile;
  static constexpr int kVecs = kScatterKeysPerThread / 4;
  static constexpr uint32_t kPer = (kBuildMaxRanges + THREADS - 1) / THREADS;  // ranges per thread at most

  // One tile; FULL: all its kTile keys are valid.
  template <bool MAGIC, bool FULL>
  __device__ __forceinline__ static void tile(const RangeArgs& a, uint32_t tile, uint32_t* s_keys, uint32_t* s_cnt,
                                              uint32_t* s_dst, uint32_t* s_warp) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t tile_pos = static_cast<uint64_t>(tile) * kTile;
    const uint32_t lo = FULL || tile_pos >= a.pre ? 0u : static_cast<uint32_t>(a.pre - tile_pos);
    const uint32_t hi = FULL ? kTile : static_cast<uint32_t>(a.n_phys - tile_pos < kTile ? a.n_phys - tile_pos : kTile);
    const uint4* t4 = reinterpret_cast<const uint4*>(a.keys_al) + tile_pos / 4 + threadIdx.x;
    auto valid = [&](uint32_t li) { return FULL || (li >= lo && li < hi); };
    uint32_t rank[kVecs * 2];  // two 16-bit ranks per register
#pragma unroll
    for (int i = 0; i < kVecs; i++) {
      const uint32_t li = (i * THREADS + threadIdx.x) * 4;
      const uint4 kv = FULL || li < hi ? __ldcg(t4 + i * THREADS) : make_uint4(0, 0, 0, 0);
      const uint32_t k[4] = {kv.x, kv.y, kv.z, kv.w};
      uint32_t rk[4];
#pragma unroll
      for (int q = 0; q < 4; q++)
        rk[q] = valid(li + q) ? atomicAdd(&s_cnt[build_range_of<MAGIC>(k[q], a)], 1u) : 0u;
      rank[2 * i] = rk[0] | rk[1] << 16;
      rank[2 * i + 1] = rk[2] | rk[3] << 16;
    }
    __syncthreads();
    // strided: reserve the runs (coalesced); consecutive: exclusive scan
    uint32_t g[kPer], c_of[kPer];
#pragma unroll
    for (uint32_t j = 0; j < kPer; j++) {
      const uint32_t r = j * THREADS + threadIdx.x;
      c_of[j] = r < a.n_ranges ? s_cnt[r] : 0u;
      g[j] = c_of[j] ? atomicAdd(a.fill + r, c_of[j]) : 0u;
    }
    const uint32_t per = (a.n_ranges + THREADS - 1) / THREADS;
    const uint32_t r0 = threadIdx.x * per;
    uint32_t sum = 0;
    for (uint32_t j = 0; j < per; j++) sum += r0 + j < a.n_ranges ? s_cnt[r0 + j] : 0u;
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= static_cast<uint32_t>(d)) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    // the warp totals before this warp's, summed by its lanes
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[lane] : 0u);
    uint32_t run = before + incl - sum;
    for (uint32_t j = 0; j < per; j++) {
      if (r0 + j < a.n_ranges) {
        const uint32_t c = s_cnt[r0 + j];
        s_cnt[r0 + j] = run;
        run += c;
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kVecs; i++) {
      const uint32_t li = (i * THREADS + threadIdx.x) * 4;
      const uint4 kv = FULL || li < hi ? __ldcs(t4 + i * THREADS) : make_uint4(0, 0, 0, 0);
      const uint32_t k[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t rk = q & 1 ? rank[2 * i + q / 2] >> 16 : rank[2 * i + q / 2] & 0xffffu;
        if (valid(li + q)) s_keys[s_cnt[build_range_of<MAGIC>(k[q], a)] + rk] = k[q];
      }
    }
    // the reservations arrive while the keys are placed
    bool over = false;
#pragma unroll
    for (uint32_t j = 0; j < kPer; j++) {
      const uint32_t r = j * THREADS + threadIdx.x;
      if (r < a.n_ranges) {
        // a reservation beyond the bucket is clamped to its end, so that the
        // 32-bit index cannot wrap into another bucket
        const uint32_t at = g[j] < a.cap ? g[j] : a.cap;
        s_dst[r] = r * a.cap + at - s_cnt[r];
        over |= g[j] + c_of[j] > a.cap;
      }
    }
    const bool any_over = __syncthreads_or(over);
    for (uint32_t i = threadIdx.x; i < a.n_ranges; i += THREADS) s_cnt[i] = 0;  // for the next tile
    if (FULL && !any_over) {
#pragma unroll 4
      for (uint32_t j = 0; j < kScatterKeysPerThread; j++) {
        const uint32_t sl = j * THREADS + threadIdx.x;
        const uint32_t key = s_keys[sl];
        a.buckets[s_dst[build_range_of<MAGIC>(key, a)] + sl] = key;
      }
    } else {
      for (uint32_t sl = threadIdx.x; sl < hi - lo; sl += THREADS) {
        const uint32_t key = s_keys[sl];
        const uint32_t r = build_range_of<MAGIC>(key, a);
        const uint32_t at = s_dst[r] + sl;
        if (at - r * a.cap < a.cap) {
          a.buckets[at] = key;
        } else {
          insert_any(a, key);
        }
      }
    }
    __syncthreads();
  }
};

// Tiles of 1024 * 16 keys: count per range (the counting atomic's result is
// the key's rank in its run, kept as 16 bits), reserve the runs in the buckets
// with coalesced global atomics while the counts are scanned, place the keys
// (read again, from L2) at run start + rank, write the runs out.  Bound by
// instruction issue and shared-memory wavefronts, hence the tiles of valid
// keys and fitting runs without a test per key.
template <bool MAGIC>
static __global__ void __launch_bounds__(kScatterThreads, 2)
key_scatter_kernel(const __grid_constant__ RangeArgs a) {
  using S = KeyScatter;
  extern __shared__ __align__(16) uint32_t s_keys[];
  uint32_t* s_cnt = s_keys + S::kTile;
  uint32_t* s_dst = s_cnt + a.n_ranges;
  __shared__ uint32_t s_warp[32];
  for (uint32_t i = threadIdx.x; i < a.n_ranges; i += S::THREADS) s_cnt[i] = 0;
  __syncthreads();
  for (uint32_t tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
    const uint64_t pos = static_cast<uint64_t>(tile) * S::kTile;
    // the CTA's next tile into L2, if it lies wholly in the key array
    const uint64_t next = pos + static_cast<uint64_t>(gridDim.x) * S::kTile;
    if (threadIdx.x == 0 && next + S::kTile <= a.n_phys) prefetch_l2(a.keys_al + next, S::kTile * 4);
    if (pos >= a.pre && a.n_phys - pos >= S::kTile) {
      S::tile<MAGIC, true>(a, tile, s_keys, s_cnt, s_dst, s_warp);
    } else {
      S::tile<MAGIC, false>(a, tile, s_keys, s_cnt, s_dst, s_warp);
    }
  }
}

// The bits of one key into its block `lb` of a range in shared memory.  Words
// sit with their index in the block XORed with bits of the block number above
// the 128-byte bank row, so that a warp's atomics on the same word of
// different blocks spread over all banks.
template <class Cfg>
struct RangeBlock {
  using Word = typename Cfg::word_t;
  using Ops = BloomOps<Cfg>;
  static constexpr uint32_t kW = Cfg::kW;
  static constexpr uint32_t kRowShift = Cfg::kBlockBytes < 128 ? clog2(128 / Cfg::kBlockBytes) : 0;

  __device__ __forceinline__ static uint32_t swizzle(uint32_t lb) { return (lb >> kRowShift) & (kW - 1); }
  // index in shared memory of word i of the range
  __device__ __forceinline__ static uint32_t slot(uint32_t i) { return i ^ swizzle(i / kW); }

  // ORs the range's words into the filter, a coalesced run of atomics per warp.
  // Another insert into the same words may run at the same time, so they are
  // never read and stored back.
  __device__ __forceinline__ static void or_out(Word* gw, const Word* s_w, uint32_t nw) {
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < nw; i += blockDim.x) {
      const Word v = s_w[slot(i)];
      if (v != 0) atomic_or_word<Word>(gw + i, v);
    }
  }

  __device__ __forceinline__ static void insert(Word* s_w, uint32_t lb, uint32_t key) {
    const uint32_t swz = swizzle(lb);
    Word* base = s_w + lb * kW;
    static_for<Ops::kS.ng>([&](auto G) {
      constexpr int g = decltype(G)::value;
      constexpr Group grp = Ops::kS.g[g];
      uint32_t* p = reinterpret_cast<uint32_t*>(base + (Ops::template group_word<g>(key) ^ swz));
      if constexpr (sizeof(Word) == 8 && grp.nbit == 1) {
        // one bit: one 32-bit atomic on the half that holds it
        constexpr BitDraw b = grp.bit[0];
        const uint32_t bit = ((hash_sel<b.sel>(key) >> b.shift) & ((1u << b.bits) - 1u)) + b.off;
        atomicOr(p + (bit >> 5), 1u << (bit & 31u));
      } else if constexpr (sizeof(Word) == 8) {
        // 32-bit atomics: 64-bit shared-memory ORs are slower
        const unsigned long long m = Ops::template group_mask<g>(key);
        const uint32_t lo = static_cast<uint32_t>(m), hi = static_cast<uint32_t>(m >> 32);
        if (lo) atomicOr(p, lo);
        if (hi) atomicOr(p + 1, hi);
      } else {
        atomicOr(p, static_cast<uint32_t>(Ops::template group_mask<g>(key)));
      }
    });
  }
};

template <class Cfg>
__global__ void __launch_bounds__(1024) bloom_build_ranges_kernel(const __grid_constant__ RangeArgs a) {
  using R = RangeBlock<Cfg>;
  using Word = typename Cfg::word_t;
  extern __shared__ __align__(16) uint32_t s_keys[];
  Word* s_w = reinterpret_cast<Word*>(s_keys);
  const uint32_t rg = blockIdx.x;
  const uint32_t fill = a.fill[rg];
  const uint32_t cnt = fill < a.cap ? fill : a.cap;
  if (cnt == 0) return;
  const uint32_t blk0 = rg << a.range_log2;
  const uint32_t left = a.addr.block_cnt - blk0;
  const uint32_t nw = (left < (1u << a.range_log2) ? left : 1u << a.range_log2) * Cfg::kW;
  Word* gw = static_cast<Word*>(a.filter) + static_cast<uint64_t>(blk0) * Cfg::kW;
  if (threadIdx.x == 0) {
    // the range that this SM takes next or soon, into L2 while this one is built
    const uint32_t nx = rg + a.prefetch;
    if (a.prefetch != 0 && nx + 1 < a.n_ranges) {
      prefetch_l2(gw + static_cast<uint64_t>(a.prefetch) * ((1u << a.range_log2) * Cfg::kW), (1u << a.range_log2) * Cfg::kBlockBytes);
      const uint32_t f = a.fill[nx];
      prefetch_l2(a.buckets + static_cast<uint64_t>(nx) * a.cap, ((f < a.cap ? f : a.cap) & ~3u) * 4);
    }
  }
  for (uint32_t i = threadIdx.x; i < (Cfg::kBlockBytes << a.range_log2) / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(s_keys)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  const uint4* bk = reinterpret_cast<const uint4*>(a.buckets + static_cast<uint64_t>(rg) * a.cap);
  constexpr uint32_t kU = 2;  // key vectors in flight per thread
  for (uint32_t v0 = threadIdx.x; v0 * 4 < cnt; v0 += kU * blockDim.x) {
    uint4 kv[kU];
#pragma unroll
    for (uint32_t u = 0; u < kU; u++)
      kv[u] = (v0 + u * blockDim.x) * 4 < cnt ? __ldcs(bk + v0 + u * blockDim.x) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (uint32_t u = 0; u < kU; u++) {
      const uint32_t k[4] = {kv[u].x, kv[u].y, kv[u].z, kv[u].w};
#pragma unroll
      for (uint32_t q = 0; q < 4; q++) {
        if ((v0 + u * blockDim.x) * 4 + q < cnt)
          R::insert(s_w, block_index(k[q] * mul_const(0), a.addr) - blk0, k[q]);
      }
    }
  }
  __syncthreads();
  R::or_out(gw, s_w, nw);
}

#endif  // __CUDACC__

}  // namespace dtlg
