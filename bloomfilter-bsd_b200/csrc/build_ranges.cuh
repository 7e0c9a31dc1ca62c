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
// partition and global atomics, 1042 so: the scatter 515 (260 Gkeys/s; 0.67
// LSU wavefronts per key, the pipe some 60 % busy, barriers and shared-memory
// latency the rest), the range build 527 (8 shared atomics of 3.5 bank cycles
// per warp and key, and the atomics on the words).
//
// A bucket holds its expected share of the keys and some slack; the keys of a
// run that does not fit are ORed into the words by the scatter itself, so any
// key distribution gives the same words.
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

// One draw of a layout known at run time: (key * mul >> shift) & (2^bits - 1),
// then `first` (word or bit) is added.
struct RangeDraw {
  uint32_t mul;     // 0: the constant hash 0
  uint32_t fields;  // shift | bits << 8 | first << 16
};
constexpr uint32_t kMaxDraws = 32;  // a word draw for each of 16 groups, 16 bit draws at most

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
  unsigned int* fill;       // per range: keys sent to its bucket, may exceed cap; last: 1 when one did (zeroed)
  uint32_t prefetch;        // the range build hints its range + prefetch into L2 (0: none)
  void* filter;
  // the layout, for the keys that find their bucket full: per group its word
  // draw, then its `nbit` bit draws (every group has as many)
  uint32_t word_bytes, w, ng, nbit;
  RangeDraw draw[kMaxDraws];
};

// The layout fields of `a` from a schedule.
inline void set_range_layout(uint32_t word_bytes, uint32_t w, const Schedule& sched, RangeArgs* a) {
  a->word_bytes = word_bytes;
  a->w = w;
  a->ng = sched.ng;
  a->nbit = sched.g[0].nbit;
  RangeDraw* out = a->draw;
  for (uint32_t g = 0; g < sched.ng; g++) {
    const Group& gr = sched.g[g];
    *out++ = {gr.wbits ? mul_const(gr.wsel) : 0u, static_cast<uint32_t>(gr.wshift | gr.wbits << 8 | gr.wconst << 16)};
    for (uint32_t j = 0; j < gr.nbit; j++) {
      const BitDraw& d = gr.bit[j];
      *out++ = {d.sel == kSelZero ? 0u : mul_const(d.sel), static_cast<uint32_t>(d.shift | d.bits << 8 | d.off << 16)};
    }
  }
}

#ifdef __CUDACC__

// Hints `bytes` (a multiple of 16) from a 16-byte aligned address into L2.
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(bytes) : "memory");
}

// The range of a key: the top bits of its block hash under POW2 addressing.
template <bool MAGIC>
__device__ __forceinline__ uint32_t build_range_of(uint32_t key, const RangeArgs& a) {
  const uint32_t h = key * mul_const(0);
  if constexpr (MAGIC) return block_index_of<true>(h, a.addr) >> a.range_log2;
  return h >> a.range_shift;
}

// What the checked write-out reads, copied from the kernel's parameters, whose
// fields would be loaded from memory again after every atomic.
struct OverflowArgs {
  Addr addr;
  uint32_t range_sel, cap, word_bytes, w, ng, nbit;  // range_sel: range_log2 (MAGIC) or range_shift
  uint32_t* buckets;
  void* filter;
};

// Inserts the keys of the lanes with `over` set straight into the words, whole
// warps only.  The word groups of a key go to neighbouring lanes, one atomic
// each and one request per 32-byte sector (as BloomOps::insert_lanes).  Buckets
// overflow where keys repeat: where lanes have their neighbour's key, the
// copies within the warp are inserted once, and bits that are set already (a
// load from L1, which may miss newer ones) take no atomic.
// stage: 32 words of shared memory of this warp's own.
template <bool MAGIC>
__device__ __forceinline__ void insert_overflow(const OverflowArgs& a, uint32_t key, bool over, uint32_t* stage,
                                                const RangeDraw* s_draw) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t todo = __ballot_sync(0xffffffffu, over);
  if (todo == 0) return;
  const bool same = __shfl_xor_sync(0xffffffffu, key, 1) == key;
  if (__popc(__ballot_sync(0xffffffffu, over && same)) >= 3) {
    bool first = false;
    if (over) first = lane == static_cast<uint32_t>(__ffs(__match_any_sync(todo, key)) - 1);
    todo = __ballot_sync(0xffffffffu, first);
  }
  if (todo >> lane & 1u) stage[__popc(todo & ((1u << lane) - 1u))] = key;
  __syncwarp();
  const uint32_t per = 32u / a.ng;  // keys per step
  const uint32_t n = __popc(todo);
  const RangeDraw* d = s_draw + (lane % a.ng) * (1 + a.nbit);
  struct Draw {
    uint32_t mul, shift, mask, first;
    __device__ __forceinline__ Draw(const RangeDraw& r)
        : mul(r.mul), shift(r.fields & 0xffu), mask((1u << (r.fields >> 8 & 0xffu)) - 1u), first(r.fields >> 16) {}
    __device__ __forceinline__ uint32_t of(uint32_t k) const { return (k * mul >> shift & mask) + first; }
  };
  const Draw word(d[0]), bit(d[1]);
  const uint32_t halves = a.word_bytes / 4;  // 32-bit words per word
  unsigned int* const base = static_cast<unsigned int*>(a.filter);
  for (uint32_t i = lane < per * a.ng ? lane / a.ng : n; i < n; i += per) {
    const uint32_t k = stage[i];
    const uint32_t blk = block_index_of<MAGIC>(k * mul_const(0), a.addr);
    unsigned int* p = base + static_cast<uint64_t>(blk) * (a.w * halves) + word.of(k) * halves;
    uint32_t b = bit.of(k);
    if (a.nbit == 1) {
      p += b >> 5;
      const uint32_t m = 1u << (b & 31u);
      if ((ld_weak_32(p) & m) == 0) atomicOr(p, m);
    } else {
      unsigned long long m = 1ull << b;
      for (uint32_t j = 2; j <= a.nbit; j++) m |= 1ull << Draw(d[j]).of(k);
      if (halves == 2) {
        unsigned long long* p2 = reinterpret_cast<unsigned long long*>(p);
        if ((ld_weak_64(p2) & m) != m) atomicOr(p2, m);
      } else if ((ld_weak_32(p) & m) != m) {
        atomicOr(p, static_cast<unsigned int>(m));
      }
    }
  }
  __syncwarp();
}

// Writes a tile's n sorted keys to their buckets, those that do not fit into
// the words.  A function of its own, all threads of the CTA: its registers
// would spill the tile loop's.
template <bool MAGIC>
__device__ __noinline__ void write_tile_checked(const RangeArgs& args, uint32_t n, uint32_t* s_keys) {
  __shared__ RangeDraw s_draw[kMaxDraws];
  if (threadIdx.x < kMaxDraws) s_draw[threadIdx.x] = args.draw[threadIdx.x];
  __syncthreads();
  const uint32_t* s_dst = s_keys + kScatterTile + args.n_ranges;
  const OverflowArgs a{args.addr, MAGIC ? args.range_log2 : args.range_shift, args.cap, args.word_bytes, args.w, args.ng,
                       args.nbit, args.buckets, args.filter};
  auto place = [&](uint32_t sl, uint32_t* key, uint32_t* at) {  // does sorted slot sl's key fit its bucket
    *key = s_keys[sl];
    const uint32_t h = *key * mul_const(0);
    const uint32_t r = (MAGIC ? block_index_of<true>(h, a.addr) : h) >> a.range_sel;
    *at = s_dst[r] + sl;
    return *at - r * a.cap < a.cap;
  };
  uint32_t over_steps = 0;  // steps in which a key of this warp does not fit
#pragma unroll 4
  for (uint32_t j = 0; j < kScatterKeysPerThread; j++) {
    const uint32_t sl = j * kScatterThreads + threadIdx.x;
    bool over = false;
    if (sl < n) {
      uint32_t key, at;
      over = !place(sl, &key, &at);
      if (!over) a.buckets[at] = key;
    }
    if (__any_sync(0xffffffffu, over)) over_steps |= 1u << j;
  }
  if (over_steps != 0) args.fill[args.n_ranges] = 1;  // tells the range build that keys repeat
  for (; over_steps != 0; over_steps &= over_steps - 1) {
    const uint32_t sl = (__ffs(over_steps) - 1) * kScatterThreads + threadIdx.x;
    uint32_t key = 0, at;
    const bool over = sl < n && !place(sl, &key, &at);
    __syncwarp();  // the keys are read: their slots are the warp's stage
    insert_overflow<MAGIC>(a, key, over, s_keys + (sl & ~31u), s_draw);
  }
}

// Shared memory of a scatter CTA (dynamic): the tile's keys sorted by range,
// the ranges' counts (then run starts), the ranges' destinations (write_tile_checked
// finds them there).
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
      write_tile_checked<MAGIC>(a, hi - lo, s_keys);
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
  static constexpr bool fits_draws() {
    for (uint32_t g = 0; g < Ops::kS.ng; g++)
      if (Ops::kS.g[g].nbit != Ops::kS.g[0].nbit) return false;
    return Ops::kS.ng * (1 + Ops::kS.g[0].nbit) <= kMaxDraws;
  }
  static_assert(fits_draws(), "RangeArgs::draw holds every layout");
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

  // TEST: bits that are set already take no atomic.
  template <bool TEST>
  __device__ __forceinline__ static void insert(Word* s_w, uint32_t lb, uint32_t key) {
    auto set = [](uint32_t* p, uint32_t m) {
      if (!TEST || (*static_cast<volatile uint32_t*>(p) & m) != m) atomicOr(p, m);
    };
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
        set(p + (bit >> 5), 1u << (bit & 31u));
      } else if constexpr (sizeof(Word) == 8) {
        // 32-bit atomics: 64-bit shared-memory ORs are slower
        const unsigned long long m = Ops::template group_mask<g>(key);
        const uint32_t lo = static_cast<uint32_t>(m), hi = static_cast<uint32_t>(m >> 32);
        if (lo) set(p, lo);
        if (hi) set(p + 1, hi);
      } else {
        set(p, static_cast<uint32_t>(Ops::template group_mask<g>(key)));
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
  const uint32_t rg = blockIdx.x, lane = threadIdx.x & 31u;
  const uint32_t fill = a.fill[rg];
  const uint32_t cnt = fill < a.cap ? fill : a.cap;
  if (cnt == 0) return;
  const bool repeats = a.fill[a.n_ranges] != 0;
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
  for (uint32_t v0 = threadIdx.x & ~31u; v0 * 4 < cnt; v0 += kU * blockDim.x) {
    const uint32_t v = v0 + lane;
    uint4 kv[kU];
#pragma unroll
    for (uint32_t u = 0; u < kU; u++)
      kv[u] = (v + u * blockDim.x) * 4 < cnt ? __ldcs(bk + v + u * blockDim.x) : make_uint4(0, 0, 0, 0);
    // Atomics on the same words wait for one another, loads do not: where
    // neighbours are often equal (copies of some 60 keys or fewer), bits are
    // tested first.
    bool same = false;
    if (repeats) {
#pragma unroll
      for (uint32_t u = 0; u < kU; u++) same |= kv[u].x == kv[u].y || kv[u].y == kv[u].z || kv[u].z == kv[u].w;
    }
    if (repeats && __popc(__ballot_sync(0xffffffffu, same && (v + blockDim.x) * 4 + 3 < cnt)) >= 3) {
      const uint32_t* b32 = reinterpret_cast<const uint32_t*>(bk);
#pragma unroll 4
      for (uint32_t j = 0; j < kU * 4; j++) {
        const uint32_t i = (v + j / 4 * blockDim.x) * 4 + j % 4;
        if (i < cnt) {
          const uint32_t key = __ldg(b32 + i);
          R::template insert<true>(s_w, block_index(key * mul_const(0), a.addr) - blk0, key);
        }
      }
      continue;
    }
#pragma unroll
    for (uint32_t u = 0; u < kU; u++) {
      const uint32_t k[4] = {kv[u].x, kv[u].y, kv[u].z, kv[u].w};
#pragma unroll
      for (uint32_t q = 0; q < 4; q++) {
        if ((v + u * blockDim.x) * 4 + q < cnt)
          R::template insert<false>(s_w, block_index(k[q] * mul_const(0), a.addr) - blk0, k[q]);
      }
    }
  }
  __syncthreads();
  R::or_out(gw, s_w, nw);
}

#endif  // __CUDACC__

}  // namespace dtlg
