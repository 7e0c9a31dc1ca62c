// cuckoo.cuh -- partial-key cuckoo filter probe and build.
//
// Reference: cuckoofilter_logic.hpp:119-521 and cuckoofilter_table.hpp:67-277.
// Table layout (identical bytes): buckets of ceil(T*B/8) bytes, tag j of a
// bucket at bit T*j (little endian), tag 0 = empty; the victim record
// {u32 index, u32 tag, bool used} follows the table at 32-bit word
// ceil(bytes/4) (cuckoofilter_logic.hpp:131-157).
//
// Probe: bit-exact with the reference (the reference's SWAR bucket tests,
// cuckoofilter_table_scalar.hpp:48-83, are exact existence tests).
//
// Build: the reference inserts one key at a time and picks kick slots with a
// thread-local mt19937 seeded from std::random_device (cuckoofilter_table.hpp:
// 197, thread.hpp:72-78), so no two of its builds agree.  The GPU build runs
// the same bounded-kick partial-key algorithm for all keys at once, each key
// starting in the emptier of its two buckets.  Buckets that are a whole 16-,
// 32- or 64-bit word are updated in the table itself, one compare-and-swap per
// step; the others on an unpacked copy (one 32-bit slot per tag), which is
// packed back afterwards.  Checked by invariants (no false negatives,
// occupancy) and FPR.
#pragma once

#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "probe.cuh"

namespace dtlg {

constexpr uint32_t kAltMul = 0x5bd1e995u;  // cuckoofilter_logic.hpp:222,246
constexpr uint32_t kMaxKicks = 500;        // cuckoofilter_logic.hpp:122

template <int T, int B>
struct CuckooCfg {
  static constexpr int kT = T, kB = B;
  static constexpr int kBytesPerBucket = (T * B + 7) / 8;
  // the bucket is one 16-, 32- or 64-bit word of the table
  static constexpr bool kWordBucket = kBytesPerBucket == 2 || kBytesPerBucket == 4 || kBytesPerBucket == 8;
  static constexpr uint32_t kTagMask = T == 32 ? 0xffffffffu : ((1u << T) - 1u);
};

struct CuckooBuildArgs {
  uint32_t* table;          // packed table (32-bit words) + victim record
  uint32_t* slots;          // unpacked: (bucket_cnt + 1) * B slots (buckets that are no word)
  const uint32_t* keys_al;
  uint64_t n_phys;
  uint32_t pre;
  uint64_t table_words;     // 32-bit words of the packed table
  uint64_t victim_word;
  Addr addr;
  unsigned long long* failed;  // keys whose tag could not be placed
  uint64_t seed;
};

#ifdef __CUDACC__

// Alternate bucket (cuckoofilter_logic.hpp:214-252).  The MAGIC form yields
// bucket_cnt (one past the end) for i == 0 and tag*M mod c == 0; the reference
// then reads the bytes after the table, and so does the probe here.
__device__ __forceinline__ uint32_t cuckoo_alt(uint32_t i, uint32_t tag, const Addr& a) {
  if (!a.magic_mode) return (i ^ (tag * kAltMul)) & a.block_cnt_mask;
  const uint32_t c = a.divisor;
  const uint32_t s = block_index(tag * kAltMul, a);
  const uint32_t x = c - s;
  return (x < i ? c : 0u) + (x - i);
}

template <class Cfg>
struct CuckooOps {
  static constexpr int kT = Cfg::kT, kB = Cfg::kB, kBPB = Cfg::kBytesPerBucket;

  __device__ __forceinline__ static void index_tag(uint32_t key, const Addr& a, uint32_t& i1,
                                                   uint32_t& tag) {
    i1 = block_index(key * mul_const(0), a);         // cuckoofilter_logic.hpp:205
    tag = (key * mul_const(1)) & Cfg::kTagMask;       // :183, :206
    tag += (tag == 0u);                          // :184
  }

  // A bucket's bytes, read with aligned loads: one word, or the two aligned
  // 32-bit words that hold a bucket of 1, 2, 3 or 6 bytes and the bucket's
  // first bit in them.
  struct Bucket {
    unsigned long long x = 0;
    unsigned long long y = 0;  // buckets of 16 bytes: the second half
    uint32_t sh = 0;
  };
  __device__ __forceinline__ static Bucket load(const void* table, uint32_t i) {
    const uint64_t o = static_cast<uint64_t>(i) * kBPB;
    const unsigned char* t8 = static_cast<const unsigned char*>(table);
    Bucket b;
    if constexpr (kBPB == 16) {
      const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(t8 + o));
      b.x = v.x;
      b.y = v.y;
    } else if constexpr (kBPB == 8) {
      b.x = __ldg(reinterpret_cast<const unsigned long long*>(t8 + o));
    } else if constexpr (kBPB == 4) {
      b.x = __ldg(reinterpret_cast<const unsigned int*>(t8 + o));
    } else {
      const uint64_t a4 = o & ~3ull;
      b.sh = static_cast<uint32_t>(o & 3u) * 8u;
      const unsigned int* w = reinterpret_cast<const unsigned int*>(t8 + a4);
      b.x = __ldg(w);
      if constexpr (kBPB > 2) b.x |= static_cast<unsigned long long>(__ldg(w + 1)) << 32;
    }
    return b;
  }
  // Does the bucket hold `tag`?  A Bucket{} holds none (no tag is 0).
  __device__ __forceinline__ static bool holds(const Bucket& b, uint32_t tag) {
    bool hit = false;
#pragma unroll
    for (int j = 0; j < kB; j++) {
      const unsigned long long x = kBPB == 16 && j >= kB / 2 ? b.y : b.x;
      const int at = kBPB == 16 ? kT * (j % (kB / 2 > 0 ? kB / 2 : 1)) : kT * j;
      hit |= (static_cast<uint32_t>(x >> (b.sh + at)) & Cfg::kTagMask) == tag;
    }
    return hit;
  }

  // The bitmask kernel of 4 CTAs per SM tests keys together too.  Buckets of 16
  // bytes gain from that at 6 CTAs only, and the second path in the kernel cost
  // the first one 2 % (t=32 b=4, 64 KiB).
  static constexpr bool kTogetherAt4 = kBPB != 16;

  // cuckoofilter_logic.hpp:346-362 for N keys at once: the buckets of all of
  // them are loaded before any is tested.  One key after the other, each
  // bucket behind a branch of its own, a thread had one load in flight, and
  // the probe ran at the loads' latency.  Bit q of the result: key q matches.
  template <int N>
  __device__ __forceinline__ static uint32_t contains_n(const ProbeArgs& a, const uint32_t (&key)[N]) {
    uint32_t i1[N], i2[N], tag[N];
    Bucket b1[N], b2[N];
#pragma unroll
    for (int q = 0; q < N; q++) {
      index_tag(key[q], a.addr, i1[q], tag[q]);
      i2[q] = cuckoo_alt(i1[q], tag[q], a.addr);
      if (!a.range_on) {
        b1[q] = load(a.filter, i1[q]);
        b2[q] = load(a.filter, i2[q]);
      } else {
        // block-range pass: only the buckets this pass owns (the result is the
        // OR over all passes)
        if (i1[q] >= a.blk_lo && i1[q] < a.blk_hi) b1[q] = load(a.filter, i1[q]);
        if (i2[q] >= a.blk_lo && i2[q] < a.blk_hi) b2[q] = load(a.filter, i2[q]);
      }
    }
    const unsigned int* v = static_cast<const unsigned int*>(a.filter) + a.victim_word;
    const uint32_t vi = __ldg(v), vt = __ldg(v + 1), vu = __ldg(v + 2) & 0xffu;
    uint32_t hits = 0;
#pragma unroll
    for (int q = 0; q < N; q++) {
      const bool in_victim = vu && tag[q] == vt && (i1[q] == vi || i2[q] == vi);
      hits |= (in_victim | holds(b1[q], tag[q]) | holds(b2[q], tag[q]) ? 1u : 0u) << q;
    }
    return hits;
  }
  // One key.  Buckets of 16 bytes are tested one after the other: both in
  // registers at once cost 3 % (2^26 probes, 64 KiB: 250 us against 256).
  __device__ __forceinline__ static bool contains(const ProbeArgs& a, uint32_t key) {
    if constexpr (kBPB == 16) {
      uint32_t i1, tag;
      index_tag(key, a.addr, i1, tag);
      const uint32_t i2 = cuckoo_alt(i1, tag, a.addr);
      const unsigned int* v = static_cast<const unsigned int*>(a.filter) + a.victim_word;
      const uint32_t vi = __ldg(v), vt = __ldg(v + 1), vu = __ldg(v + 2) & 0xffu;
      const bool in_victim = vu && tag == vt && (i1 == vi || i2 == vi);
      if (a.range_on) {
        const bool r1 = i1 >= a.blk_lo && i1 < a.blk_hi, r2 = i2 >= a.blk_lo && i2 < a.blk_hi;
        return in_victim | (r1 && holds(load(a.filter, i1), tag)) | (r2 && holds(load(a.filter, i2), tag));
      }
      return in_victim | holds(load(a.filter, i1), tag) | holds(load(a.filter, i2), tag);
    } else {
      const uint32_t k[1] = {key};
      return contains_n<1>(a, k) != 0u;
    }
  }

  // cuckoofilter_table.hpp:111-136: tag j of bucket i from the packed table.
  __device__ __forceinline__ static uint32_t read_tag(const uint32_t* table, uint64_t i, int j) {
    const uint64_t bit = i * (kBPB * 8ull) + static_cast<uint64_t>(kT) * j;
    const uint64_t w = bit >> 5;
    const uint32_t sh = static_cast<uint32_t>(bit & 31u);
    unsigned long long x = table[w];
    if (sh + kT > 32) x |= static_cast<unsigned long long>(table[w + 1]) << 32;
    return static_cast<uint32_t>(x >> sh) & Cfg::kTagMask;
  }
};

template <class Cfg>
__global__ void cuckoo_unpack_kernel(const uint32_t* table, uint32_t* slots, uint32_t bucket_cnt) {
  const uint64_t n = static_cast<uint64_t>(bucket_cnt) * Cfg::kB;
  for (uint64_t s = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; s < n;
       s += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    slots[s] = CuckooOps<Cfg>::read_tag(table, s / Cfg::kB, static_cast<int>(s % Cfg::kB));
  }
}

__device__ __forceinline__ uint32_t kick_rand(uint64_t& s) {  // xorshift64* (Vigna 2014)
  s ^= s >> 12;
  s ^= s << 25;
  s ^= s >> 27;
  return static_cast<uint32_t>((s * 2685821657736338717ull) >> 32);
}

__device__ __forceinline__ unsigned short bucket_cas(unsigned short* p, unsigned short c, unsigned short v) {
  return atomicCAS(p, c, v);
}
__device__ __forceinline__ unsigned int bucket_cas(unsigned int* p, unsigned int c, unsigned int v) {
  return atomicCAS(p, c, v);
}
__device__ __forceinline__ unsigned long long bucket_cas(unsigned long long* p, unsigned long long c,
                                                         unsigned long long v) {
  return atomicCAS(p, c, v);
}

// Buckets that are one word of the packed table.  A bucket's value is what a
// load or a lost compare-and-swap last saw.
template <class Cfg>
struct WordBuckets {
  static constexpr int kT = Cfg::kT, kB = Cfg::kB;
  using Word = typename std::conditional<Cfg::kBytesPerBucket == 8, unsigned long long,
                                         typename std::conditional<Cfg::kBytesPerBucket == 4, unsigned int,
                                                                   unsigned short>::type>::type;
  using Value = Word;
  __device__ __forceinline__ static Word* at(const CuckooBuildArgs& a, uint32_t i) {
    return reinterpret_cast<Word*>(a.table) + i;
  }
  __device__ __forceinline__ static Value load(const CuckooBuildArgs& a, uint32_t i) { return __ldcg(at(a, i)); }
  __device__ __forceinline__ static uint32_t tag_of(Value v, int j) {
    return static_cast<uint32_t>(v >> (kT * j)) & Cfg::kTagMask;
  }
  __device__ __forceinline__ static uint32_t free_slots(const Value& v) {
    uint32_t n = 0;
#pragma unroll
    for (int j = 0; j < kB; j++) n += tag_of(v, j) == 0u;
    return n;
  }
  // The shift of the first empty slot, -1 when the bucket is full.
  __device__ __forceinline__ static int empty_slot(const Value& v) {
    int sh = -1;
#pragma unroll
    for (int j = kB - 1; j >= 0; j--)
      if (tag_of(v, j) == 0u) sh = kT * j;
    return sh;
  }
  // The tag into an empty slot of bucket i, false when it is full (or after
  // kRaces lost races: the key then goes on to its other bucket).
  static constexpr int kRaces = 64;
  __device__ __forceinline__ static bool insert(const CuckooBuildArgs& a, uint32_t i, Value& v, uint32_t tag) {
    for (int n = 0; n < kRaces; n++) {
      const int sh = empty_slot(v);
      if (sh < 0) return false;
      const Word seen = bucket_cas(at(a, i), v, static_cast<Word>(v | static_cast<Word>(tag) << sh));
      if (seen == v) return true;
      v = seen;
    }
    return false;
  }
  // Swaps the tag with the one in slot r and returns that; 0: it went into an
  // empty slot.  Equal tags need no swap: thousands of copies of one key, more
  // than its buckets can hold, must not fight over the two words.
  __device__ __forceinline__ static uint32_t kick(const CuckooBuildArgs& a, uint32_t i, Value& v, uint32_t tag,
                                                  uint32_t r) {
    for (int n = 0; n < kRaces; n++) {
      if (insert(a, i, v, tag)) return 0u;
      const uint32_t old = tag_of(v, static_cast<int>(r));
      if (old == tag || old == 0u) break;
      const Word seen =
          bucket_cas(at(a, i), v, static_cast<Word>(v ^ static_cast<Word>(old ^ tag) << (kT * r)));
      if (seen == v) return old;
      v = seen;
    }
    return tag;
  }
};

// Buckets of one 32-bit slot per tag in the unpacked copy.
template <class Cfg>
struct SlotBuckets {
  static constexpr int kB = Cfg::kB;
  struct Value {
    uint32_t tag[kB];
  };
  __device__ __forceinline__ static uint32_t* at(const CuckooBuildArgs& a, uint32_t i) {
    return a.slots + static_cast<uint64_t>(i) * kB;
  }
  __device__ __forceinline__ static Value load(const CuckooBuildArgs& a, uint32_t i) {
    Value v;
    if constexpr (kB == 4) {
      const uint4 x = __ldcg(reinterpret_cast<const uint4*>(at(a, i)));
      v.tag[0] = x.x; v.tag[1] = x.y; v.tag[2] = x.z; v.tag[3] = x.w;
    } else {
#pragma unroll
      for (int j = 0; j < kB; j++) v.tag[j] = __ldcg(at(a, i) + j);
    }
    return v;
  }
  __device__ __forceinline__ static uint32_t tag_of(const Value& v, int j) { return v.tag[j]; }
  __device__ __forceinline__ static uint32_t free_slots(const Value& v) {
    uint32_t n = 0;
#pragma unroll
    for (int j = 0; j < kB; j++) n += v.tag[j] == 0u;
    return n;
  }
  __device__ __forceinline__ static bool insert(const CuckooBuildArgs& a, uint32_t i, Value& v, uint32_t tag) {
    bool done = false;
#pragma unroll
    for (int j = 0; j < kB; j++) {
      if (!done && v.tag[j] == 0u) {
        v.tag[j] = atomicCAS(at(a, i) + j, 0u, tag);
        done = v.tag[j] == 0u;
      }
    }
    return done;
  }
  __device__ __forceinline__ static uint32_t kick(const CuckooBuildArgs& a, uint32_t i, Value& v, uint32_t tag,
                                                  uint32_t r) {
    bool same = false;  // equal tags need no swap (see WordBuckets::kick)
#pragma unroll
    for (int j = 0; j < kB; j++) same |= static_cast<uint32_t>(j) == r && v.tag[j] == tag;
    return same ? tag : atomicExch(at(a, i) + r, tag);
  }
};

// cuckoofilter_logic.hpp:292-322 for one key.  The reference tries bucket 1,
// then bucket 2; here both are loaded at once and the emptier one is tried
// first, which keeps the buckets level.
template <class Cfg, class S>
__device__ __forceinline__ void cuckoo_insert_key(const CuckooBuildArgs& a, uint32_t key, uint64_t pos) {
  constexpr int kB = Cfg::kB;
  const uint32_t c = a.addr.block_cnt;  // bucket c lies past the table: never written here
  uint32_t cur, tag;
  CuckooOps<Cfg>::index_tag(key, a.addr, cur, tag);
  uint32_t other = cuckoo_alt(cur, tag, a.addr);
  typename S::Value v = S::load(a, cur), w = S::load(a, other < c ? other : cur);
  if (other < c && S::free_slots(w) > S::free_slots(v)) {
    const uint32_t i = cur;
    cur = other;
    other = i;
    const typename S::Value x = v;
    v = w;
    w = x;
  }
  bool done = S::insert(a, cur, v, tag);
  if (!done) {
    cur = other;
    if (cur < c) done = S::insert(a, cur, w, tag);
    v = w;
  }
  uint64_t rng = a.seed ^ (0x9E3779B97F4A7C15ull * (pos + 1));
  // `cur` was full when last seen (as v).  A kick takes a slot whose tag has
  // room in its other bucket, if there is one (all of them are looked at at
  // once), else a random one: the kernel ends with its longest chain of kicks.
  auto kick = [&](auto look) {
    if (cur < c) {
      uint32_t r = kick_rand(rng) % kB;
      if constexpr (decltype(look)::value) {
        uint32_t to[kB];
        typename S::Value x[kB];
#pragma unroll
        for (int j = 0; j < kB; j++) {
          to[j] = cuckoo_alt(cur, S::tag_of(v, j), a.addr);
          x[j] = S::load(a, to[j] < c ? to[j] : cur);
        }
        const uint32_t at = r;
#pragma unroll
        for (int j = 0; j < kB; j++) {
          // not always the first with room: keys that kick from one bucket at
          // the same time then pick different slots
          if (to[j] < c && S::free_slots(x[j]) != 0u && (r == at || static_cast<uint32_t>(j) < at)) r = j;
        }
      }
      const uint32_t old = S::kick(a, cur, v, tag, r);
      if (old == 0u) {
        done = true;
        return;
      }
      tag = old;
    }
    cur = cuckoo_alt(cur, tag, a.addr);
    if (cur < c) {
      v = S::load(a, cur);
      done = S::insert(a, cur, v, tag);
    }
  };
  // Once a key is lost, the table is full and looking ahead only costs (twice
  // the keys that fit, t=16 b=4: 21.0 ms throughout, 13.0 for 16 kicks only, but
  // these lose 300 of 200 000 keys at load 0.97 that it places).
  uint32_t count = 0;
  for (; count < kMaxKicks && !done; count++) {
    if ((count & 15u) == 15u && __ldcg(a.failed) != 0) break;
    kick(std::true_type{});
  }
  for (; count < kMaxKicks && !done; count++) kick(std::false_type{});
  if (!done) {
    // victim cache (cuckoofilter_logic.hpp:318-320); when it is taken the
    // tag in hand is lost, the reference's `insert == false`.
    uint32_t* vr = a.table + a.victim_word;
    if (atomicCAS(vr + 2, 0u, 1u) == 0u) {
      vr[0] = cur;
      vr[1] = tag;
    } else {
      atomicAdd(a.failed, 1ull);
    }
  }
}

// All keys in parallel, one per thread.  Bound by the chains of dependent L2
// round trips (key, buckets, compare-and-swap, then the kicks of the few keys
// that find both buckets full) and by the longest of them; four keys per
// thread with their loads and first swaps in flight together was slower (129
// against 103 us: the buckets are chosen on older counts, so more keys kick).
// t=16 b=4, 3 000 001 keys at load 0.9: 199 us with unpack, pack and random
// kicks, about 100 us so; 2^26 keys at load 0.95 7.4 -> 2.8 ms.
template <class Cfg>
__global__ void __launch_bounds__(256) cuckoo_insert_kernel(const __grid_constant__ CuckooBuildArgs a) {
  using S = typename std::conditional<Cfg::kWordBucket, WordBuckets<Cfg>, SlotBuckets<Cfg>>::type;
  for (uint64_t p = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; p < a.n_phys;
       p += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    if (p >= a.pre) cuckoo_insert_key<Cfg, S>(a, __ldg(a.keys_al + p), p);
  }
}

// Packs the slot array back into the reference's byte layout, one 32-bit
// output word per thread; bits outside tags keep their old value.
template <class Cfg>
__global__ void cuckoo_pack_kernel(uint32_t* table, const uint32_t* slots, uint32_t bucket_cnt,
                                   uint64_t table_words) {
  constexpr int kT = Cfg::kT, kB = Cfg::kB, kBPB = Cfg::kBytesPerBucket;
  for (uint64_t w = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; w < table_words;
       w += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint64_t b0 = (w * 4) / kBPB;
    uint64_t b1 = (w * 4 + 3) / kBPB;
    if (b1 >= bucket_cnt) b1 = bucket_cnt - 1;
    unsigned long long bits = 0, mask = 0;
    for (uint64_t bb = b0; bb <= b1; bb++) {
#pragma unroll
      for (int j = 0; j < kB; j++) {
        const int64_t rel = static_cast<int64_t>(bb * kBPB * 8 + static_cast<uint64_t>(kT) * j) -
                            static_cast<int64_t>(w * 32);
        const unsigned long long tv = slots[bb * kB + j] & Cfg::kTagMask;
        const unsigned long long tm = Cfg::kTagMask;
        if (rel >= 32 || rel <= -kT) continue;
        if (rel >= 0) {
          bits |= tv << rel;
          mask |= tm << rel;
        } else {
          bits |= tv >> (-rel);
          mask |= tm >> (-rel);
        }
      }
    }
    const uint32_t m32 = static_cast<uint32_t>(mask);
    table[w] = (table[w] & ~m32) | (static_cast<uint32_t>(bits) & m32);
  }
}

template <class Cfg>
__global__ void cuckoo_count_kernel(const uint32_t* table, uint32_t bucket_cnt, uint64_t victim_word,
                                    unsigned long long* count) {
  unsigned long long c = 0;
  const uint64_t n = static_cast<uint64_t>(bucket_cnt) * Cfg::kB;
  for (uint64_t s = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; s < n;
       s += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    c += CuckooOps<Cfg>::read_tag(table, s / Cfg::kB, static_cast<int>(s % Cfg::kB)) != 0u;
  }
  for (int d = 16; d > 0; d >>= 1) c += __shfl_xor_sync(0xffffffffu, c, d);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
  if (blockIdx.x == 0 && threadIdx.x == 0 && (table[victim_word + 2] & 0xffu)) atomicAdd(count, 1ull);
}

#endif  // __CUDACC__

}  // namespace dtlg
