// api.cu -- the C ABI of libdtlg.so (include/dtlg.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/dtlg.h"
#include "filter_handle.hpp"
#include "host_config.hpp"
#include "registry.hpp"
#include "result_slot.hpp"

using namespace dtlg;

namespace dtlg {

// ---- registry ----------------------------------------------------------------
static std::vector<BloomKernels>& bloom_table() {
  static std::vector<BloomKernels> t;
  return t;
}
static std::vector<CuckooKernels>& cuckoo_table() {
  static std::vector<CuckooKernels> t;
  return t;
}
static std::vector<BcfKernels>& bcf_table() {
  static std::vector<BcfKernels> t;
  return t;
}
void register_bloom(const BloomKernels& k) { bloom_table().push_back(k); }
void register_cuckoo(const CuckooKernels& k) { cuckoo_table().push_back(k); }
void register_bcf(const BcfKernels& k) { bcf_table().push_back(k); }
static std::vector<ClassicKernels>& classic_table() {
  static std::vector<ClassicKernels> t;
  return t;
}
void register_classic(const ClassicKernels& k) { classic_table().push_back(k); }
const ClassicKernels* find_classic() { return classic_table().empty() ? nullptr : &classic_table()[0]; }
const BcfKernels* find_bcf(uint32_t t, uint32_t a) {
  for (const auto& e : bcf_table())
    if (e.t == t && e.a == a) return &e;
  return nullptr;
}
const BloomKernels* find_bloom(uint32_t wb, uint32_t w, uint32_t s, uint32_t z, uint32_t k) {
  for (const auto& e : bloom_table())
    if (e.word_bytes == wb && e.w == w && e.s == s && e.z == z && e.k == k) return &e;
  return nullptr;
}
const CuckooKernels* find_cuckoo(uint32_t t, uint32_t b) {
  for (const auto& e : cuckoo_table())
    if (e.t == t && e.b == b) return &e;
  return nullptr;
}
int registered_bloom_count() { return static_cast<int>(bloom_table().size()); }

// ---- per-device state ----------------------------------------------------------
namespace {
thread_local std::string g_last_cuda_error;

struct DeviceState {
  bool init = false;
  int sms = 0;
  cudaMemPool_t pool = nullptr;
  ResultSlots slots;
};
std::mutex g_mu;
DeviceState g_dev[64];

dtlg_status cuda_fail(cudaError_t e) {
  g_last_cuda_error = cudaGetErrorString(e);
  return DTLG_ERR_CUDA;
}

#define DTLG_CUDA(x)                         \
  do {                                       \
    cudaError_t _e = (x);                    \
    if (_e != cudaSuccess) return cuda_fail(_e); \
  } while (0)

dtlg_status device_state(DeviceState** out) {
  int dev = 0;
  DTLG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return DTLG_ERR_CUDA;
  std::lock_guard<std::mutex> lk(g_mu);
  DeviceState& s = g_dev[dev];
  if (!s.init) {
    DTLG_CUDA(cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, dev));
    // A library-private stream-ordered pool for per-call workspaces; it keeps
    // its memory between calls instead of returning it at every sync.
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    DTLG_CUDA(cudaMemPoolCreate(&s.pool, &props));
    uint64_t thr = ~0ull;
    DTLG_CUDA(cudaMemPoolSetAttribute(s.pool, cudaMemPoolAttrReleaseThreshold, &thr));
    s.init = true;
  }
  *out = &s;
  return DTLG_OK;
}

// Workspace of one probe call: header (tile counter, error word, count) then
// one look-back status word per tile.
struct WsHeader {
  unsigned int tile_ctr;
  unsigned int err;
  unsigned long long count;
  unsigned int done;
  unsigned int pad[27];
};
static_assert(sizeof(WsHeader) == 128, "header is one 128-byte line");

// Status words of the fused plan for up to n_phys keys: those of its largest
// tiles, or of its smallest where these are used (a bound that never falls as
// n_phys grows, so a workspace sized for more keys always serves fewer).
uint64_t probe_tiles(uint64_t n_phys) {
  return std::max<uint64_t>((n_phys + kProbeTile - 1) / kProbeTile,
                            std::min<uint64_t>((n_phys + 1023) / 1024, kFusedSumTiles));
}
static_assert(kFusedOneKey <= kFusedOneRound && (kFusedOneRound + 1023) / 1024 <= kFusedSumTiles,
              "the status words hold one word per tile of every shape");

// Two-pass layout inside the same workspace: header | status words | bitmask.
constexpr uint64_t kTwoPassMinKeys = 1ull << 20;
uint64_t bits_words(uint64_t n_phys) { return (n_phys + 31) / 32; }
uint32_t compact_tiles(uint64_t n_phys) {
  const uint64_t words = bits_words(n_phys), tile = kCompactThreads * compact_rows(words);
  return static_cast<uint32_t>((words + tile - 1) / tile);
}
size_t status_bytes(uint64_t n_phys) {
  // as probe_tiles: a bound that never falls as n_phys grows
  const uint64_t words = bits_words(n_phys);
  const uint64_t c = std::max<uint64_t>((words + kCompactThreads * 8 - 1) / (kCompactThreads * 8),
                                        std::min<uint64_t>((words + kCompactThreads - 1) / kCompactThreads, kCompactSumTiles));
  return static_cast<size_t>(((std::max(probe_tiles(n_phys), c) * 8 + 255) / 256) * 256);
}
size_t round256(uint64_t b) { return static_cast<size_t>(((b + 255) / 256) * 256); }
uint32_t part_tiles(uint64_t n_phys) { return static_cast<uint32_t>((n_phys + kPartTile - 1) / kPartTile); }

// Workspace: header | status words | match bitmask | [partitioned probe:
// partition header (range fill counters) | per-tile overflow masks |
// (key, position) pairs in one segment per range]
struct WsLayout {
  size_t bits_off, part_off, tflags_off, pairs_off, total_small, total;
};
WsLayout ws_layout(uint64_t n_phys) {
  WsLayout l{};
  l.bits_off = sizeof(WsHeader) + status_bytes(n_phys);
  l.part_off = l.bits_off + round256(bits_words(n_phys) * 4);
  l.total_small = l.part_off;
  l.tflags_off = l.part_off + kPartHeaderBytes;
  l.pairs_off = l.tflags_off + round256(static_cast<uint64_t>(part_tiles(n_phys)) * 8);
  l.total = l.pairs_off + round256(part_pair_capacity(n_phys) * 8 + 16);
  return l;
}
size_t workspace_bytes(uint64_t n_phys) { return ws_layout(n_phys).total; }

int compact_occupancy() {
  static int occ = [] {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, compact_kernel<8>, kCompactThreads, 0);
    return std::max(1, n);
  }();
  return occ;
}

// Block-range passes of the two-pass probe.  Random probes over more than
// ~256 MiB of filter run out of the GPU's address-translation reach (B200: the
// probe rate falls from ~62 to ~25 Gkeys/s between 256 and 512 MiB), so larger
// filters are probed in passes of about 256 MiB each; filters up to 160 MiB
// take one pass.  dtlg_set_probe_passes overrides the choice.
uint32_t probe_passes(const dtlg_filter* f) {
  // a classic Bloom key's k words lie anywhere in the filter, and a key
  // matches only if all are set: its probe cannot be split by word range
  if (f->qk) return 1;
  const uint64_t bytes = (f->d.m_actual + 7) / 8;
  uint64_t r = f->probe_passes;
  if (r == 0 && f->ck) {
    // Cuckoo buckets are 1-16 bytes but an L2 miss fills 64 bytes, so a table
    // beyond L2 wastes most of its DRAM traffic: probe it in passes whose
    // bucket range (<= 72 MiB) stays in the 126 MB L2.  B200, t=16 b=4,
    // 141 MB table, 2^28 probes: 1 pass 52.3, 2 passes 81.4, 3 passes 64.9 Gkeys/s.
    r = bytes <= (64ull << 20) ? 1 : (bytes + (72ull << 20) - 1) / (72ull << 20);
  } else if (r == 0) {
    r = bytes <= (160ull << 20) ? 1 : std::max<uint64_t>(2, (bytes + (128ull << 20)) / (256ull << 20));
  }
  r = std::min<uint64_t>(r, 16);
  r = std::min<uint64_t>(r, std::max<uint32_t>(1, f->d.addr.block_cnt));
  return static_cast<uint32_t>(std::max<uint64_t>(1, r));
}

dtlg_status check_filter_ptr(const void* p) {
  if (!p) return DTLG_ERR_NULL;
  if (reinterpret_cast<uintptr_t>(p) & 15u) return DTLG_ERR_ALIGNMENT;
  return DTLG_OK;
}

// Probe kernel plan for n keys: 1 = fused (probe + ordered compaction in one
// kernel), 2 = match bitmask in block-range passes + compaction,
// 3 = partitioned probe (Bloom and blocked cuckoo filters: one block per key)
// + compaction, 4 = match bitmask against a shared-memory copy of a filter of
// at most kSmemMaxBytes (Bloom and classic Bloom filters) + compaction.
// Automatic choice (measured on B200, u64 w=8 s=8 k=8, 2^26-2^28 probes):
// below 2^20 keys the single fused kernel; Bloom filters above 160 MiB the
// partitioned probe (256 MiB: 68.6 vs 62.5 Gkeys/s; 512 MiB: 64 vs 54); else
// the bitmask kernel (L2-resident filters: 113 vs 76 Gkeys/s partitioned).
// Plan 4 is offered up to kSmemMaxBytes (below every sm_100 opt-in limit,
// 227 KiB) but never chosen automatically: on B200 a small filter read through
// L1 probes faster than a shared-memory copy (64 KiB u64 w=8 s=8 k=8 filter,
// 2^28 probes: 141.5 Gkeys/s plan 2, 101.5 plan 4 -- random 16-byte shared
// loads conflict on banks, L1 hits do not).  The autotuner times it.
constexpr uint64_t kSmemMaxBytes = 192ull << 10;
// Filters larger than this take the L1 no-allocate loads in plan 2 (B200,
// u64 w=8 s=8 k=8, 2^28 probes, allocating: 128 KiB 155, 256 KiB 126, 512 KiB
// 112 Gkeys/s; not allocating, 1-8 MiB: 128.7).
constexpr uint64_t kL1NoAllocBytes = 256ull << 10;

// Filters just beyond the single-pass limit that are probed by the bitmask
// plan in its block-range passes: layouts of 64-byte blocks whose words the
// hash picks among four or more, smaller blocks that pick from all of their
// words, u32 of one or two words per block, and zoned u32 z=2.  us for 2^26
// probes, bitmask (8 CTAs per SM) / partitioned:
//   MiB                 168      184      200      208      224      256
//   u32 w=16 s=1 k=4    581/661  611/666  644/671  660/673  682/667  741/649
//   u32 w=16 s=2 k=4    584/611  619/628  650/628  671/642
//   u64 w=8 s=1 k=4     607/669  632/674  661/678  675/682  690/675
//   u64 w=8 s=2         843/832  864/845  870/847  880/859  861/836
//   zoned u32 w=16 z=2  587/569  625/591  654/593
//   u32 w=1 k=4         494/534  544/538  590/539      (176: 518/539)
//   u32 w=2 s=2 k=8     516/532  554/533               (176: 534/532)
//   u32 w=2, w=4 s=1    556/601  583/604  615/601
//   u64 w=2 s=1 k=4     582/618  601/616  626/616
// u64 w=8 s=2, zoned u32 and the largest u32 w=16 s=1 filters would be 1 to 14 %
// faster partitioned; they stay here, as the ABI tests have it, with an eighth of
// a byte of workspace per key instead of 8.3.  The others are partitioned from 160
// MiB on (at 168 MiB, 2^27 probes: u64 w=8 s=4 1878/1230, u32 w=16 s=8 1357/1178,
// u64 w=1 1244/1020, zoned u32 w=16 z=4 1241/1174; 2^26: u32 w=4 s=4 546/534).
bool bitmask_band(const dtlg_filter* f) {
  if (f->d.kind != Kind::kBloom && f->d.kind != Kind::kZoned) return false;
  const uint64_t fbytes = (f->d.m_actual + 7) / 8;
  if (fbytes <= (160ull << 20)) return false;
  // the limits leave room for MAGIC sizes, which round a request up
  const bool u32 = f->d.word_bytes == 4;
  if (f->d.kind == Kind::kZoned) return u32 && f->d.z == 2 && fbytes <= (200ull << 20);
  if (f->d.w * f->d.word_bytes == 64 && f->d.s * 4 <= f->d.w)
    return fbytes <= (u32 && f->d.s == 1 ? 264ull << 20 : 210ull << 20);
  if (f->d.s == 1 && f->d.w > 1) return fbytes <= (194ull << 20);
  return u32 && f->d.w <= 2 && f->d.s == f->d.w && fbytes <= (f->d.w == 1 ? 182ull << 20 : 176ull << 20);
}

int probe_plan(const dtlg_filter* f, uint64_t n) {
  int mode = f->probe_mode;
  const bool partitioned = f->pk->probe_pairs[0] != nullptr;
  const uint64_t fbytes = (f->d.m_actual + 7) / 8;
  const bool smem = f->pk->probe_smem != nullptr && fbytes <= kSmemMaxBytes;
  if (mode == 3 && !partitioned) mode = 2;
  if (mode == 4 && !smem) mode = 2;
  if (mode == 0) {
    if (n < kTwoPassMinKeys) {
      mode = 1;
    } else if (bitmask_band(f)) {
      mode = 2;
    } else {
      mode = (partitioned && fbytes > (160ull << 20)) ? 3 : 2;
    }
  }
  return mode;
}

// Cuckoo probes: keys tested one by one or together (contains_n), at 6 CTAs per
// SM (variant 0) or 4 (1).  Tables that hit L1 on part of the loads only are
// probed key by key at 4 CTAs: with more loads in flight the lines are gone
// before they are used again.  us for 2^26 probes, 0 one by one / 0 together / 1
// one by one / 1 together:
//          16 KiB           200 KiB          320 KiB          512 KiB          64 MiB
//   16/4   254/256/251/258  265/269/285/279  423/413/390/385  448/436/448/451  549/536/536/564
//   16/1   251/253/243/247  261/261/274/264  407/421/398/381  438/430/455/463  544/530/537/564
//   8/4    268/268/262/266  285/277/293/276  422/421/394/385  442/430/443/454  548/532/537/533
//   4/4    341/342/342/346  363/353/363/354  445/440/397/419  470/457/476/500  578/560/568/601
//   12/4   361/361/357/381  415/402/411/420  498/495/496/491  581/580/573/559  695/691/674/649
//   32/2   219/222/218/230  250/252/256/261  396/414/400/374  441/433/449/441  551/536/537/560
//   32/4   276/280/246/262  314/328/281/292  430/443/401/418  492/497/444/464  608/602/528/570
// In two passes (beyond 64 MiB) more of the loads miss L2, and variant 0 with the
// keys together is ahead: 16/4 at 146 MiB 853/841/979/888, 12/4 1057/1043/1122/1074;
// buckets of 16 bytes from 120 MiB on (98 MiB 679/674/664/667, 146 MiB 834/800/942/831).
struct CuckooForm {
  int variant;
  bool together;
};
CuckooForm cuckoo_form(const dtlg_filter* f) {
  const uint64_t kib = f->d.m_actual >> 13;
  const uint32_t t = f->d.t;
  const bool two_pass = probe_passes(f) > 1;
  if (t * f->d.b == 128) return two_pass && kib >= (120u << 10) ? CuckooForm{0, true} : CuckooForm{1, false};
  if (two_pass) return {0, true};
  if (kib >= 480) return {t == 12 ? 1 : 0, true};
  if (kib >= 160 && kib < 230 && t != 12 && t != 32) return {0, true};
  return {1, false};
}

// Variant of the bitmask kernel, 0 = 6 CTAs per SM (40 registers) or 1 = 4 (64
// registers), for a filter read in one pass.  us for 2^26 probes, 0 / 1, in L2
// (8 MiB), at 64 and at 96 MiB, where more of the loads come from the far half
// of the L2 or from DRAM and more warps in flight hide them:
//   u64 w=8 s=8 k=8      342/382 383/454 506/595     u32 w=16 z=2   315/320 336/360 492/513
//   u32 w=16 s=8         336/344 372/395 500/527     u64 w=8 s=2    599/672 638/690 793/797
//   u64 w=8 z=2          338/333 366/379 495/514     u64 w=8 z=4    434/410 441/464 522/603
//   u64 w=8 s=4          469/459 480/503 539/625     u32 w=16 z=4   375/374 378/394 502/521
//   u32 w=16 s=1 k=4     444/442 450/432 489/498     u64 w=4 s=4    364/357 385/379 480/520
//   u32 w=1 k=4          289/293 299/291 503/492     u64 w=16 k=16  717/611 723/659 784/761
// (at 112 MiB u64 w=4 s=4 580/588, u32 w=8 s=8 477/485 at 96 MiB but 563/542 at 108)
// (in one pass the 8-CTA, 32-register form was slower than 0 everywhere but for
// u64 w=8 s=2 beyond 64 MiB, 723 at 96, and z=4 and s=4 at 80 to 96).  Bloom
// layouts whose kernel 0 spills take kernel 1.
int bits_variant_for(const dtlg_filter* f) {
  if (f->ck) return cuckoo_form(f).variant;
  const uint64_t mib = f->d.m_actual >> 23;
  // classic Bloom, k = 4: 1 MiB 391 / 415, 64 MiB 427 / 485; k = 8 567 / 634,
  // 635 / 769; k = 2 340 / 332 at 8 MiB
  if (f->qk) return f->d.k >= 4 && mib >= 1 && mib <= 100 ? 0 : 1;
  if (!f->bk || f->d.k > 8) return 1;
  const uint32_t block = f->d.w * f->d.word_bytes, s = f->d.s, w = f->d.w;
  const bool zoned = f->d.kind == Kind::kZoned, u32 = f->d.word_bytes == 4;
  if (block == 32) return mib >= 68 && mib <= (u32 ? 98 : 114) ? 0 : 1;
  if (block != 64) return 1;
  if (zoned) return (u32 && f->d.z == 2) || mib >= 60 ? 0 : 1;
  if (s >= w) return 0;
  if (u32) return s * 2 == w || (mib >= 88 && mib <= 116) ? 0 : 1;
  if (s == 1) return mib >= 72 && mib <= 116 ? 0 : 1;
  return s == 2 ? (mib <= 88 ? 0 : 1) : (mib >= 60 ? 0 : 1);
}

// Register-budget variant of the bitmask / pair kernels for plan `mode`: the
// caller's, else as above for the bitmask plan in one pass, form 2 in the band
// above, 0 for the pair probe of Bloom filters, 1 for that of the others.  In
// the band (192 MiB, 2^27 probes, 8 / 6 / 4 CTAs per SM, us): u64 w=8 s=2 1736
// / 1844 / 2014, zoned u32 w=16 z=2 1237 / 1447 / 1636, u32 w=16 s=1 1225 / 1222
// / 1407.
// Pair probe (2^27 probes, 512 MiB, 8 / 6 / 4 CTAs per SM, us): u64 w=8 s=8 k=8
// 1195 / 1243 / 1294; the form of 8 keeps its lead where it spills (7 layouts,
// all k >= 12: u64 w=8 s=8 k=16 at 512 MiB 83.0 against 79.7 Gkeys/s).
// The caller's 0 is form 2 where the bitmask plan takes several passes, so that
// the tuner reaches what the planner takes in the band.
int probe_variant(const dtlg_filter* f, int mode) {
  if (f->bits_variant >= 0 && f->bits_variant < kBitsVariants)
    return mode == 2 && f->bits_variant == 0 && probe_passes(f) > 1 ? 2 : f->bits_variant;
  if (mode == 3) return (f->d.kind == Kind::kBloom || f->d.kind == Kind::kZoned) ? 0 : 1;
  int v = bitmask_band(f) ? 2 : bits_variant_for(f);
  if (v != 1 && f->bk) {
    const occ_fn spill = f->pk->bits_local_bytes[v];
    if (spill && spill() != 0) v = 1;
  }
  return v;
}

// Ranges of the partitioned probe and build: 2^L blocks each, about 8 MiB of
// filter and at most kMaxRanges of them.  A range shares L2 with the pair
// stream and the match mask's atomics; smaller ranges are re-read less (B200,
// u64 w=8 s=8 k=8, 2^28 probes, 32 / 16 / 8 MiB ranges: 512 MiB filter 85.8 /
// 87.2 / 89.9 Gkeys/s, 256 MiB 94.8 / 97.0 / 96.2; 512 MiB build from 2^28
// keys 19.9 / 19.0 / 18.5 ms).
void partition_ranges(const dtlg_filter* f, uint32_t* range_log2, uint32_t* n_ranges) {
  const uint64_t block_bytes = static_cast<uint64_t>(f->d.w) * f->d.word_bytes;
  const uint64_t nb = f->d.addr.block_cnt;
  uint32_t L = 0;
  while ((1ull << L) * block_bytes < (8ull << 20) && (1ull << L) < nb) L++;
  while (((nb + (1ull << L) - 1) >> L) > static_cast<uint64_t>(kMaxRanges)) L++;
  *range_log2 = L;
  *n_ranges = static_cast<uint32_t>((nb + (1ull << L) - 1) >> L);
}

// Groups keys_al[pre, n_phys) by filter range: (key, logical position) pairs
// in one segment per range, in the workspace's pair area (partitioned probe
// and build).  The partition header must be zeroed before (it is, with the
// match mask, by one memset).  One kernel, grids of resident CTAs only: the
// tiles are strided over the grid, so a second, partial wave would finish its
// share late.  spill: optional exact list of the pairs that did not fit.
cudaError_t launch_partition(const dtlg_filter* f, const uint32_t* keys_al, uint64_t n_phys, uint32_t pre,
                             char* wsb, const WsLayout& lay, int sms, cudaStream_t stream, PartArgs* out,
                             uint2* spill = nullptr) {
  PartArgs pa{};
  pa.keys_al = keys_al;
  pa.n_phys = n_phys;
  pa.pre = pre;
  pa.addr = f->d.addr;
  pa.block_mul = mul_const(f->xk ? 1 : 0);
  partition_ranges(f, &pa.range_log2, &pa.n_ranges);
  pa.range_shift = 32 - clog2(f->d.addr.block_cnt) + pa.range_log2;  // POW2 only
  pa.n_tiles = part_tiles(n_phys);
  part_segments(n_phys - pre, f->d.addr.block_cnt, pa.range_log2, pa.n_ranges, &pa.seg_cap, &pa.last_cap);
  pa.hdr = reinterpret_cast<PartHeader*>(wsb + lay.part_off);
  pa.tile_overflow = reinterpret_cast<unsigned long long*>(wsb + lay.tflags_off);
  pa.pairs = reinterpret_cast<uint2*>(wsb + lay.pairs_off);
  pa.spill = spill;
  auto occupancy = [](void (*k)(PartArgs)) {
    int o = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k, kPartThreads, 0) == cudaSuccess ? std::max(1, o) : 1;
  };
  static const int occ_pow2 = occupancy(part_scatter_kernel<false>);
  static const int occ_magic = occupancy(part_scatter_kernel<true>);
  const bool magic = pa.addr.magic_mode != 0;
  const int sgrid = static_cast<int>(
      std::min<uint64_t>(pa.n_tiles, static_cast<uint64_t>(sms) * (magic ? occ_magic : occ_pow2)));
  if (magic) {
    part_scatter_kernel<true><<<sgrid, kPartThreads, 0, stream>>>(pa);
  } else {
    part_scatter_kernel<false><<<sgrid, kPartThreads, 0, stream>>>(pa);
  }
  *out = pa;
  return cudaGetLastError();
}

constexpr size_t kSlotBytes = sizeof(WsHeader) + static_cast<size_t>(kFusedSumTiles) * 8;

// Blocking probes that run on a result slot: the fused plan's one-round shapes.
bool on_slot(const dtlg_filter* f, const uint32_t* keys, uint32_t n) {
  if (n == 0 || probe_plan(f, n) != 1) return false;
  return fused_shape(static_cast<uint64_t>(n) + ((reinterpret_cast<uintptr_t>(keys) & 15u) >> 2)).rounds == 1;
}

// Waits for the outcome of the slot's current call: polls its word for a while
// (the kernel's write arrives microseconds before a stream synchronization
// returns; the match list is complete by then), then synchronizes, which also
// reports errors.  1024 keys: 32.4 us per blocking call with a workspace
// allocated, zeroed, copied back and freed, 18.7 us on a slot (and 15.8 with
// the binding's raw stream handle).
cudaError_t wait_for_slot(const ResultSlot& s, cudaStream_t stream, unsigned long long* word) {
  const volatile unsigned long long* w = s.host;
  const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(200);
  for (uint32_t i = 0; (*w >> 32) != s.ticket; i++) {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
    if ((i & 63u) == 63u && std::chrono::steady_clock::now() > until) {
      const cudaError_t e = cudaStreamSynchronize(stream);
      if (e != cudaSuccess) return e;
      if ((*w >> 32) != s.ticket) return cudaErrorUnknown;
    }
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  *word = *w;
  return cudaSuccess;
}

// Payload columns copied along with the match positions (probe -> gather).
struct GatherSpec {
  uint32_t n_cols;
  uint32_t col_bytes[kMaxGatherCols];
  const void* cols[kMaxGatherCols];
  void* out_cols[kMaxGatherCols];
};

// Enqueues the probe of `keys[0..n)`; the count goes to count_dev.  With
// `gather`, the compaction also copies the matching rows of the payload
// columns (the fused single-kernel plan has no compaction pass of its own,
// so gathers always take the bitmask plan).
dtlg_status launch_probe(const dtlg_filter* f, const uint64_t* words, const uint32_t* keys, uint32_t n,
                         uint32_t* out, uint32_t offset, unsigned long long* count_dev, void* ws,
                         size_t ws_bytes, cudaStream_t stream, const GatherSpec* gather = nullptr,
                         const ResultSlot* slot = nullptr) {
  DeviceState* ds = nullptr;
  dtlg_status st = device_state(&ds);
  if (st) return st;
  if (n == 0) {
    DTLG_CUDA(cudaMemsetAsync(count_dev, 0, sizeof(unsigned long long), stream));
    return DTLG_OK;
  }
  const uint32_t pre = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(keys) & 15u) >> 2);
  const uint64_t n_phys = static_cast<uint64_t>(n) + pre;
  int mode = probe_plan(f, n);
  if (gather && mode == 1) mode = 2;
  const FusedShape shape = fused_shape(n_phys);
  const uint32_t tiles = mode == 1 ? shape.n_tiles : compact_tiles(n_phys);
  const WsLayout lay = ws_layout(n_phys);
  if (ws_bytes < (slot ? kSlotBytes : mode == 3 ? lay.total : lay.total_small)) return DTLG_ERR_WORKSPACE;
  // a batch of one fused tile takes no ticket and waits for nobody, and the
  // kernel clears the error word itself
  const bool one_tile = mode == 1 && tiles == 1;
  if (!one_tile && !slot) DTLG_CUDA(cudaMemsetAsync(ws, 0, sizeof(WsHeader) + static_cast<size_t>(tiles) * 8, stream));
  char* wsb = static_cast<char*>(ws);
  WsHeader* h = static_cast<WsHeader*>(ws);
  ProbeArgs a{};
  a.filter = words;
  a.keys_al = keys - pre;
  a.n_phys = n_phys;
  a.pre = pre;
  a.match_offset = offset;
  a.out = out;
  a.count_out = count_dev;
  a.status = reinterpret_cast<unsigned long long*>(h + 1);
  a.tile_ctr = &h->tile_ctr;
  a.err = &h->err;
  a.n_tiles = tiles;
  set_filter_args(f->d, &a);
  // blocks of >= 32 bytes are read with 256-bit loads when the words are
  // 32-byte aligned (every plan; the fused plan read them as two 128-bit
  // loads before, which doubled its L1 wavefronts)
  a.vec32 = (reinterpret_cast<uintptr_t>(words) & 31u) == 0 ? 1u : 0u;
  if (mode == 1) {
    // the fused plan reads Bloom filters that cannot live in L1 without
    // allocating there, as the bitmask plan does (below)
    a.l1na = (f->bk != nullptr && (f->d.m_actual / 8) > kL1NoAllocBytes) ? 1u : 0u;
    if (slot) {
      a.done = &h->done;
      a.result = slot->host_dev;
      a.ticket = slot->ticket;
    }
    DTLG_CUDA(f->pk->probe(a, shape, ds->sms, stream));
    return DTLG_OK;
  }
  uint32_t* bits = reinterpret_cast<uint32_t*>(wsb + lay.bits_off);
  const int v = probe_variant(f, mode);
  if (mode == 4) {
    // the whole filter in every CTA's shared memory
    const uint32_t words32 = static_cast<uint32_t>((f->d.m_actual + 31) / 32);
    DTLG_CUDA(f->pk->probe_smem(a, bits, words32, (n_phys + 127) / 128, ds->sms, stream));
  } else if (mode == 2) {
    // Random blocks of a Bloom filter that cannot live in L1 are read without
    // allocating in L1 (B200, u64 w=8 s=8 k=8, 2^28 probes: 8 MiB filter
    // 118.5 -> 127.1 Gkeys/s; a 64 KiB L1-resident filter falls from 150.8 to
    // 71.1 without L1 allocation, and the partitioned plan's pair probe from
    // 76.0 to 72.9, so both keep allocating).  Not for the other kinds:
    // cuckoo buckets 75.6 -> 47.9, blocked cuckoo (128 MiB) 102.1 -> 98.9,
    // classic Bloom unchanged.
    a.l1na = (f->bk != nullptr && (f->d.m_actual / 8) > kL1NoAllocBytes) ? 1u : 0u;
    a.together = f->ck != nullptr && cuckoo_form(f).together ? 1u : 0u;
    // match bitmask, in block-range passes over large filters (each pass
    // probes only the keys whose block lies in its range, so the concurrently
    // touched part of the filter stays within the GPU's address-translation reach)
    const probe_bits_fn bfn = f->pk->probe_bits[v];
    const occ_fn bocc = f->pk->bits_blocks_per_sm[v];
    const uint64_t chunks = (n_phys + 127) / 128;  // one warp-chunk = 128 keys
    const uint64_t max_grid = static_cast<uint64_t>(ds->sms) * std::max(1, bocc());
    const int bgrid = static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>((chunks + 7) / 8, max_grid)));
    const uint32_t passes = probe_passes(f);
    const uint32_t nb = f->d.addr.block_cnt;
    for (uint32_t r = 0; r < passes; r++) {
      a.range_on = passes > 1 ? 1u : 0u;
      a.blk_lo = static_cast<uint32_t>(static_cast<uint64_t>(nb) * r / passes);
      a.blk_hi = r + 1 == passes ? 0xFFFFFFFFu : static_cast<uint32_t>(static_cast<uint64_t>(nb) * (r + 1) / passes);
      DTLG_CUDA(bfn(a, bits, r > 0 ? 1 : 0, bgrid, stream));
    }
  } else {
    // partitioned probe: keys grouped by filter range, probed range by range;
    // one memset zeroes the match mask and the partition header after it
    PartArgs pa{};
    DTLG_CUDA(cudaMemsetAsync(bits, 0, lay.part_off - lay.bits_off + kPartHeaderBytes, stream));
    DTLG_CUDA(launch_partition(f, a.keys_al, n_phys, pre, wsb, lay, ds->sms, stream, &pa));
    PairsArgs pr{};
    pr.probe = a;
    pr.part = pa;
    pr.bits = bits;
    pr.pre = pre;
    const int qgrid = static_cast<int>(static_cast<uint64_t>(ds->sms) * std::max(1, f->pk->pairs_blocks_per_sm[v]()));
    DTLG_CUDA(f->pk->probe_pairs[v](pr, qgrid, stream));
  }
  // ordered compaction of the bitmask
  CompactArgs c{};
  c.bits = bits;
  c.n_words = bits_words(n_phys);
  c.pre = pre;
  c.match_offset = offset;
  c.out = out;
  c.count_out = count_dev;
  c.status = a.status;
  c.tile_ctr = a.tile_ctr;
  c.err = a.err;
  c.n_tiles = tiles;
  if (gather) {
    c.n_cols = gather->n_cols;
    for (uint32_t i = 0; i < gather->n_cols; i++) {
      c.col_bytes[i] = gather->col_bytes[i];
      c.cols[i] = gather->cols[i];
      c.out_cols[i] = gather->out_cols[i];
    }
  }
  const int cgrid = static_cast<int>(std::min<uint64_t>(tiles, static_cast<uint64_t>(ds->sms) * compact_occupancy()));
  switch (compact_rows(c.n_words)) {
    case 2: compact_kernel<2><<<cgrid, kCompactThreads, 0, stream>>>(c); break;
    case 4: compact_kernel<4><<<cgrid, kCompactThreads, 0, stream>>>(c); break;
    default: compact_kernel<8><<<cgrid, kCompactThreads, 0, stream>>>(c);
  }
  DTLG_CUDA(cudaGetLastError());
  return DTLG_OK;
}

// Build plan of a blocked Bloom or blocked cuckoo filter (one block per key)
// for n keys that are not built range by range (range_build): 1 = one kernel of
// global atomics, 2 = keys grouped by L2-sized block range first (the probe's
// partition).  Automatic: the partitioned build for Bloom filters beyond 80 MiB
// and batches of >= 2^20 keys (u64 w=8
// s=8 k=8, plan 1 -> plan 2: 512 MiB from 2^28 keys 10.55 -> 4.07 ms; 256 MiB
// 4.23 -> 2.07 ms; 96 MiB (12 bits/key, MAGIC) 1.22 -> 1.09 ms; 64 MiB stays
// with plan 1, 0.51 against 0.60 ms).  A blocked cuckoo key takes one or two
// compare-and-swaps, too few to repay the partition (256 MiB, 2^26 keys:
// 2.60 -> 2.70 ms), so its plan 2 is only taken on request.
int block_build_plan(const dtlg_filter* f, uint64_t n) {
  if (f->build_mode == 1 || f->build_mode == 2) return f->build_mode;
  const uint64_t bytes = (f->d.m_actual + 7) / 8;
  return (f->bk != nullptr && n >= kTwoPassMinKeys && bytes > (80ull << 20)) ? 2 : 1;
}

// The range-by-range build (build_ranges.cuh) of a blocked Bloom filter from
// n_phys keys: fills in its ranges and bucket capacity, false where another
// plan is taken.  It updates every word once and handles 80 to 250 Gkeys/s
// whatever the filter's size, where the one-kernel build does 75 to 180 in L2,
// by the sectors and words a key touches, and the coarse partition 65 to 90
// beyond.  Per-build us, other plan -> range by range:
//   beyond 80 MiB, one key per 40 bytes or more: u64 w=8 s=8 k=8 2^26 keys /
//   128 MiB 1002 -> 508, 2^22 / 181 MiB 130 -> 107; u32 w=1 k=4 610 -> 390, 121
//   -> 114 (at 64 bytes per key 142 -> 144, and u32 w=16 s=8 133 -> 151);
//   in L2, blocks of 64 bytes whose words all take bits (two sectors per key)
//   or are picked one by one, one key per 8 bytes or more: u64 w=8 s=8 2^22 /
//   8 MiB 58 -> 45, 2^24 / 64 MiB 229 -> 164 (2^22 / 64 MiB 58 -> 65); u32
//   w=16 z=2 2^23 / 16 MiB 86 -> 63; u64 w=8 s=2 2^22 / 8 MiB 81 -> 44;
//   other layouts in L2 only for very many keys: 2^26 / 64 MiB u32 w=1 390 ->
//   340, u64 w=4 s=4 634 -> 577, u64 w=8 z=4 633 -> 602, but 2^24 / 32 MiB 93
//   -> 105, 150 -> 168, 150 -> 175.
// A range is one CTA, so a filter of few ranges would leave most SMs idle: 64 of
// them at least (u64 w=8 s=8, one-kernel build -> range by range: 256 KiB, 32
// ranges, 2^22 keys 65 -> 89, 2^26 967 -> 1237; 512 KiB, 64 ranges, 68 -> 68,
// 925 -> 731), 256 for the other layouts (2^26 keys: u64 w=4 s=4 256 KiB 772 ->
// 1920, 1 MiB 569 -> 644, 2 MiB 569 -> 560).
// Repeated keys: 2^24 copies of D keys, u64 w=8 s=8, us per build, 8 MiB and 128
// MiB: D = 1 17245 -> 281, 85268 -> 289; 1000 336 -> 230, 689 -> 259; 10 000 240
// -> 224, 358 -> 265; 10^6 239 -> 141, 292 -> 184.  It loses where few copies of
// few keys meet small batches: 2^22 copies of 10 000 keys 68 -> 79, 113 -> 124.
bool range_build(const dtlg_filter* f, uint64_t n_phys, RangeArgs* a, uint32_t* range_bytes) {
  if (!f->bk || f->build_mode != 0 || n_phys < (1ull << 22) || n_phys > 0x70000000ull) return false;
  const uint64_t bytes = (f->d.m_actual + 7) / 8;
  const uint64_t block_bytes = static_cast<uint64_t>(f->d.w) * f->d.word_bytes;
  const bool wide = block_bytes >= 64 && (f->d.kind == Kind::kBloom || f->d.word_bytes == 4);
  if (bytes > (80ull << 20) ? bytes > 40 * n_phys : !(wide ? bytes <= 8 * n_phys : n_phys >= (48ull << 20)))
    return false;
  // the largest ranges that still make 512 of them (a few per SM): longer runs
  // for the scatter (2^27 keys over 2048 / 4096 ranges: 496 / 668 us)
  uint32_t rb = kBuildRangeBytes;
  while (rb > (8u << 10) && bytes / rb < 512) rb /= 2;
  a->range_log2 = 0;
  while ((block_bytes << a->range_log2) < rb) a->range_log2++;
  const uint64_t ranges = (f->d.addr.block_cnt + (1ull << a->range_log2) - 1) >> a->range_log2;
  if (ranges < (wide ? 64u : 256u) || ranges > kBuildMaxRanges) return false;
  a->n_ranges = static_cast<uint32_t>(ranges);
  a->range_shift = 32 - clog2(f->d.addr.block_cnt) + a->range_log2;  // POW2 only
  const uint64_t share = (n_phys << a->range_log2) / f->d.addr.block_cnt + 1;
  // More than its share, for where keys repeat the ranges' shares differ: a
  // quarter (10 000 keys 2^22 times in 8 MiB: 79 us, with an eighth 88), a
  // sixteenth for large batches, whose scatter slows down as the buckets spread
  // (2^27 keys over 2048 ranges: 515 us, with a quarter 526).
  a->cap = static_cast<uint32_t>((share + share / (n_phys < (1ull << 25) ? 4 : 16) + 512 + 3) & ~3ull);
  *range_bytes = rb;
  return true;
}

// Enqueues the range-by-range build; cudaErrorMemoryAllocation when there is
// no room for the buckets (4.3 to 5 bytes per key), with nothing enqueued.
cudaError_t launch_range_build(const dtlg_filter* f, uint64_t* words, const uint32_t* keys_al, uint64_t n_phys,
                               uint32_t pre, RangeArgs ra, uint32_t range_bytes, const DeviceState& ds,
                               cudaStream_t stream) {
  const size_t bucket_bytes = round256(static_cast<uint64_t>(ra.n_ranges) * ra.cap * 4);
  char* ws = nullptr;
  if (cudaMallocFromPoolAsync(reinterpret_cast<void**>(&ws), bucket_bytes + (ra.n_ranges + 1) * 4, ds.pool, stream) !=
      cudaSuccess) {
    cudaGetLastError();
    return cudaErrorMemoryAllocation;
  }
  ra.keys_al = keys_al;
  ra.n_phys = n_phys;
  ra.pre = pre;
  ra.addr = f->d.addr;
  ra.buckets = reinterpret_cast<uint32_t*>(ws);
  ra.fill = reinterpret_cast<unsigned int*>(ws + bucket_bytes);
  ra.filter = words;
  // a range of the largest size has an SM to itself: while it is built, the
  // one that the SM takes next comes into L2 (2^24 keys / 256 MiB 214 -> 206
  // us, zoned u32 198 -> 188; full ranges gain nothing, 2^27 keys 1017 / 1014,
  // u32 w=1 743 / 773; smaller ranges share the SM and take no hint)
  ra.prefetch = range_bytes == kBuildRangeBytes ? static_cast<uint32_t>(ds.sms) : 0u;
  set_range_layout(f->d.word_bytes, f->d.w,
                   make_schedule(f->d.word_bytes * 8, f->d.w, f->d.s, f->d.z, f->d.k, true), &ra);
  ra.n_tiles = static_cast<uint32_t>((n_phys + kScatterTile - 1) / kScatterTile);
  const auto scatter = ra.addr.magic_mode ? key_scatter_kernel<true> : key_scatter_kernel<false>;
  const size_t smem = kScatterTile * 4 + ra.n_ranges * 8;
  int occ = 0;
  cudaError_t e = cudaMemsetAsync(ra.fill, 0, (ra.n_ranges + 1) * 4, stream);
  if (e == cudaSuccess) e = allow_dynamic_smem(scatter, kScatterTile * 4 + kBuildMaxRanges * 8);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, scatter, kScatterThreads, smem);
  if (e == cudaSuccess) {
    const uint32_t grid = std::min<uint32_t>(ra.n_tiles, static_cast<uint32_t>(ds.sms) * std::max(1, occ));
    scatter<<<grid, kScatterThreads, smem, stream>>>(ra);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = f->bk->build_ranges(ra, range_bytes, stream);
  cudaFreeAsync(ws, stream);
  return e;
}

int grid_for(uint64_t items, int sms) {
  return static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>((items + 255) / 256, static_cast<uint64_t>(sms) * 8)));
}

dtlg_status cuckoo_insert(const dtlg_filter* f, uint64_t* words, const uint32_t* keys, uint32_t n,
                          uint64_t* failed_out, cudaStream_t stream) {
  DeviceState* ds = nullptr;
  dtlg_status st = device_state(&ds);
  if (st) return st;
  if (failed_out) *failed_out = 0;
  if (n == 0) return DTLG_OK;
  const FilterDesc& d = f->d;
  const bool packed = f->ck->word_bucket;
  const uint64_t slots_n = packed ? 0 : (static_cast<uint64_t>(d.addr.block_cnt) + 1) * d.b;
  uint32_t* slots = nullptr;
  unsigned long long* failed = nullptr;
  const uint64_t slot_bytes = (slots_n * 4 + 255) & ~255ull;
  DTLG_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&slots), slot_bytes + 256, ds->pool, stream));
  failed = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(slots) + slot_bytes);
  DTLG_CUDA(cudaMemsetAsync(failed, 0, 8, stream));
  uint32_t* table = reinterpret_cast<uint32_t*>(words);
  if (!packed) {
    DTLG_CUDA(cudaMemsetAsync(slots + static_cast<uint64_t>(d.addr.block_cnt) * d.b, 0, d.b * 4, stream));
    f->ck->unpack(table, slots, d.addr.block_cnt, grid_for(slots_n, ds->sms), stream);
  }
  const uint32_t pre = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(keys) & 15u) >> 2);
  CuckooBuildArgs a{};
  a.table = table;
  a.slots = slots;
  a.keys_al = keys - pre;
  a.n_phys = static_cast<uint64_t>(n) + pre;
  a.pre = pre;
  a.table_words = d.word_cnt;
  a.victim_word = d.victim_word;
  a.addr = d.addr;
  a.failed = failed;
  static std::atomic<uint64_t> seed_ctr{0x243F6A8885A308D3ull};
  a.seed = seed_ctr.fetch_add(0x9E3779B97F4A7C15ull);
  // one key per thread and no more: a thread held up by a long chain of kicks
  // keeps no other keys waiting
  f->ck->insert(a, static_cast<int>(std::min<uint64_t>((a.n_phys + 255) / 256, 1u << 22)), stream);
  if (!packed) f->ck->pack(table, slots, d.addr.block_cnt, d.word_cnt, grid_for(d.word_cnt, ds->sms), stream);
  unsigned long long lost = 0;
  ResultSlot* slot = ds->slots.acquire(kSlotBytes);
  unsigned long long* to = slot ? slot->host + 2 : &lost;
  cudaError_t e = cudaMemcpyAsync(to, failed, 8, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaFreeAsync(slots, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (slot && e != cudaSuccess) {
    ds->slots.drop(slot);
  } else if (slot) {
    lost = *to;
    ds->slots.release(slot);
  }
  DTLG_CUDA(e);
  DTLG_CUDA(cudaGetLastError());
  if (failed_out) *failed_out = lost;
  return lost ? DTLG_ERR_CUCKOO_FULL : DTLG_OK;
}

}  // namespace

dtlg_status cuda_error_status(cudaError_t e) { return cuda_fail(e); }
}  // namespace dtlg

// =============================================================================
extern "C" {

const char* dtlg_version(void) { return "dtlg 0.1 (sm_100a)"; }

const char* dtlg_last_cuda_error(void) { return dtlg::g_last_cuda_error.c_str(); }

const char* dtlg_status_string(dtlg_status s) {
  switch (s) {
    case DTLG_OK: return "ok";
    case DTLG_ERR_INVALID_CONFIG: return "invalid configuration";
    case DTLG_ERR_SIZE: return "filter size out of range (block count must not exceed 2^31)";
    case DTLG_ERR_NULL: return "null pointer";
    case DTLG_ERR_ALIGNMENT: return "filter words must be 16-byte aligned";
    case DTLG_ERR_CUDA: return "CUDA error";
    case DTLG_ERR_ALLOC: return "allocation failed";
    case DTLG_ERR_CUCKOO_FULL: return "cuckoo filter full: some keys could not be inserted";
    case DTLG_ERR_TIMEOUT: return "a bounded device wait timed out";
    case DTLG_ERR_WORKSPACE: return "workspace too small";
    case DTLG_ERR_UNSUPPORTED: return "unsupported operation";
  }
  return "unknown status";
}

dtlg_status dtlg_bloom_create(const dtlg_bloom_config* cfg, uint64_t m, dtlg_filter** out) {
  if (!cfg || !out) return DTLG_ERR_NULL;
  *out = nullptr;
  dtlg_filter* f = new dtlg_filter();
  const int rc = describe_bloom(cfg->word_size, cfg->word_cnt_per_block, cfg->sector_cnt, cfg->zone_cnt,
                                cfg->k, m, &f->d);
  if (rc) {
    delete f;
    return rc == 1 ? DTLG_ERR_INVALID_CONFIG : DTLG_ERR_SIZE;
  }
  f->bk = find_bloom(f->d.word_bytes, f->d.w, f->d.s, f->d.z, f->d.k);
  if (!f->bk) {
    delete f;
    return DTLG_ERR_INVALID_CONFIG;
  }
  f->pk = &f->bk->pk;
  *out = f;
  return DTLG_OK;
}

dtlg_status dtlg_cuckoo_create(const dtlg_cuckoo_config* cfg, uint64_t m, dtlg_filter** out) {
  if (!cfg || !out) return DTLG_ERR_NULL;
  *out = nullptr;
  dtlg_filter* f = new dtlg_filter();
  const int rc = describe_cuckoo(cfg->bits_per_tag, cfg->tags_per_bucket, m, &f->d);
  if (rc) {
    delete f;
    return rc == 1 ? DTLG_ERR_INVALID_CONFIG : DTLG_ERR_SIZE;
  }
  f->ck = find_cuckoo(f->d.t, f->d.b);
  if (!f->ck) {
    delete f;
    return DTLG_ERR_INVALID_CONFIG;
  }
  f->pk = &f->ck->pk;
  *out = f;
  return DTLG_OK;
}

dtlg_status dtlg_classic_bloom_create(const dtlg_classic_bloom_config* cfg, uint64_t m, dtlg_filter** out) {
  if (!cfg || !out) return DTLG_ERR_NULL;
  *out = nullptr;
  if (cfg->addr_mode > 1) return DTLG_ERR_INVALID_CONFIG;
  dtlg_filter* f = new dtlg_filter();
  const int rc = describe_classic(cfg->k, m, cfg->addr_mode == 1, &f->d);
  if (rc) {
    delete f;
    return rc == 1 ? DTLG_ERR_INVALID_CONFIG : DTLG_ERR_SIZE;
  }
  f->qk = find_classic();
  if (!f->qk) {
    delete f;
    return DTLG_ERR_INVALID_CONFIG;
  }
  f->pk = &f->qk->pk;
  *out = f;
  return DTLG_OK;
}

dtlg_status dtlg_blocked_cuckoo_create(const dtlg_blocked_cuckoo_config* cfg, uint64_t m, dtlg_filter** out) {
  if (!cfg || !out) return DTLG_ERR_NULL;
  *out = nullptr;
  dtlg_filter* f = new dtlg_filter();
  const int rc = describe_bcf(cfg->block_size_bytes, cfg->tag_size_bits, cfg->associativity, m, &f->d);
  if (rc) {
    delete f;
    return rc == 1 ? DTLG_ERR_INVALID_CONFIG : DTLG_ERR_SIZE;
  }
  f->xk = find_bcf(f->d.t, f->d.b);
  if (!f->xk) {
    delete f;
    return DTLG_ERR_INVALID_CONFIG;
  }
  f->pk = &f->xk->pk;
  *out = f;
  return DTLG_OK;
}

void dtlg_destroy(dtlg_filter* f) { delete f; }

uint64_t dtlg_size_in_bytes(const dtlg_filter* f) { return f ? (f->d.m_actual + 7) / 8 : 0; }
uint64_t dtlg_size(const dtlg_filter* f) { return f ? f->d.size_u64 : 0; }
uint64_t dtlg_alloc_words_u64(const dtlg_filter* f) { return f ? f->d.alloc_u64 : 0; }
int dtlg_kind(const dtlg_filter* f) { return f ? static_cast<int>(f->d.kind) : -1; }
uint64_t dtlg_block_cnt(const dtlg_filter* f) { return f ? f->d.addr.block_cnt : 0; }
int dtlg_is_magic(const dtlg_filter* f) { return f ? static_cast<int>(f->d.addr.magic_mode) : 0; }

size_t dtlg_name(const dtlg_filter* f, char* buf, size_t cap) {
  if (!f) return 0;
  const std::string s = filter_name(f->d);
  if (buf && cap > s.size()) {
    std::memcpy(buf, s.c_str(), s.size() + 1);
  } else if (buf && cap) {
    buf[0] = 0;
  }
  return s.size();
}

dtlg_status dtlg_batch_insert(const dtlg_filter* f, uint64_t* words, const uint32_t* keys, uint32_t n,
                              uint64_t* failed_out, dtlg_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (!f) return DTLG_ERR_NULL;
  if (failed_out) *failed_out = 0;
  if (n && !keys) return DTLG_ERR_NULL;
  if (dtlg_status st = check_filter_ptr(words)) return st;
  if (f->ck) return cuckoo_insert(f, words, keys, n, failed_out, stream);
  if (n == 0) return DTLG_OK;
  DeviceState* ds = nullptr;
  if (dtlg_status st = device_state(&ds)) return st;
  const uint32_t pre = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(keys) & 15u) >> 2);
  if (f->qk) {
    ClassicBuildArgs c{};
    c.filter = reinterpret_cast<uint32_t*>(words);
    c.keys_al = keys - pre;
    c.n_phys = static_cast<uint64_t>(n) + pre;
    c.pre = pre;
    c.addr = f->d.addr;
    c.k = f->d.k;
    c.bit_shift = f->d.bit_shift;
    c.bit_mask = f->d.bit_mask;
    DTLG_CUDA(f->qk->build(c, grid_for(c.n_phys, ds->sms), stream));
    return DTLG_OK;
  }
  if (f->xk) {
    // blocked cuckoo: inserts never fail (bcf.cpp:36-40)
    BcfBuildArgs b{};
    b.filter = words;
    b.keys_al = keys - pre;
    b.n_phys = static_cast<uint64_t>(n) + pre;
    b.pre = pre;
    b.addr = f->d.addr;
    b.bucket_bits = f->d.bucket_bits;
    b.hash_shift = f->d.hash_shift;
    static std::atomic<uint64_t> seed_ctr{0x13198A2E03707344ull};
    b.seed = seed_ctr.fetch_add(0x9E3779B97F4A7C15ull);
    if (block_build_plan(f, n) == 2) {
      // keys grouped by L2-sized block range first, as for Bloom filters; the
      // pairs that overflow their segment go to an exact spill list after the
      // workspace (a blocked cuckoo key must be inserted exactly once)
      const WsLayout lay = ws_layout(b.n_phys);
      void* ws = nullptr;
      if (cudaMallocFromPoolAsync(&ws, lay.total + round256(b.n_phys * 8), ds->pool, stream) == cudaSuccess) {
        PartArgs pa{};
        char* wsb = static_cast<char*>(ws);
        cudaError_t e = cudaMemsetAsync(wsb + lay.part_off, 0, kPartHeaderBytes, stream);
        if (e == cudaSuccess)
          e = launch_partition(f, b.keys_al, b.n_phys, pre, wsb, lay, ds->sms, stream, &pa,
                               reinterpret_cast<uint2*>(wsb + lay.total));
        if (e == cudaSuccess) e = f->xk->insert_pairs(b, pa, grid_for(n, ds->sms), stream);
        cudaFreeAsync(ws, stream);
        DTLG_CUDA(e);
        return DTLG_OK;
      }
      cudaGetLastError();  // no room for the partition: the one-kernel build
    }
    DTLG_CUDA(f->xk->insert(b, grid_for(b.n_phys, ds->sms), stream));
    return DTLG_OK;
  }
  const uint64_t n_phys = static_cast<uint64_t>(n) + pre;
  RangeArgs ra{};
  uint32_t range_bytes = 0;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (range_build(f, n_phys, &ra, &range_bytes) &&
      cudaStreamIsCapturing(stream, &capturing) == cudaSuccess && capturing == cudaStreamCaptureStatusNone) {
    const cudaError_t e = launch_range_build(f, words, keys - pre, n_phys, pre, ra, range_bytes, *ds, stream);
    if (e != cudaErrorMemoryAllocation) {
      DTLG_CUDA(e);
      return DTLG_OK;
    }
  }
  if (block_build_plan(f, n) == 2) {
    // keys grouped by L2-sized block range first (the probe's partition), then
    // inserted range by range: the atomic ORs hit lines that sit in L2
    const WsLayout lay = ws_layout(n_phys);
    void* ws = nullptr;
    if (cudaMallocFromPoolAsync(&ws, lay.total, ds->pool, stream) == cudaSuccess) {
      PartArgs pa{};
      char* wsb = static_cast<char*>(ws);
      cudaError_t e = cudaMemsetAsync(wsb + lay.part_off, 0, kPartHeaderBytes, stream);
      if (e == cudaSuccess) e = launch_partition(f, keys - pre, n_phys, pre, wsb, lay, ds->sms, stream, &pa);
      if (e == cudaSuccess) {
        const uint64_t vec = (static_cast<uint64_t>(n) + 1) / 2;
        e = f->bk->build_pairs(pa, words, f->d.addr, grid_for(vec, ds->sms), stream);
      }
      cudaFreeAsync(ws, stream);
      DTLG_CUDA(e);
      return DTLG_OK;
    }
    // no room for the partition's 8 bytes per key: the one-kernel build
    // needs no workspace (same words)
    cudaGetLastError();
  }
  BuildArgs a{};
  a.filter = words;
  a.keys_al = keys - pre;
  a.n_phys = n_phys;
  a.pre = pre;
  a.addr = f->d.addr;
  DTLG_CUDA(f->bk->build(a, grid_for((a.n_phys + 3) / 4, ds->sms), stream));
  return DTLG_OK;
}

dtlg_status dtlg_set_build_options(dtlg_filter* f, int mode) {
  if (!f) return DTLG_ERR_NULL;
  if (mode < 0 || mode > 2) return DTLG_ERR_INVALID_CONFIG;
  f->build_mode = mode;
  return DTLG_OK;
}

int dtlg_build_plan(const dtlg_filter* f, uint32_t key_cnt) {
  if (!f || key_cnt == 0) return 0;
  RangeArgs ra{};
  uint32_t range_bytes = 0;
  if (range_build(f, key_cnt, &ra, &range_bytes)) return 3;
  return f->bk || f->xk ? block_build_plan(f, key_cnt) : 1;
}

size_t dtlg_probe_workspace_size(uint32_t key_cnt) { return workspace_bytes(static_cast<uint64_t>(key_cnt) + 3); }

dtlg_status dtlg_set_l2_fetch_granularity(int bytes, int* in_effect) {
  if (!(bytes == 0 || bytes == 32 || bytes == 64 || bytes == 128)) return DTLG_ERR_INVALID_CONFIG;
  DTLG_CUDA(cudaDeviceSetLimit(cudaLimitMaxL2FetchGranularity, static_cast<size_t>(bytes)));
  size_t v = 0;
  DTLG_CUDA(cudaDeviceGetLimit(&v, cudaLimitMaxL2FetchGranularity));
  if (in_effect) *in_effect = static_cast<int>(v);
  return DTLG_OK;
}

int dtlg_probe_kernel_count(const dtlg_filter* f, uint32_t key_cnt) {
  if (!f || key_cnt == 0) return 0;
  const int mode = probe_plan(f, key_cnt);
  // plan 3: partition scatter, pair probe, overflow keys, compaction
  return mode == 1 ? 1 : (mode == 2 ? static_cast<int>(probe_passes(f)) + 1 : (mode == 4 ? 2 : 4));
}

dtlg_status dtlg_set_probe_passes(dtlg_filter* f, int passes) {
  if (!f) return DTLG_ERR_NULL;
  if (passes < 0 || passes > 16) return DTLG_ERR_INVALID_CONFIG;
  f->probe_passes = passes;
  return DTLG_OK;
}

dtlg_status dtlg_set_probe_options(dtlg_filter* f, int mode, int variant) {
  if (!f) return DTLG_ERR_NULL;
  if (mode < 0 || mode > 4 || variant < -1 || variant >= kBitsVariants) return DTLG_ERR_INVALID_CONFIG;
  f->probe_mode = mode;
  f->bits_variant = variant;
  return DTLG_OK;
}

dtlg_status dtlg_batch_contains_ws(const dtlg_filter* f, const uint64_t* words, const uint32_t* keys,
                                   uint32_t n, uint32_t* out, uint32_t offset, uint64_t* count_dev,
                                   void* ws, size_t ws_bytes, dtlg_stream_t stream) {
  if (!f || !count_dev || (n && (!keys || !out)) || !ws) return DTLG_ERR_NULL;
  if (dtlg_status st = check_filter_ptr(words)) return st;
  return launch_probe(f, words, keys, n, out, offset, reinterpret_cast<unsigned long long*>(count_dev), ws,
                      ws_bytes, reinterpret_cast<cudaStream_t>(stream));
}

dtlg_status dtlg_batch_contains_gather(const dtlg_filter* f, const uint64_t* words, const uint32_t* keys,
                                       uint32_t n, uint32_t n_cols, const void* const* cols,
                                       const uint32_t* col_bytes, void* const* out_cols, uint32_t* match_positions,
                                       uint32_t offset, uint64_t* count_dev, void* ws, size_t ws_bytes,
                                       dtlg_stream_t stream) {
  if (!f || !count_dev || !ws || (n && !keys)) return DTLG_ERR_NULL;
  if (n_cols > kMaxGatherCols || (n_cols == 0 && !match_positions)) return DTLG_ERR_INVALID_CONFIG;
  if (n_cols && (!cols || !col_bytes || !out_cols)) return DTLG_ERR_NULL;
  GatherSpec g{};
  g.n_cols = n_cols;
  for (uint32_t i = 0; i < n_cols; i++) {
    if (col_bytes[i] != 4 && col_bytes[i] != 8) return DTLG_ERR_INVALID_CONFIG;
    if (n && (!cols[i] || !out_cols[i])) return DTLG_ERR_NULL;
    g.col_bytes[i] = col_bytes[i];
    g.cols[i] = cols[i];
    g.out_cols[i] = out_cols[i];
  }
  if (dtlg_status st = check_filter_ptr(words)) return st;
  return launch_probe(f, words, keys, n, match_positions, offset, reinterpret_cast<unsigned long long*>(count_dev),
                      ws, ws_bytes, reinterpret_cast<cudaStream_t>(stream), &g);
}

dtlg_status dtlg_batch_contains_async(const dtlg_filter* f, const uint64_t* words, const uint32_t* keys,
                                      uint32_t n, uint32_t* out, uint32_t offset, uint64_t* count_dev,
                                      dtlg_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (!f || !count_dev || (n && (!keys || !out))) return DTLG_ERR_NULL;
  if (dtlg_status st = check_filter_ptr(words)) return st;
  DeviceState* ds = nullptr;
  if (dtlg_status st = device_state(&ds)) return st;
  const size_t ws_bytes = dtlg_probe_workspace_size(n);
  void* ws = nullptr;
  DTLG_CUDA(cudaMallocFromPoolAsync(&ws, ws_bytes, ds->pool, stream));
  dtlg_status st = launch_probe(f, words, keys, n, out, offset, reinterpret_cast<unsigned long long*>(count_dev),
                                ws, ws_bytes, stream);
  cudaFreeAsync(ws, stream);
  return st;
}

dtlg_status dtlg_batch_contains(const dtlg_filter* f, const uint64_t* words, const uint32_t* keys, uint32_t n,
                                uint32_t* out, uint32_t offset, uint64_t* match_cnt, dtlg_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (!f || !match_cnt || (n && (!keys || !out))) return DTLG_ERR_NULL;
  if (dtlg_status st = check_filter_ptr(words)) return st;
  DeviceState* ds = nullptr;
  if (dtlg_status st = device_state(&ds)) return st;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  DTLG_CUDA(cudaStreamIsCapturing(stream, &capturing));
  ResultSlot* slot = capturing == cudaStreamCaptureStatusNone ? ds->slots.acquire(kSlotBytes) : nullptr;
  dtlg_status st = DTLG_OK;
  if (slot && on_slot(f, keys, n)) {
    WsHeader* h = static_cast<WsHeader*>(slot->dev);
    cudaError_t e = slot->fresh ? cudaMemsetAsync(slot->dev, 0, kSlotBytes, stream) : cudaSuccess;
    slot->fresh = false;
    if (++slot->ticket == 0) slot->ticket = 1;
    if (e == cudaSuccess)
      st = launch_probe(f, words, keys, n, out, offset, &h->count, slot->dev, kSlotBytes, stream, nullptr, slot);
    unsigned long long word = 0;
    if (e == cudaSuccess && st == DTLG_OK) e = wait_for_slot(*slot, stream, &word);
    if (e != cudaSuccess || st != DTLG_OK) {
      if (e != cudaSuccess) st = cuda_fail(e);
      ds->slots.drop(slot);
      return st;
    }
    ds->slots.release(slot);
    const bool err = (word & kResultErr) != 0;
    *match_cnt = err ? ~0ull : word & (kResultErr - 1u);
    return err ? DTLG_ERR_TIMEOUT : DTLG_OK;
  }
  // the other plans: a workspace of their own; its header (error word, count)
  // is copied to the slot's pinned words
  const size_t ws_bytes = dtlg_probe_workspace_size(n);
  void* ws = nullptr;
  cudaError_t e = cudaMallocFromPoolAsync(&ws, ws_bytes, ds->pool, stream);
  WsHeader host{};
  void* to = slot ? static_cast<void*>(slot->host + 2) : &host;
  if (e == cudaSuccess) {
    WsHeader* h = static_cast<WsHeader*>(ws);
    st = launch_probe(f, words, keys, n, out, offset, &h->count, ws, ws_bytes, stream);
    if (st == DTLG_OK) e = cudaMemcpyAsync(to, h, 16, cudaMemcpyDeviceToHost, stream);
    cudaFreeAsync(ws, stream);
    if (st == DTLG_OK && e == cudaSuccess) e = cudaStreamSynchronize(stream);
  }
  if (slot && (st != DTLG_OK || e != cudaSuccess)) {
    ds->slots.drop(slot);  // a copy into its words may still be on its way
  } else if (slot) {
    std::memcpy(&host, to, 16);
    ds->slots.release(slot);
  }
  if (st != DTLG_OK) return st;
  DTLG_CUDA(e);
  if (n == 0) host = WsHeader{};
  *match_cnt = host.count;
  return host.err ? DTLG_ERR_TIMEOUT : DTLG_OK;
}

dtlg_status dtlg_insert(const dtlg_filter* f, uint64_t* words, uint32_t key, dtlg_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  DeviceState* ds = nullptr;
  if (dtlg_status st = device_state(&ds)) return st;
  uint32_t* k = nullptr;
  DTLG_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&k), 16, ds->pool, stream));
  DTLG_CUDA(cudaMemcpyAsync(k, &key, 4, cudaMemcpyHostToDevice, stream));
  dtlg_status st = dtlg_batch_insert(f, words, k, 1, nullptr, stream_);
  cudaFreeAsync(k, stream);
  DTLG_CUDA(cudaStreamSynchronize(stream));
  return st;
}

dtlg_status dtlg_contains(const dtlg_filter* f, const uint64_t* words, uint32_t key, int* result,
                          dtlg_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (!result) return DTLG_ERR_NULL;
  DeviceState* ds = nullptr;
  if (dtlg_status st = device_state(&ds)) return st;
  uint32_t* k = nullptr;
  DTLG_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&k), 64, ds->pool, stream));
  DTLG_CUDA(cudaMemcpyAsync(k, &key, 4, cudaMemcpyHostToDevice, stream));
  uint64_t cnt = 0;
  dtlg_status st = dtlg_batch_contains(f, words, k, 1, k + 4, 0, &cnt, stream_);
  cudaFreeAsync(k, stream);
  DTLG_CUDA(cudaStreamSynchronize(stream));
  *result = cnt ? 1 : 0;
  return st;
}

dtlg_status dtlg_count_occupied_slots(const dtlg_filter* f, const uint64_t* words, uint64_t* count,
                                      dtlg_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (!f || !count) return DTLG_ERR_NULL;
  if (!f->ck) return DTLG_ERR_UNSUPPORTED;
  if (dtlg_status st = check_filter_ptr(words)) return st;
  DeviceState* ds = nullptr;
  if (dtlg_status st = device_state(&ds)) return st;
  unsigned long long* c = nullptr;
  DTLG_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&c), 8, ds->pool, stream));
  DTLG_CUDA(cudaMemsetAsync(c, 0, 8, stream));
  const uint64_t slots = static_cast<uint64_t>(f->d.addr.block_cnt) * f->d.b;
  f->ck->count(reinterpret_cast<const uint32_t*>(words), f->d.addr.block_cnt, f->d.victim_word, c,
               grid_for(slots, ds->sms), stream);
  unsigned long long h = 0;
  DTLG_CUDA(cudaMemcpyAsync(&h, c, 8, cudaMemcpyDeviceToHost, stream));
  cudaFreeAsync(c, stream);
  DTLG_CUDA(cudaStreamSynchronize(stream));
  *count = h;
  return DTLG_OK;
}

}  // extern "C"
