// Skew-aware minibatch localisation without a full sort.
//
// Produces exactly what the sort-based path (radix_sort.cu + localize.cu)
// produces -- the sorted unique key list, CSC segment offsets, the CSR column
// remap, the CSC row index, the head bitmap and the owner slice offsets -- but
// groups the nonzeros instead of sorting them. It replaces the reference's
// Localizer::CountUniqIndex + RemapIndex (util/localizer.h:97-221) and the
// thread merge sort under it (util/parallel_sort.h:14-41) on the hot path.
//
// Why: a click-log minibatch is dominated by a few very frequent keys (under a
// Zipf law the thousand most frequent ids carry half of the nonzeros) while most
// distinct keys occur once or twice. An LSD radix sort moves every nonzero once
// per digit; here a nonzero is moved once.
//
//   1. sample     a strided sample of the keys is counted in a small global hash
//                 table; keys that occur often in it become "hot" (at most 2048).
//   2. count      every CTA walks a contiguous slice of the input and counts, in
//                 shared memory, its nonzeros per hot key and, for all others
//                 ("cold"), per bucket (bucket = top bits of the key, so buckets
//                 are ordered by key). The bin of every nonzero and its place
//                 among the slice's nonzeros of that bin are kept in one word, so
//                 that no later step looks a key up or counts again.
//   3. scan/plan  prefix sums give every slice a private output place per bin (no
//                 look-back chain) and every bucket its output range.
//   4. scatter    a cold nonzero goes to its bucket as one 64-bit word (key | row),
//                 or as key and row.
//   5. bucket     one CTA per bucket: a shared-memory table de-duplicates the
//                 bucket's keys and counts them. The table is order preserving
//                 (home slot = leading bits of the key, linear probing without
//                 wrap-around), so the occupied slots read in address order are
//                 sorted up to a permutation inside each run of adjacent slots;
//                 a key's rank is a prefix count plus a look at its own run, and
//                 nothing is sorted. Hot keys that fall into the bucket are
//                 merged in, and every cold nonzero's row goes to its final CSC
//                 place. What depends on the buckets in front (a key's index in
//                 the list) stays relative to the bucket: its unique keys are
//                 left, in order, where its words were, and every cold nonzero
//                 gets its key's rank. So no bucket waits for another.
//   6. finish     every CTA adds up the buckets' numbers of keys for itself. The
//                 key lists close up, and the nonzeros are walked in input order
//                 once more: a cold one's column is its bucket's first index plus
//                 its rank, a hot one goes to its CSC place.
//
// Inside a key's CSC segment the nonzeros are in no particular order (the sort
// based path lists them by position).
//
// When the keys are not spread evenly over the key space (a bucket far above the
// average), or a bucket holds more distinct keys than its table can take, a
// device flag is raised, the remaining steps return at once, and the caller's
// gated sort-based path (psb_sort_pairs_gated + psb_localize2_gated) does the
// work instead. No step waits inside the kernel for another CTA.
#include "psb_common.cuh"
#include "psb_cuda.h"
#include <type_traits>

namespace psb {

static constexpr u32 kSampMin = 1u << 14;         // elements sampled: a quarter of them, between these two
static constexpr u32 kSampMax = 1u << 16;
static constexpr u32 kSampSlots = 2 * kSampMax;   // sample hash table (global memory), largest
// Hot-key lookup table: buckets of four 32-bit entries {20-bit tag, 11-bit hot index}, one 16-byte load each. A
// bucket overflows into the next one; with at most half a key per bucket on average a look-up needs more than one
// bucket for one key in 500, so the lanes of a warp hardly ever wait for one another's probe sequences. (13.1 M
// nonzeros: the step around it 955 us with 64-bit keys, linear probing and one element at a time, 916 us so.)
static constexpr u32 kHotBuckets = 4096;
static constexpr u32 kHotSlots = 4 * kHotBuckets;
static constexpr u32 kHotNone = 0xFFFFFFFFu;      // free entry (a tag never has its top bit set)
static constexpr u32 kHotMax = 2048;              // hot keys at most
static constexpr int kWalkThreads = 1024;         // count / scatter CTAs
static constexpr int kBucketThreads = 256;
static constexpr u32 kRunMax = 64;                // longest probe sequence / run of adjacent occupied slots
static constexpr u32 kMaxBuckets = 8192;
// The word that the count leaves per nonzero: its bin above its place among its slice's nonzeros of that bin.
static constexpr int kPlaceBits = 18;
static constexpr u32 kPlaceMask = (1u << kPlaceBits) - 1;
static_assert(kMaxBuckets + kHotMax <= 1u << (32 - kPlaceBits), "a bin fits above the place");
static constexpr u32 kWalkSplit = 2;              // scatter and finish: CTAs that share a slice
static constexpr int kHintShift = 5;              // one row hint per 32 positions
// Rows beyond this many positions get their hints from the whole grid: a warp takes 32 rows in turn. (13.1 M nonzeros in
// rows of 32,000: 498, 491 and 491 us with 2^15, 2^13 and 2^12; 0.39 M in rows of 6000: 79, 78 and 82.)
static constexpr u32 kLongRow = 1u << 13;
static constexpr u32 kLongHints = kLongRow >> kHintShift;
// A bucket's table comes in two sizes. 2^11 home slots serve minibatches in which keys repeat, the usual
// case; 2^12 those in which nearly every nonzero has its own key. Shared memory (and CTAs per SM) with compact keys of
// 32 bits: 28 KB (six; five with a payload, for its registers) and 54 KB (four); of 64 bits: 36 KB (five) and 71 KB
// (three). The sample decides (k_bl_plan), both kernels are launched and the one that was not chosen returns at once.
template <int kBits> struct BucketShape {
  static constexpr u32 kHs = 1u << kBits;                  // home slots
  static constexpr u32 kHsAll = kHs + 2 * kRunMax;         // plus the spill area behind the last home slot
  static constexpr u32 kHsWords = kHsAll / 32;             // occupancy bitmap words
  static constexpr u32 kDistinctMax = kHs / 2;             // distinct keys a bucket may hold
  static constexpr int kEntriesPerThread = kDistinctMax / kBucketThreads;
  static constexpr size_t smem_bytes(size_t key_bytes) {
    return kHsAll * (key_bytes + 4 + 2) + kDistinctMax * (4 + 2) + 2 * kHsWords * 4;
  }
};
static constexpr u32 kHotFlag = 1u << 31;         // segment starts on their way to the finish: a hot key's

// control words
enum { kCtlNumHot = 0, kCtlFallback = 1, kCtlSampleDistinct = 2, kCtlBigTables = 3, kCtlWords = 16 };

struct BLP {
  // input
  const void* in;
  int in_kind;            // 0 = uint64 keys, 1 = uint32 ids (hashed), 2 = uint64 ids (hashed)
  u64 seed;
  u32 n;
  int lo;                 // low key bits that are always zero (they carry the row when packed)
  int packed;
  int pay;                // words that travel beside a cold nonzero's key: row (not packed) and value, 0 to 2
  int nb_bits;            // log2(number of buckets)
  u32 NB, NBINS;          // buckets; NB + kHotMax
  u32 G, chunk;           // slices of the input and elements per slice
  u32 samp_m, samp_stride, samp_slots, hot_thresh, cold_limit;
  // rows
  const u32* row_ptr; u32 n_rows, fixed_z;
  const float* vals;
  // scratch
  u64* samp_key; u32* samp_cnt;
  u32* hot_tab; u64* hot_key;
  u32* ctl;
  u32* part;              // [G][NBINS]
  u32* bin_total;         // [NBINS]
  u32* cold_base;         // [NB + 1] where a bucket's cold words start: one place per cold nonzero and per hot key
  u32* pos_base;          // [NB + 1] where its CSC segments start
  u64* shot_key; u32* shot_h;       // hot keys sorted by key
  u32* bucket_hot_off;    // [NB + 1]
  u32* hot_seg;           // [kHotMax] where a hot key's segment starts
  u32* hot_loc;           // [kHotMax] its bucket (above 12 bits) and its rank there
  u32* bucket_d;          // [NB] unique keys per bucket
  u32* row_hint;          // [n / 32 + 2], with row_ptr only: the row of every 32nd position
  u64* cold_words;        // [n] cold keys by bucket; behind a bucket's CTA its unique keys in order
  u32* payload;           // [pay * n] beside them; then the unique keys' segment starts
  u32* place;             // [n] bin and place of every nonzero
  unsigned short* rank;   // [n] rank of every cold nonzero's key in its bucket, in the order of cold_words
  // outputs
  u64* ukeys; u32* seg_off; u32* csr_col; u32* csc_row; float* csc_val;
  u32* flagbits; u32* wordbase; u32* n_unique;
  const u64* bounds; int S; u32* own_off; u32* gate_out;
};

// The steps are launched with programmatic stream serialisation: a step's CTAs come in while the step before it drains, and
// wait here, before they read anything, until it has ended and its stores are visible (so all the steps before it
// have, too). The next step may come in from here on. Launched one by one, 64,000 nonzeros take 53 us instead of 70 and
// 3.9 M 202 instead of 216; replayed from a graph, 49 and 50, 197 and 194.
__device__ __forceinline__ void behind_the_step_before() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ u64 bl_key_of(const BLP& p, u32 i) {
  if (p.in_kind == 0) return ((const u64*)p.in)[i];
  u64 id = p.in_kind == 1 ? (u64)((const u32*)p.in)[i] : ((const u64*)p.in)[i];
  return hash_id_to_key(id, p.seed);
}
__device__ __forceinline__ u32 hot_hash(u64 key) {              // bucket: top 12 bits; tag: low 20 bits
  return ((u32)(key >> 32) ^ (u32)key) * 0x9E3779B1u;
}
// Largest r in [lo, hi) with row_ptr[r] <= pos; row_ptr[lo] <= pos.
__device__ __forceinline__ u32 row_search(const u32* __restrict__ row_ptr, u32 lo, u32 hi, u32 pos) {
  while (hi - lo > 1) {
    const u32 mid = (lo + hi) >> 1;
    if (row_ptr[mid] <= pos) lo = mid; else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ u32 row_of_pos(const BLP& p, u32 pos, u32 zinv) {
  if (p.row_ptr == nullptr) {
    u32 r = __umulhi(pos, zinv);
    while (pos - r * p.fixed_z >= p.fixed_z) ++r;              // the estimate is at most two short
    return r;
  }
  // Ragged rows: the hints of the position's block of 32 and of the next one bracket the row, so that the
  // search takes a step or two instead of log2(n_rows) dependent loads per nonzero (3.9 M nonzeros in 100,000
  // rows: localisation and margins 579 -> 466 us).
  const u32 b = pos >> kHintShift;
  // (clamped: row offsets that do not ascend from 0 to n leave hints unwritten)
  const u32 lo = min(p.row_hint[b], p.n_rows - 1), hi = min(p.row_hint[b + 1], p.n_rows - 1) + 1;
  return row_search(p.row_ptr, lo, max(lo + 1, hi), pos);
}

// Positions [b, e) of row r, within the input whatever the offsets are.
__device__ __forceinline__ void row_range(const BLP& p, u32 r, u32& b, u32& e) {
  b = r == 0 ? 0u : p.row_ptr[r];
  e = r + 1 == p.n_rows ? p.n : min(p.n, p.row_ptr[r + 1]);
}

// ---------------------------------------------------------------- 0. clean scratch
// Everything that starts as zeros or ones, and the row hints, in one launch instead of one per region.
__global__ void __launch_bounds__(256) k_bl_clear(const BLP p, uint4* zero, u32 zero4, uint4* ones, u32 ones4, u32 flag_words) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const u32 gsize = gridDim.x * blockDim.x, gtid = blockIdx.x * blockDim.x + threadIdx.x;
  for (u32 i = gtid; i < zero4; i += gsize) zero[i] = make_uint4(0, 0, 0, 0);
  for (u32 i = gtid; i < ones4; i += gsize) ones[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
  for (u32 i = gtid; i < flag_words; i += gsize) p.flagbits[i] = 0;
  if (p.row_ptr != nullptr) {
    // Row hints for steps 4 and 6, up to the block behind the last position: every row writes those of the blocks that
    // start in it, with its whole warp where they are many. (3.9 M nonzeros in 100,000 rows: this kernel 3.2 us; 9.4 with a
    // search of log2(rows) dependent loads per hint.) A row beyond kLongRow writes those in front of its first multiple of
    // kLongRow and one at every multiple; k_bl_sample fills in the rest.
    const u32 lane = threadIdx.x & 31;
    for (u32 r0 = gtid - lane; r0 < p.n_rows; r0 += gsize) {
      const u32 r = r0 + lane;
      u32 b = 0, e = 0;
      if (r < p.n_rows) row_range(p, r, b, e);
      const u32 h0 = (b + 31) >> kHintShift, h1 = e > b ? (e + 31) >> kHintShift : h0;
      const bool longer = h1 > h0 + 16;
      if (!longer) for (u32 h = h0; h < h1; ++h) p.row_hint[h] = r;
      for (u32 m = __ballot_sync(0xffffffffu, longer); m; m &= m - 1) {
        const int first = __ffs(m) - 1;
        const u32 a0 = __shfl_sync(0xffffffffu, h0, first), a1 = __shfl_sync(0xffffffffu, h1, first);
        const bool very = __shfl_sync(0xffffffffu, e - b, first) > kLongRow;
        const u32 mark = (a0 + kLongHints - 1) & ~(kLongHints - 1), a2 = very ? min(a1, mark) : a1;
        for (u32 h = a0 + lane; h < a2; h += 32) p.row_hint[h] = r0 + first;
        if (very) for (u32 h = mark + kLongHints * lane; h < a1; h += 32 * kLongHints) p.row_hint[h] = r0 + first;
      }
    }
    if (gtid == 0) p.row_hint[((p.n - 1) >> kHintShift) + 1] = p.n_rows - 1;
  }
}

// ---------------------------------------------------------------- 1. sample
// (Counted in shared memory per CTA first, it takes as long: 65,536 elements 9 us like this, 10 that way; 16,384 5 and 6.)
__global__ void __launch_bounds__(256) k_bl_sample(const BLP p) {
  behind_the_step_before();
  const u32 j = blockIdx.x * blockDim.x + threadIdx.x;
  if (p.row_ptr != nullptr) {
    // Row hints of very long rows: a warp per stretch of kLongRow positions, from the hint at its start. (The localisation of
    // one row of 13.1 M nonzeros: 538 us with all of its hints written by one warp, 477 so; of 3.9 M 200 and 181.)
    const u32 lane = threadIdx.x & 31, stretches = (p.n + kLongRow - 1) / kLongRow;
    for (u32 m = j >> 5; m < stretches; m += gridDim.x * blockDim.x >> 5) {
      const u32 r = min(p.row_hint[m * kLongHints], p.n_rows - 1);
      u32 b, e;
      row_range(p, r, b, e);
      if (e <= b || e - b <= kLongRow) continue;
      const u32 h1 = (min(e, m * kLongRow + kLongRow) + 31) >> kHintShift;
      for (u32 h = m * kLongHints + 1 + lane; h < h1; h += 32) p.row_hint[h] = r;
    }
  }
  const bool valid = j < p.samp_m;
  const u64 key = valid ? bl_key_of(p, j * p.samp_stride) : kEmptyKey;
  // equal keys of a warp count once (the most frequent key would otherwise take thousands of
  // atomics on one address)
  const u32 m = __match_any_sync(0xffffffffu, key);
  if (!valid || (int)(threadIdx.x & 31) != __ffs(m) - 1) return;
  u32 slot = (u32)(fmix64(key) & (p.samp_slots - 1));
  for (u32 probe = 0; probe < p.samp_slots; ++probe) {
    u64 old = atomicCAS(&p.samp_key[slot], kEmptyKey, key);
    if (old == kEmptyKey || old == key) { atomicAdd(&p.samp_cnt[slot], (u32)__popc(m)); return; }
    slot = (slot + 1) & (p.samp_slots - 1);
  }
}

// Keys counted often enough become hot. One atomic per CTA on each of the two counters (131,072 places: 4.1 us; 7.1 with one
// per warp and per key, which queue up on the two addresses).
static constexpr int kHotThreads = 1024;
__global__ void __launch_bounds__(kHotThreads) k_bl_hot(const BLP p) {
  behind_the_step_before();
  __shared__ u32 s_n, s_base;
  const u32 s = blockIdx.x * kHotThreads + threadIdx.x;
  const u32 c = s < p.samp_slots ? p.samp_cnt[s] : 0u;
  if (threadIdx.x == 0) s_n = 0;
  // distinct keys of the sample (how much keys repeat decides the size of the buckets' tables)
  const u32 occ = (u32)__syncthreads_count(c > 0);
  const bool hot = c >= p.hot_thresh;
  const u32 mine = hot ? atomicAdd(&s_n, 1u) : 0u;
  __syncthreads();
  if (threadIdx.x == 0) {
    if (occ) atomicAdd(&p.ctl[kCtlSampleDistinct], occ);
    s_base = s_n ? atomicAdd(&p.ctl[kCtlNumHot], s_n) : 0u;
  }
  __syncthreads();
  if (!hot) return;
  const u64 key = p.samp_key[s];
  const u32 h = s_base + mine;
  if (h >= kHotMax) return;                                    // more candidates than places: the rest stay cold
  p.hot_key[h] = key;
  const u32 hash = hot_hash(key), entry = ((hash & 0xFFFFFu) << 11) | h;
  u32 slot = (hash >> 20) * 4;
  for (u32 probe = 0; probe < kHotSlots; ++probe) {
    if (atomicCAS(&p.hot_tab[slot], kHotNone, entry) == kHotNone) return;
    slot = (slot + 1) & (kHotSlots - 1);
  }
}

// Four consecutive elements of the input (from element i on; those at or behind `end` are zero), by 16-byte loads
// where the alignment allows it.
struct Four { u64 k[4]; };
__device__ __forceinline__ Four load_input(const BLP& p, u32 i, u32 end) {
  Four r;
  const bool wide = i + 3 < end && (((size_t)p.in) & 15) == 0;
  if (p.in_kind == 1) {
    u32 id[4] = {0, 0, 0, 0};
    if (wide) {
      const uint4 v = *reinterpret_cast<const uint4*>((const u32*)p.in + i);
      id[0] = v.x; id[1] = v.y; id[2] = v.z; id[3] = v.w;
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) if (i + q < end) id[q] = ((const u32*)p.in)[i + q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) r.k[q] = id[q];
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) r.k[q] = 0;
    if (wide) {
      const ulonglong2* v = reinterpret_cast<const ulonglong2*>((const u64*)p.in + i);
      const ulonglong2 a = v[0], c = v[1];
      r.k[0] = a.x; r.k[1] = a.y; r.k[2] = c.x; r.k[3] = c.y;
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) if (i + q < end) r.k[q] = ((const u64*)p.in)[i + q];
    }
  }
  return r;
}
__device__ __forceinline__ u64 to_key(const BLP& p, u64 in) { return p.in_kind == 0 ? in : hash_id_to_key(in, p.seed); }

// Rows of consecutive positions.
struct RowWalk {
  u32 row, left;                                   // left (fixed-length rows): positions up to the next row
  __device__ __forceinline__ RowWalk(const BLP& p, u32 pos, u32 zinv) {
    row = row_of_pos(p, pos, zinv);
    left = p.row_ptr == nullptr ? (row + 1) * p.fixed_z - pos : 0u;
  }
  // to position pos + 1, which has a row
  __device__ __forceinline__ void next(const BLP& p, u32 pos) {
    if (p.row_ptr == nullptr) {
      if (--left == 0) { ++row; left = p.fixed_z; }
    } else if (row + 1 < p.n_rows && p.row_ptr[row + 1] <= pos + 1) {
      ++row;
      // behind a run of empty rows: searched, since one thread would walk all of it (20,000 nonzeros with
      // 100,000 empty rows in their midst: 7.0 ms row by row, 0.09 ms like this, as without them)
      if (row + 1 < p.n_rows && p.row_ptr[row + 1] <= pos + 1) row = row_of_pos(p, pos + 1, 0);
    }
  }
};

// ---------------------------------------------------------------- 2. count
// Shared memory: hot table | hot keys | one counter per bin. Bound by instruction issue (hash, look-up) and the
// shared-memory accesses. Keeping each nonzero's bin and place (the counter's old value, which a reduction would not
// return) takes 14 us of 72 for 13.1 M nonzeros, and saves the scatter its look-ups and counters and the finish all of it.
__global__ void __launch_bounds__(kWalkThreads) k_bl_count(const BLP p) {
  behind_the_step_before();
  extern __shared__ __align__(16) unsigned char smem[];
  uint4* s_hot = reinterpret_cast<uint4*>(smem);
  u64* s_hkey = reinterpret_cast<u64*>(smem + kHotSlots * 4);
  u32* s_bin = reinterpret_cast<u32*>(smem + kHotSlots * 4 + kHotMax * 8);
  const u32 nh = min(p.ctl[kCtlNumHot], kHotMax);
  const int t = threadIdx.x;
  for (u32 i = t; i < kHotBuckets; i += kWalkThreads) s_hot[i] = reinterpret_cast<const uint4*>(p.hot_tab)[i];
  for (u32 i = t; i < nh; i += kWalkThreads) s_hkey[i] = p.hot_key[i];
  for (u32 i = t; i < p.NBINS; i += kWalkThreads) s_bin[i] = 0;
  __syncthreads();
  const u32 begin = blockIdx.x * p.chunk;
  const u32 end = min(p.n, begin + p.chunk);
  const int bshift = 64 - p.nb_bits;
  // The bin of a key: its place among the hot keys, else its bucket.
  auto bin_of = [&](u64 key) -> u32 {
    if (nh) {
      const u32 hash = hot_hash(key), tag = hash & 0xFFFFFu;
      u32 at = hash >> 20;
      for (u32 probe = 0; probe < kHotBuckets; ++probe) {
        const uint4 e = s_hot[at];
        u32 hit = kHotNone;                        // a tag that matches is almost always the key
        if ((e.x >> 11) == tag) hit = e.x;
        if ((e.y >> 11) == tag) hit = e.y;
        if ((e.z >> 11) == tag) hit = e.z;
        if ((e.w >> 11) == tag) hit = e.w;
        if (hit != kHotNone) {
          if (s_hkey[hit & 0x7FFu] == key) return p.NB + (hit & 0x7FFu);
          // another key with the tag: look at every entry of the bucket that has it
          const u32 es[4] = {e.x, e.y, e.z, e.w};
          for (int k = 0; k < 4; ++k)
            if ((es[k] >> 11) == tag && s_hkey[es[k] & 0x7FFu] == key) return p.NB + (es[k] & 0x7FFu);
        }
        if (e.w == kHotNone) break;                // entries fill a bucket from the front: nothing in the next one
        at = (at + 1) & (kHotBuckets - 1);
      }
    }
    return (u32)(key >> bshift);
  };
  // Four consecutive elements per thread and trip, the next trip's loads in flight while these are handled: all
  // look-ups, then all counts, then the store, so that no element waits for another's chain. Plain shared-memory
  // atomics, also for the hot keys: lanes that hit one address serialise inside the instruction, which costs far
  // less than finding the groups first.
  const u32 step = 4u * kWalkThreads;
  u32 i = begin + 4u * t;
  Four nxt = load_input(p, i, end);
  for (; i < end; i += step) {
    const Four cur = nxt;
    nxt = load_input(p, i + step < end ? i + step : end, end);
    const u32 nvalid = min(4u, end - i);
    u32 bin[4], at[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) bin[q] = (u32)q < nvalid ? bin_of(to_key(p, cur.k[q])) : 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) at[q] = (u32)q < nvalid ? atomicAdd(&s_bin[bin[q]], 1u) : 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) at[q] |= bin[q] << kPlaceBits;
    if (nvalid == 4) {
      *reinterpret_cast<uint4*>(p.place + i) = make_uint4(at[0], at[1], at[2], at[3]);
    } else {
#pragma unroll
      for (int q = 0; q < 3; ++q) if ((u32)q < nvalid) p.place[i + q] = at[q];
    }
  }
  __syncthreads();
  u32* my_part = p.part + (size_t)blockIdx.x * p.NBINS;
  for (u32 k = t; k < p.NBINS; k += kWalkThreads) my_part[k] = s_bin[k];
}

// What a CTA of the scatter or the finish has of the input: a share of one slice.
struct Share {
  u32 slice, begin, end;
  __device__ __forceinline__ Share(const BLP& p) {
    slice = blockIdx.x / kWalkSplit;
    const u32 part = (p.chunk / kWalkSplit + 3) & ~3u, b = slice * p.chunk, e = min(p.n, b + p.chunk);
    begin = min(e, b + (blockIdx.x % kWalkSplit) * part);
    end = blockIdx.x % kWalkSplit == kWalkSplit - 1 ? e : min(e, begin + part);
  }
};
__device__ __forceinline__ uint4 load_places(const BLP& p, u32 i, u32 end) {
  if (i + 3 < end) return __ldcs(reinterpret_cast<const uint4*>(p.place + i));
  uint4 v = make_uint4(0, 0, 0, 0);
  if (i < end) v.x = p.place[i];
  if (i + 1 < end) v.y = p.place[i + 1];
  if (i + 2 < end) v.z = p.place[i + 2];
  return v;
}

// ---------------------------------------------------------------- 4. scatter
// Cold nonzeros to their buckets. Bound by the stores, each a sector of its own (a slice has five words for a bucket):
// 13.1 M nonzeros, 6 M of them cold: 106 us, 56 us without the stores (149 us with the keys looked up and counted again).
__global__ void __launch_bounds__(kWalkThreads, 2) k_bl_scatter(const BLP p) {
  behind_the_step_before();
  extern __shared__ __align__(16) u32 s_base[];
  if (p.ctl[kCtlFallback]) return;
  const Share sh(p);
  const int t = threadIdx.x;
  const u32* part = p.part + (size_t)sh.slice * p.NBINS;
  for (u32 i = t; i < p.NB; i += kWalkThreads) s_base[i] = part[i] + p.cold_base[i];
  __syncthreads();
  const u32 zinv = p.fixed_z ? (u32)(0xffffffffu / p.fixed_z) : 0u;
  const u32 step = 4u * kWalkThreads;
  u32 i = sh.begin + 4u * t;
  Four nk = load_input(p, i, sh.end);
  uint4 np = load_places(p, i, sh.end);
  for (; i < sh.end; i += step) {
    const Four cur = nk;
    const u32 at[4] = {np.x, np.y, np.z, np.w};
    const u32 j = i + step < sh.end ? i + step : sh.end;
    nk = load_input(p, j, sh.end);
    np = load_places(p, j, sh.end);
    // the row of a position is found here, where neighbouring threads look at neighbouring rows, and travels with
    // the key: looked up where the nonzeros arrive in key order, it is three dependent random loads each
    RowWalk r(p, i, zinv);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (i + q >= sh.end) break;
      if (q > 0) r.next(p, i + q - 1);
      const u32 bin = at[q] >> kPlaceBits;
      if (bin >= p.NB) continue;
      const u32 dst = s_base[bin] + (at[q] & kPlaceMask);
      p.cold_words[dst] = to_key(p, cur.k[q]) | (p.packed ? (u64)r.row : 0ull);
      if (p.pay == 2) reinterpret_cast<uint2*>(p.payload)[dst] = make_uint2(r.row, __float_as_uint(p.vals[i + q]));
      else if (p.pay == 1) p.payload[dst] = p.packed ? __float_as_uint(p.vals[i + q]) : r.row;
    }
  }
}

// ---------------------------------------------------------------- 3. scan + plan
// Per bin: exclusive prefix over the slices (in place) and the bin's total. A CTA takes 32 bins, each of its warps
// an eighth of the slices, all of them fetched at once. (148 slices x 10,240 bins: 3.4 us; 7.7 us with one thread per
// bin, sixteen slices at a time.)
static constexpr int kScanWarps = 8, kScanKeep = 20;
__global__ void __launch_bounds__(32 * kScanWarps) k_bl_scan(const BLP p) {
  behind_the_step_before();
  __shared__ u32 s_sum[kScanWarps][32];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5, bin = blockIdx.x * 32 + lane;
  const u32 per = (p.G + kScanWarps - 1) / kScanWarps, c0 = min(p.G, w * per), c1 = min(p.G, c0 + per);
  const bool have = bin < p.NBINS;
  u32* col = p.part + bin;
  u32 v[kScanKeep], sum = 0;
  if (have) {
#pragma unroll
    for (u32 k = 0; k < kScanKeep; ++k) v[k] = c0 + k < c1 ? col[(size_t)(c0 + k) * p.NBINS] : 0u;
#pragma unroll
    for (u32 k = 0; k < kScanKeep; ++k) sum += v[k];
    for (u32 c = c0 + kScanKeep; c < c1; ++c) sum += col[(size_t)c * p.NBINS];
  }
  s_sum[w][lane] = sum;
  __syncthreads();
  if (!have) return;
  u32 run = 0, total = 0;
#pragma unroll
  for (u32 k = 0; k < kScanWarps; ++k) {
    const u32 x = s_sum[k][lane];
    if (k < w) run += x;
    total += x;
  }
#pragma unroll
  for (u32 k = 0; k < kScanKeep; ++k) {
    if (c0 + k < c1) col[(size_t)(c0 + k) * p.NBINS] = run;
    run += v[k];
  }
  for (u32 c = c0 + kScanKeep; c < c1; ++c) {
    const u32 x = col[(size_t)c * p.NBINS];
    col[(size_t)c * p.NBINS] = run;
    run += x;
  }
  if (w == 0) p.bin_total[bin] = total;
}

// One CTA: the hot keys grouped by bucket, and per bucket the offset of its cold words, the final output offset and
// its first hot key. Every thread owns adjacent buckets and two adjacent hot
// keys, kept in registers; the three prefix sums go through one block scan, and four buckets go out in one store:
// a lone SM is bound by the number of sectors it asks for. 8192 buckets: 9 us (18 us as four scans of arrays in
// shared memory, and as long with one scan and a store per bucket), all of it on the critical path.
static constexpr int kPlanPer = kMaxBuckets / 1024;               // buckets per thread at most
__device__ __forceinline__ u32 plan_pad(u32 i) { return i + (i >> 5); }   // adjacent entries of a thread: no bank conflicts
__global__ void __launch_bounds__(1024) k_bl_plan(const BLP p) {
  behind_the_step_before();
  extern __shared__ __align__(16) unsigned char smem[];
  u32* s_hn = reinterpret_cast<u32*>(smem);         // [NB, padded] hot nonzeros per bucket
  u32* s_hc = s_hn + plan_pad(p.NB);                // [NB, padded] hot keys per bucket, then the place of the next one
  __shared__ u32 s_tot[3][32];
  __shared__ u32 s_max;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const u32 nh = min(p.ctl[kCtlNumHot], kHotMax);
  const int bshift = 64 - p.nb_bits;
  const u32 per = (p.NB + 1023) / 1024, b0 = t * per;
  if (t == 0) s_max = 0;
  // all global loads first
  u64 hk[2];
  u32 ht[2];
  __align__(16) u32 cold[kPlanPer];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const u32 i = 2 * t + k;
    hk[k] = i < nh ? p.hot_key[i] : 0;
    ht[k] = i < nh ? p.bin_total[p.NB + i] : 0u;
  }
#pragma unroll
  for (int k = 0; k < kPlanPer; ++k) cold[k] = 0;
  if (per >= 4) {                                   // one SM moves a sector per request: four buckets to a request
#pragma unroll
    for (int k = 0; k < kPlanPer; k += 4)
      if ((u32)k < per) *reinterpret_cast<uint4*>(&cold[k]) = *reinterpret_cast<const uint4*>(p.bin_total + b0 + k);
  } else {
#pragma unroll
    for (int k = 0; k < 2; ++k) cold[k] = (u32)k < per && b0 + k < p.NB ? p.bin_total[b0 + k] : 0u;
  }
  for (u32 i = t; i < 2 * plan_pad(p.NB); i += 1024) s_hn[i] = 0;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (2 * t + k < nh) {
      const u32 b = plan_pad((u32)(hk[k] >> bshift));
      atomicAdd(&s_hn[b], ht[k]);
      atomicAdd(&s_hc[b], 1u);
    }
  __syncthreads();
  // {cold words, all nonzeros, hot keys} before this thread's buckets. A bucket has room among the cold words for its
  // hot keys too (every one of them stands for nonzeros that are not there): its unique keys go there in the end.
  u32 v[3] = {0, 0, 0}, mx = 0;
#pragma unroll
  for (int k = 0; k < kPlanPer; ++k)
    if ((u32)k < per && b0 + k < p.NB) {
      const u32 b = plan_pad(b0 + k);
      v[0] += cold[k] + s_hc[b]; v[1] += cold[k] + s_hn[b]; v[2] += s_hc[b];
      mx = max(mx, cold[k]);
    }
  atomicMax(&s_max, mx);
  u32 x[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    x[q] = v[q];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(0xffffffffu, x[q], o);
      if (lane >= o) x[q] += y;
    }
    if (lane == 31) s_tot[q][w] = x[q];
  }
  __syncthreads();
  if (w < 3) {                                      // warp q turns the 32 totals of value q into prefixes
    u32 y = s_tot[w][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 z = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += z;
    }
    s_tot[w][lane] = y;
  }
  __syncthreads();
  u32 run[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) run[q] = (w ? s_tot[q][w - 1] : 0u) + x[q] - v[q];
  __align__(16) u32 out[3][kPlanPer];
#pragma unroll
  for (int k = 0; k < kPlanPer; ++k)
    if ((u32)k < per && b0 + k < p.NB) {
      const u32 b = plan_pad(b0 + k), c = s_hc[b];
      out[0][k] = run[0]; out[1][k] = run[1]; out[2][k] = run[2];
      run[0] += cold[k] + c; run[1] += cold[k] + s_hn[b];
      s_hc[b] = run[2];
      run[2] += c;
    }
  u32* const dst[3] = {p.cold_base, p.pos_base, p.bucket_hot_off};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (per >= 4) {
#pragma unroll
      for (int k = 0; k < kPlanPer; k += 4)
        if ((u32)k < per) *reinterpret_cast<uint4*>(dst[q] + b0 + k) = *reinterpret_cast<const uint4*>(&out[q][k]);
    } else {
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if ((u32)k < per && b0 + k < p.NB) dst[q][b0 + k] = out[q][k];
    }
  }
  __syncthreads();
  // hot keys grouped by bucket (any order inside a bucket: the bucket kernel puts them into its table)
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (2 * t + k < nh) {
      const u32 at = atomicAdd(&s_hc[plan_pad((u32)(hk[k] >> bshift))], 1u);
      p.shot_key[at] = hk[k];
      p.shot_h[at] = 2 * t + k;
    }
  if (t == 0) {
    p.cold_base[p.NB] = s_tot[0][31]; p.pos_base[p.NB] = s_tot[1][31]; p.bucket_hot_off[p.NB] = s_tot[2][31];
    if (s_max > p.cold_limit) p.ctl[kCtlFallback] = 1;   // keys are not spread evenly: use the sort
    // more than three quarters of the sampled nonzeros have a key of their own: the big tables
    p.ctl[kCtlBigTables] = (4ull * p.ctl[kCtlSampleDistinct] > 3ull * p.samp_m) ? 1u : 0u;
  }
}
static_assert(kHotMax == 2 * 1024, "two hot keys per thread of k_bl_plan");

// ---------------------------------------------------------------- 5. per-bucket grouping
template <typename CK> struct CkT;
template <> struct CkT<u32> { static constexpr u32 kEmpty = 0xFFFFFFFFu; };
template <> struct CkT<u64> { static constexpr u64 kEmpty = 0xFFFFFFFFFFFFFFFFull; };

// Home slot of a compact key with `rem` significant bits: its leading kBits bits (order preserving).
template <typename CK, int kBits>
__device__ __forceinline__ u32 bucket_home(CK ck, int rem) {
  return rem >= kBits ? (u32)(ck >> (rem - kBits)) : (u32)(ck << (kBits - rem));
}

template <typename CK, int kBits>
__device__ __forceinline__ int bucket_find(const CK* s_key, CK ck, int rem) {
  u32 slot = bucket_home<CK, kBits>(ck, rem);
  for (u32 probe = 0; probe < kRunMax; ++probe, ++slot) {
    const CK k = s_key[slot];
    if (k == ck) return (int)slot;
    if (k == CkT<CK>::kEmpty) return -1;
  }
  return -1;
}

// Finds or inserts ck; returns the slot, or -1 when the probe sequence got longer than kRunMax
// (keys that are not spread evenly inside the bucket). A new key sets its bit in the occupancy bitmap.
template <typename CK, int kBits>
__device__ __forceinline__ int bucket_insert(CK* s_key, u32* s_bits, CK ck, int rem) {
  u32 slot = bucket_home<CK, kBits>(ck, rem);
  for (u32 probe = 0; probe < kRunMax; ++probe, ++slot) {
    CK k = s_key[slot];
    if (k == ck) return (int)slot;
    if (k == CkT<CK>::kEmpty) {
      k = atomicCAS(&s_key[slot], CkT<CK>::kEmpty, ck);
      if (k == CkT<CK>::kEmpty) { atomicOr(&s_bits[slot >> 5], 1u << (slot & 31)); return (int)slot; }
      if (k == ck) return (int)slot;
    }
  }
  return -1;
}

// Exclusive block scan of one value per thread (kBucketThreads threads); total to every thread.
__device__ __forceinline__ u32 bucket_block_scan(u32 v, u32* s_warp /* 9 words */, u32* total) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  u32 x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    u32 y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) s_warp[w] = x;
  __syncthreads();
  u32 pre = x - v, tot = 0;
#pragma unroll
  for (int i = 0; i < kBucketThreads / 32; ++i) { const u32 sw = s_warp[i]; if (i < w) pre += sw; tot += sw; }
  *total = tot;
  return pre;
}

// kPay: something travels beside the keys' words (BLP::pay is not 0). Bound by the latencies of its short phases, which
// the CTAs of an SM overlap. 13.1 M nonzeros, 8192 buckets: 117 us, and 222 us with the index of the bucket's first
// key fetched by a look-back over the buckets in front (42 us) and every nonzero's column stored where the nonzero came
// from (50 us).
template <typename CK, int kBits, bool kPay>
__global__ void __launch_bounds__(kBucketThreads) k_bl_bucket(const BLP p) {
  behind_the_step_before();
  typedef BucketShape<kBits> Sh;
  constexpr u32 kHsAll = Sh::kHsAll, kHsWords = Sh::kHsWords, kDistinctMax = Sh::kDistinctMax;
  constexpr int kEntriesPerThread = Sh::kEntriesPerThread;
  extern __shared__ __align__(16) unsigned char smem[];
  CK* s_key = reinterpret_cast<CK*>(smem);                                     // table: compact keys
  u32* s_cnt = reinterpret_cast<u32*>(s_key + kHsAll);                         // per slot: count, then cursor
  u32* s_start = s_cnt + kHsAll;                                               // per distinct key, slot order
  u32* s_bits = s_start + kDistinctMax;                                        // occupancy bitmap
  u32* s_hbits = s_bits + kHsWords;                                            // slots that hold a hot key
  unsigned short* s_rank = reinterpret_cast<unsigned short*>(s_hbits + kHsWords);  // per slot: hot index, then rank
  unsigned short* s_dense = s_rank + kHsAll;                                   // occupied slots in slot order
  __shared__ u32 s_ovf, s_stop, s_warp[kBucketThreads / 32 + 1];
  const int t = threadIdx.x;
  if ((p.ctl[kCtlBigTables] != 0) != (kBits == 12)) return;
  const int sh_l = p.nb_bits, sh_r = p.nb_bits + p.lo;
  const int rem = 64 - sh_r;                    // significant bits of a compact key
  const u64 rowmask = p.packed ? ((1ull << p.lo) - 1) : 0ull;
  const bool row_beside = kPay && !p.packed, val_beside = kPay && p.vals != nullptr;
  for (u32 b = blockIdx.x; b < p.NB; b += gridDim.x) {
  const u32 cb = p.cold_base[b], ce = p.cold_base[b + 1], pb = p.pos_base[b];
  const u32 h0 = p.bucket_hot_off[b], h1 = p.bucket_hot_off[b + 1];
  // one thread reads the flag for the whole CTA: other CTAs may raise it at any moment
  if (t == 0) { s_stop = ld_relaxed_gpu(&p.ctl[kCtlFallback]); s_ovf = 0; }
  {
    // keys = all ones, counts = 0, bitmaps = 0, with 16-byte stores (while the loads are on their way)
    uint4* k4 = reinterpret_cast<uint4*>(s_key);
    const u32 nk4 = kHsAll * sizeof(CK) / 16;
    for (u32 i = t; i < nk4; i += kBucketThreads) k4[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    uint4* c4 = reinterpret_cast<uint4*>(s_cnt);
    for (u32 i = t; i < kHsAll / 4; i += kBucketThreads) c4[i] = make_uint4(0, 0, 0, 0);
    for (u32 i = t; i < 2 * kHsWords; i += kBucketThreads) s_bits[i] = 0;
  }
  const u32 nb = ce - cb - (h1 - h0);
  // The first four nonzeros of every thread stay in registers for both passes over the bucket
  // (a bucket of average size has no more), the rest is read again in pass 2.
  u64 w0[4];
  uint2 p0[4];                                     // row and value, as far as they travel beside the key
  auto beside = [&](u32 j) -> uint2 {
    if (!kPay) return make_uint2(0u, 0u);
    if (p.pay == 2) return reinterpret_cast<const uint2*>(p.payload)[cb + j];
    const u32 x = p.payload[cb + j];
    return make_uint2(x, x);
  };
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const u32 j = t + q * kBucketThreads;
    w0[q] = j < nb ? p.cold_words[cb + j] : 0;
    p0[q] = j < nb ? beside(j) : make_uint2(0u, 0u);
  }
  __syncthreads();
  if (s_stop) return;
  // hot keys of this bucket enter the table with their total count
  for (u32 i = h0 + t; i < h1; i += kBucketThreads) {
    const u32 h = p.shot_h[i];
    const CK ck = (CK)((p.shot_key[i] << sh_l) >> sh_r);
    const int slot = bucket_insert<CK, kBits>(s_key, s_bits, ck, rem);
    if (slot < 0) { s_ovf = 1; continue; }
    s_cnt[slot] = p.bin_total[p.NB + h];
    s_rank[slot] = (unsigned short)h;
    atomicOr(&s_hbits[slot >> 5], 1u << (slot & 31));
  }
  // pass 1 over the bucket's nonzeros: distinct keys and their counts
  for (u32 j0 = t; j0 < nb; j0 += 4 * kBucketThreads) {
    u64 wd[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 j = j0 + q * kBucketThreads;
      wd[q] = j0 == (u32)t ? w0[q] : (j < nb ? p.cold_words[cb + j] : 0);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 j = j0 + q * kBucketThreads;
      if (j >= nb) break;
      const CK ck = (CK)((wd[q] << sh_l) >> sh_r);
      const int slot = bucket_insert<CK, kBits>(s_key, s_bits, ck, rem);
      if (slot < 0) { s_ovf = 1; continue; }
      atomicAdd(&s_cnt[slot], 1u);
    }
  }
  __syncthreads();
  // occupied slots in slot order: prefix over the bitmap words, then one thread per word lists its slots
  u32 d = 0;
  const u32 myw = t < (int)kHsWords ? s_bits[t] : 0u;
  const u32 wpre = bucket_block_scan((u32)__popc(myw), s_warp, &d);
  if (d > kDistinctMax && t == 0) s_ovf = 1;
  __syncthreads();
  if (s_ovf) {
    // keys bunched inside the bucket (or too many of them): hand the whole minibatch to the sort-based path
    if (t == 0) st_relaxed_gpu(&p.ctl[kCtlFallback], 1u);
    return;
  }
  if (t == 0) p.bucket_d[b] = d;
  {
    u32 wbits = myw, k = wpre;
    while (wbits) {
      const int bit = __ffs(wbits) - 1;
      s_dense[k++] = (unsigned short)(32 * t + bit);
      wbits &= wbits - 1;
    }
  }
  __syncthreads();
  // nonzeros before every distinct key, in slot order (a thread takes adjacent entries)
  const u32 ipt = (d + kBucketThreads - 1) / kBucketThreads;
  const u32 i0 = min(d, (u32)t * ipt), i1 = min(d, i0 + ipt);
  u32 sum = 0;
  for (u32 i = i0; i < i1; ++i) sum += s_cnt[s_dense[i]];
  u32 dummy;
  u32 run = bucket_block_scan(sum, s_warp, &dummy);
  for (u32 i = i0; i < i1; ++i) { s_start[i] = run; run += s_cnt[s_dense[i]]; }
  __syncthreads();
  // Rank and segment start of every distinct key: the prefix at the first entry of its run of adjacent
  // occupied slots, plus the smaller keys of that run (a run is a permutation of its sorted order).
  u32 my_rank[kEntriesPerThread], my_start[kEntriesPerThread];
  bool bad = false;
#pragma unroll
  for (int k = 0; k < kEntriesPerThread; ++k) {
    const u32 i = t + k * kBucketThreads;
    my_rank[k] = 0xFFFFFFFFu; my_start[k] = 0;
    if (i >= d) continue;
    const u32 slot = s_dense[i];
    const CK key = s_key[slot];
    u32 j = i;                                      // first entry of the run
    while (j > 0 && (u32)s_dense[j - 1] + 1 == (u32)s_dense[j]) {
      --j;
      if (i - j > 2 * kRunMax) { bad = true; break; }
    }
    u32 r = j, st = s_start[j];
    for (u32 q = j; q < d; ++q) {
      if (q > j && (u32)s_dense[q - 1] + 1 != (u32)s_dense[q]) break;
      if (q - j > 4 * kRunMax) { bad = true; break; }
      const u32 sq = s_dense[q];
      if (s_key[sq] < key) { ++r; st += s_cnt[sq]; }
    }
    my_rank[k] = r; my_start[k] = st;
  }
  if (bad) s_ovf = 1;
  __syncthreads();
  if (s_ovf) {
    if (t == 0) st_relaxed_gpu(&p.ctl[kCtlFallback], 1u);
    return;
  }
#pragma unroll
  for (int k = 0; k < kEntriesPerThread; ++k) {
    if (my_rank[k] == 0xFFFFFFFFu) continue;
    const u32 i = t + k * kBucketThreads, slot = s_dense[i];
    const bool is_hot = (s_hbits[slot >> 5] >> (slot & 31)) & 1u;
    const u32 hh = is_hot ? s_rank[slot] : 0u;
    s_cnt[slot] = my_start[k];
    s_rank[slot] = (unsigned short)my_rank[k];
    s_start[i] = my_start[k] | (is_hot ? kHotFlag : 0u);
    if (is_hot) {                                  // for the finish, which places this key's nonzeros
      p.hot_seg[hh] = pb + my_start[k];
      p.hot_loc[hh] = (b << 12) | my_rank[k];
    }
  }
  __syncthreads();
  // pass 2: every nonzero's row to its place, and the rank of its key
  for (u32 j0 = t; j0 < nb; j0 += 4 * kBucketThreads) {
    u64 wd[4];
    uint2 ps[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 j = j0 + q * kBucketThreads;
      const bool first = j0 == (u32)t;
      wd[q] = first ? w0[q] : (j < nb ? p.cold_words[cb + j] : 0);
      ps[q] = first ? p0[q] : (j < nb ? beside(j) : make_uint2(0u, 0u));
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 j = j0 + q * kBucketThreads;
      if (j >= nb) break;
      const CK ck = (CK)((wd[q] << sh_l) >> sh_r);
      const int slot = bucket_find<CK, kBits>(s_key, ck, rem);
      if (slot < 0) continue;                     // cannot happen: the key was inserted in pass 1
      const u32 P = pb + atomicAdd(&s_cnt[slot], 1u);
      p.csc_row[P] = row_beside ? ps[q].x : (u32)(wd[q] & rowmask);
      if (val_beside) p.csc_val[P] = __uint_as_float(ps[q].y);
      p.rank[cb + j] = s_rank[slot];
    }
  }
  __syncthreads();
  // the unique keys and their segment starts, in order, over the words and what travelled beside them
  u32* seg = p.payload + (size_t)cb * max(1, p.pay);
  const u64 bucket_bits = (u64)b << (64 - p.nb_bits);
  for (u32 i = t; i < d; i += kBucketThreads) {
    const u32 slot = s_dense[i], r = s_rank[slot];
    p.cold_words[cb + r] = bucket_bits | ((u64)s_key[slot] << p.lo);
    seg[r] = s_start[i];
  }
  __syncthreads();       // the tables are rebuilt for the next bucket
  }
}

// ---------------------------------------------------------------- 6. finish
// Shared memory: per bucket the index of its first unique key and the place of this slice's first cold word; per hot
// key its index and the place of this slice's first nonzero. Bound by memory: a place read and a column written per
// nonzero, a 2-byte gather per cold and a 4-byte store of its own per hot one (13.1 M nonzeros: 110 us).
__global__ void __launch_bounds__(kWalkThreads, 2) k_bl_finish(const BLP p) {
  behind_the_step_before();
  extern __shared__ __align__(16) u32 s_first[];   // [NB + 4] [NB] [kHotMax] [kHotMax]
  __shared__ u32 s_tot[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const u32 skip = p.ctl[kCtlFallback];
  if (blockIdx.x == 0 && t == 0) *p.gate_out = skip;
  if (skip) return;
  u32* s_base = s_first + p.NB + 4;
  u32* s_hot_u = s_base + p.NB;
  u32* s_hot_at = s_hot_u + kHotMax;
  const Share sh(p);
  const u32* part = p.part + (size_t)sh.slice * p.NBINS;
  const u32 nh = min(p.ctl[kCtlNumHot], kHotMax);
  // a thread adds up adjacent buckets
  const u32 per = (p.NB + kWalkThreads - 1) / kWalkThreads, b0 = min(p.NB, t * per), b1 = min(p.NB, b0 + per);
  u32 cnt[kPlanPer], sum = 0;
#pragma unroll
  for (int k = 0; k < kPlanPer; ++k) {
    cnt[k] = b0 + k < b1 ? p.bucket_d[b0 + k] : 0u;
    sum += cnt[k];
  }
  for (u32 i = t; i < p.NB; i += kWalkThreads) s_base[i] = part[i] + p.cold_base[i];
  for (u32 h = t; h < nh; h += kWalkThreads) {
    s_hot_u[h] = p.hot_loc[h];
    s_hot_at[h] = p.hot_seg[h] + part[p.NB + h];
  }
  u32 x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_tot[w] = x;
  __syncthreads();
  u32 run = x - sum, total = 0;
#pragma unroll
  for (int k = 0; k < kWalkThreads / 32; ++k) {
    const u32 y = s_tot[k];
    if (k < w) run += y;
    total += y;
  }
#pragma unroll
  for (int k = 0; k < kPlanPer; ++k) {
    if (b0 + k < b1) s_first[b0 + k] = run;
    run += cnt[k];
  }
  if (t == 0) s_first[p.NB] = total;
  __syncthreads();
  for (u32 h = t; h < nh; h += kWalkThreads) {
    const u32 loc = s_hot_u[h];
    s_hot_u[h] = s_first[loc >> 12] + (loc & 0xFFFu);
  }
  __syncthreads();
  // (a) the unique keys close up: a warp per bucket
  const u32 pw = p.pay > 1 ? 2u : 1u;
  for (u32 b = blockIdx.x * (kWalkThreads / 32) + w; b < p.NB; b += gridDim.x * (kWalkThreads / 32)) {
    const u32 first = s_first[b], d = s_first[b + 1] - first;
    const u64* keys = p.cold_words + p.cold_base[b];
    const u32* seg = p.payload + (size_t)p.cold_base[b] * pw;
    const u32 pb = p.pos_base[b], pe = p.pos_base[b + 1];
    for (u32 r0 = lane; r0 < d; r0 += 128) {
      u64 key[4];
      u32 st[4], nx[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const u32 r = r0 + 32 * q;
        key[q] = r < d ? keys[r] : 0;
        st[q] = r < d ? seg[r] : 0u;
        nx[q] = r + 1 < d ? seg[r + 1] : 0u;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const u32 r = r0 + 32 * q;
        if (r >= d) break;
        const u32 u = first + r, P = pb + (st[q] & ~kHotFlag), e = r + 1 < d ? pb + (nx[q] & ~kHotFlag) : pe;
        p.ukeys[u] = key[q];
        p.seg_off[u] = P;
        atomicOr(&p.flagbits[P >> 5], 1u << (P & 31));
        // number of segment heads before every 32-aligned position inside the segment (a hot key's: below)
        if (!(st[q] & kHotFlag))
          for (u32 wd = (P + 31) >> 5; (wd << 5) < e; ++wd) p.wordbase[wd] = ((wd << 5) == P) ? u : u + 1;
      }
    }
  }
  // (b) the number of keys and the owners' shares of them
  if (blockIdx.x == 0) {
    for (u32 s = w; s < (u32)p.S; s += kWalkThreads / 32) {
      const u64 bound = p.bounds[s];
      const u32 b = (u32)(bound >> (64 - p.nb_bits));
      const u32 first = s_first[b], d = s_first[b + 1] - first;
      const u64* keys = p.cold_words + p.cold_base[b];
      u32 below = 0;
      if (bound << p.nb_bits)                      // (no key of a bucket lies below its first)
        for (u32 r = lane; r < d; r += 32) below += keys[r] < bound ? 1u : 0u;
      below = __reduce_add_sync(0xffffffffu, below);
      if (lane == 0) p.own_off[s] = first + below;
    }
    if (t == 0) {
      p.own_off[p.S] = total;
      p.seg_off[total] = p.n;
      *p.n_unique = total;
    }
  }
  // (c) the nonzeros in input order
  const u32 zinv = p.fixed_z ? (u32)(0xffffffffu / p.fixed_z) : 0u;
  const u32 step = 4u * kWalkThreads;
  u32 i = sh.begin + 4u * t;
  uint4 np = load_places(p, i, sh.end);
  for (; i < sh.end; i += step) {
    const u32 at[4] = {np.x, np.y, np.z, np.w};
    np = load_places(p, i + step < sh.end ? i + step : sh.end, sh.end);
    u32 u[4];
    bool any_hot = false;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 bin = at[q] >> kPlaceBits;
      u[q] = 0;
      if (i + q >= sh.end) continue;
      if (bin < p.NB) u[q] = p.rank[s_base[bin] + (at[q] & kPlaceMask)];
      else any_hot = true;
    }
    if (any_hot) {
      RowWalk r(p, i, zinv);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (i + q >= sh.end) break;
        if (q > 0) r.next(p, i + q - 1);
        const u32 bin = at[q] >> kPlaceBits;
        if (bin < p.NB) continue;
        const u32 h = bin - p.NB, P = s_hot_at[h] + (at[q] & kPlaceMask);
        u[q] = s_hot_u[h];
        p.csc_row[P] = r.row;
        if (p.csc_val) p.csc_val[P] = p.vals[i + q];
        if ((P & 31u) == 0) p.wordbase[P >> 5] = P == p.hot_seg[h] ? u[q] : u[q] + 1;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 bin = at[q] >> kPlaceBits;
      if (i + q < sh.end && bin < p.NB) u[q] += s_first[bin];
    }
    if (i + 3 < sh.end) {
      *reinterpret_cast<uint4*>(p.csr_col + i) = make_uint4(u[0], u[1], u[2], u[3]);
    } else {
#pragma unroll
      for (int q = 0; q < 3; ++q) if (i + q < sh.end) p.csr_col[i + q] = u[q];
    }
  }
}

template <typename... A>
static void launch_step(void (*fn)(A...), u32 grid, u32 block, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid); c.blockDim = dim3(block); c.dynamicSmemBytes = smem; c.stream = stream;
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &a; c.numAttrs = 1;
  cudaLaunchKernelEx(&c, fn, args...);
}

// scratch layout (bytes), shared by the size query and the launcher
struct BlLayout {
  size_t zero_begin, samp_cnt, ctl, zero_end;
  size_t ff_begin, samp_key, hot_tab, ff_end;
  size_t hot_key, part, bin_total, cold_base, pos_base, shot_key, shot_h, bucket_hot_off,
      hot_seg, hot_loc, bucket_d, row_hint, total;
};
static size_t al(size_t x) { return (x + 255) & ~(size_t)255; }
static BlLayout bl_layout(u32 NB, u32 G, u32 n, u32 samp_slots) {
  BlLayout L;
  size_t o = 0;
  const u32 NBINS = NB + kHotMax;
  L.zero_begin = o;
  L.samp_cnt = o; o = al(o + (size_t)samp_slots * 4);
  L.ctl = o; o = al(o + kCtlWords * 4);
  L.zero_end = o;
  L.ff_begin = o;
  L.samp_key = o; o = al(o + (size_t)samp_slots * 8);
  L.hot_tab = o; o = al(o + (size_t)kHotSlots * 4);
  L.ff_end = o;
  L.hot_key = o; o = al(o + kHotMax * 8);
  L.part = o; o = al(o + (size_t)G * NBINS * 4);
  L.bin_total = o; o = al(o + (size_t)NBINS * 4);
  L.cold_base = o; o = al(o + (size_t)(NB + 1) * 4);
  L.pos_base = o; o = al(o + (size_t)(NB + 1) * 4);
  L.shot_key = o; o = al(o + kHotMax * 8);
  L.shot_h = o; o = al(o + kHotMax * 4);
  L.bucket_hot_off = o; o = al(o + (size_t)(NB + 1) * 4);
  L.hot_seg = o; o = al(o + kHotMax * 4);
  L.hot_loc = o; o = al(o + kHotMax * 4);
  L.bucket_d = o; o = al(o + (size_t)NB * 4);
  L.row_hint = o; o = al(o + ((size_t)(n >> kHintShift) + 2) * 4);
  L.total = o;
  return L;
}

static u32 bl_num_buckets(u32 n) {
  // about 1600 nonzeros per bucket at most on average: even a minibatch without any repeated key
  // fills a bucket's table to 40 % only, so runs of adjacent occupied slots stay short
  u32 nb = 64;
  while (nb < kMaxBuckets && (size_t)nb * 1600 < n) nb <<= 1;
  // a small minibatch gets more and smaller buckets, so that its few CTAs' worth of work is spread over the
  // SMs (390,000 nonzeros in 256 buckets kept 256 CTAs busy for 49 us; with the smaller sample and walk grid the
  // training step on them went from 231 to 180 us)
  while (nb < 512 && (size_t)nb * 512 <= n) nb <<= 1;
  return nb;
}
// Slices of the input: one per SM, and as many as keep a nonzero's place in its bits.
static u32 bl_most_slices(u32 n) { return max((u32)max(1, psb_device_sm_count()), (u32)(((size_t)n + kPlaceMask) >> kPlaceBits)); }
// Resident CTAs of a bucket kernel.
static u32 bl_bucket_ctas(const void* fn, size_t smem) {
  int per = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, kBucketThreads, smem);
  return (u32)max(1, per) * (u32)max(1, psb_device_sm_count());
}

}  // namespace psb

using namespace psb;

extern "C" size_t psb_bucket_localize_scratch_bytes(uint32_t max_n) {
  // sized for the largest bucket count; the per-nonzero buffers are the caller's
  return bl_layout(kMaxBuckets, bl_most_slices(max_n), max_n, kSampSlots).total;
}

// Groups the n nonzeros of a minibatch by key. Inputs as for psb_sort_pairs (in, in_kind, seed);
// low_zero_bits = number of low key bits that are zero in every key (64 - significant bits of a
// narrow hashed key); when n_rows - 1 fits in them the row rides in the key word. Outputs as for psb_localize2; work buffers,
// alignment and what may be null: psb_cuda.h.
extern "C" int psb_bucket_localize(const void* in, int in_kind, psb_u64 seed, uint32_t n, int low_zero_bits,
                                   const uint32_t* row_ptr, uint32_t n_rows, uint32_t fixed_z,
                                   const float* vals, const psb_u64* bounds, int S,
                                   psb_u64* cold_words, uint32_t* beside, uint32_t* places,
                                   psb_u64* ukeys, uint32_t* seg_off, uint32_t* csr_col, uint32_t* csc_row,
                                   float* csc_val, uint32_t* flagbits, uint32_t* wordbase,
                                   uint32_t* n_unique, uint32_t* own_off, void* scratch, uint32_t* /*status: nothing waits*/,
                                   uint32_t* gate_out, cudaStream_t stream) {
  if (S < 1 || S > 64) return -(int)cudaErrorInvalidValue;
  if (row_ptr == nullptr && fixed_z == 0) return -(int)cudaErrorInvalidValue;
  if (low_zero_bits < 0 || low_zero_bits > 48 || in_kind < 0 || in_kind > 2) return -(int)cudaErrorInvalidValue;
  if (n == 0) {
    cudaMemsetAsync(n_unique, 0, sizeof(u32), stream);
    cudaMemsetAsync(own_off, 0, sizeof(u32) * (S + 1), stream);
    cudaMemsetAsync(seg_off, 0, sizeof(u32), stream);
    cudaMemsetAsync(gate_out, 0, sizeof(u32), stream);
    return -(int)cudaGetLastError();
  }
  if (vals == nullptr || csc_val == nullptr) vals = nullptr, csc_val = nullptr;   // values move only from one to the other
  BLP p{};
  p.in = in; p.in_kind = in_kind; p.seed = seed; p.n = n;
  p.lo = low_zero_bits;
  if (row_ptr == nullptr) n_rows = (n + fixed_z - 1) / fixed_z;
  else n_rows = max(n_rows, 1u);                    // nonzeros without a row are row 0's, as in the sort-based path
  p.packed = (low_zero_bits > 0 && n_rows > 0 && (low_zero_bits >= 32 || ((n_rows - 1) >> low_zero_bits) == 0)) ? 1 : 0;
  p.pay = (p.packed ? 0 : 1) + (vals != nullptr ? 1 : 0);
  if (cold_words == nullptr || beside == nullptr || places == nullptr ||
      ((((size_t)cold_words) | ((size_t)beside) | ((size_t)places) | ((size_t)csr_col)) & 15) != 0)
    return -(int)cudaErrorInvalidValue;
  p.NB = bl_num_buckets(n);
  p.nb_bits = 0;
  while ((1u << p.nb_bits) < p.NB) ++p.nb_bits;
  p.NBINS = p.NB + kHotMax;
  // no more slices than get a full trip of 4096 elements (every CTA fills its shared tables first)
  p.G = min(bl_most_slices(n), (n + 4 * kWalkThreads - 1) / (4 * kWalkThreads));
  p.chunk = ((n + p.G - 1) / p.G + 3) & ~3u;
  p.samp_m = min(n, max(kSampMin, min(kSampMax, n / 4)));
  p.samp_slots = 2;
  while (p.samp_slots < 2 * p.samp_m) p.samp_slots <<= 1;
  p.samp_stride = n / p.samp_m;
  // hot: about half an average bucket or more, judged from the sample
  p.hot_thresh = max(4u, p.samp_m / p.NB / 2);
  p.cold_limit = max(32768u, 16u * (n / p.NB));
  p.row_ptr = row_ptr; p.n_rows = n_rows; p.fixed_z = fixed_z; p.vals = vals;
  const BlLayout L = bl_layout(p.NB, p.G, n, p.samp_slots);
  unsigned char* sc = (unsigned char*)scratch;
  p.samp_key = (u64*)(sc + L.samp_key); p.samp_cnt = (u32*)(sc + L.samp_cnt);
  p.hot_tab = (u32*)(sc + L.hot_tab);
  p.hot_key = (u64*)(sc + L.hot_key);
  p.ctl = (u32*)(sc + L.ctl); p.part = (u32*)(sc + L.part); p.bin_total = (u32*)(sc + L.bin_total);
  p.cold_base = (u32*)(sc + L.cold_base); p.pos_base = (u32*)(sc + L.pos_base);
  p.shot_key = (u64*)(sc + L.shot_key); p.shot_h = (u32*)(sc + L.shot_h);
  p.bucket_hot_off = (u32*)(sc + L.bucket_hot_off); p.hot_seg = (u32*)(sc + L.hot_seg);
  p.hot_loc = (u32*)(sc + L.hot_loc); p.bucket_d = (u32*)(sc + L.bucket_d); p.row_hint = (u32*)(sc + L.row_hint);
  p.cold_words = (u64*)cold_words; p.payload = beside; p.place = places; p.rank = (unsigned short*)(places + n);
  p.ukeys = (u64*)ukeys; p.seg_off = seg_off; p.csr_col = csr_col; p.csc_row = csc_row; p.csc_val = csc_val;
  p.flagbits = flagbits; p.wordbase = wordbase; p.n_unique = n_unique;
  p.bounds = (const u64*)bounds; p.S = S; p.own_off = own_off; p.gate_out = gate_out;

  const u32 zero4 = (u32)((L.zero_end - L.zero_begin) / 16), ones4 = (u32)((L.ff_end - L.ff_begin) / 16);
  k_bl_clear<<<psb_device_sm_count() * 2, 256, 0, stream>>>(p, (uint4*)(sc + L.zero_begin), zero4, (uint4*)(sc + L.ff_begin),
                                                            ones4, (n + 31) / 32);
  launch_step(k_bl_sample, (p.samp_m + 255) / 256, 256, 0, stream, p);
  launch_step(k_bl_hot, (p.samp_slots + kHotThreads - 1) / kHotThreads, kHotThreads, 0, stream, p);
  const size_t count_smem = kHotSlots * 4 + kHotMax * 8 + (size_t)p.NBINS * 4;
  const size_t scatter_smem = (size_t)p.NB * 4, finish_smem = (size_t)(2 * p.NB + 4 + 2 * kHotMax) * 4;
  const int remaining = 64 - p.nb_bits - p.lo;      // key bits that distinguish keys inside a bucket
  const bool ck32 = remaining <= 31;
  const size_t plan_smem = (size_t)(p.NB + p.NB / 32) * 8;
  static const bool attr_set = [] {
    auto most = [](const void* fn, size_t bytes) { cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); };
    most((const void*)k_bl_count, kHotSlots * 4 + kHotMax * 8 + (size_t)(kMaxBuckets + kHotMax) * 4);
    most((const void*)k_bl_plan, (size_t)(kMaxBuckets + kMaxBuckets / 32) * 8);
    most((const void*)k_bl_scatter, (size_t)kMaxBuckets * 4);
    most((const void*)k_bl_finish, (size_t)(2 * kMaxBuckets + 4 + 2 * kHotMax) * 4);
    return true;
  }();
  (void)attr_set;
  launch_step(k_bl_count, p.G, kWalkThreads, count_smem, stream, p);
  launch_step(k_bl_scan, (p.NBINS + 31) / 32, 32 * kScanWarps, 0, stream, p);
  launch_step(k_bl_plan, 1, 1024, plan_smem, stream, p);
  launch_step(k_bl_scatter, p.G * kWalkSplit, kWalkThreads, scatter_smem, stream, p);
  auto bucket = [&](auto key, auto bits, auto pay) {
    typedef decltype(key) CK;
    constexpr int kBits = decltype(bits)::value;
    constexpr size_t smem = BucketShape<kBits>::smem_bytes(sizeof(CK));
    const auto fn = k_bl_bucket<CK, kBits, decltype(pay)::value>;
    static const u32 ctas = [fn] {
      cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      return bl_bucket_ctas((const void*)fn, smem);
    }();
    launch_step(fn, min(p.NB, ctas), kBucketThreads, smem, stream, p);
  };
  auto buckets = [&](auto key, auto pay) {
    bucket(key, std::integral_constant<int, 11>(), pay);
    bucket(key, std::integral_constant<int, 12>(), pay);
  };
  if (p.pay) {
    if (ck32) buckets(u32(), std::true_type()); else buckets(u64(), std::true_type());
  } else {
    if (ck32) buckets(u32(), std::false_type()); else buckets(u64(), std::false_type());
  }
  launch_step(k_bl_finish, p.G * kWalkSplit, kWalkThreads, finish_smem, stream, p);
  return -(int)cudaGetLastError();
}
