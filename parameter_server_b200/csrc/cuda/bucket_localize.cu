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
//                 are ordered by key).
//   3. scan/plan  prefix sums give every CTA a private output cursor per bin (no
//                 look-back chain), every bucket its output range, every hot key
//                 its place in the hot stream.
//   4. scatter    the same walk again: a cold nonzero goes to its bucket as one
//                 64-bit word (key | position), a hot nonzero's position goes to
//                 its key's list.
//   5. bucket     one CTA per bucket: a shared-memory table de-duplicates the
//                 bucket's keys and counts them. The table is order preserving
//                 (home slot = leading bits of the key, linear probing without
//                 wrap-around), so the occupied slots read in address order are
//                 sorted up to a permutation inside each run of adjacent slots;
//                 a key's rank is a prefix count plus a look at its own run, and
//                 nothing is sorted. Hot keys that fall into the bucket are
//                 merged in, a chained scan over the buckets (decoupled
//                 look-back, in ticket order) gives the global index of the
//                 bucket's first unique key, and every nonzero is written to its
//                 final CSC position.
//   6. hot emit   the hot keys' position lists are written to the CSC ranges
//                 that step 5 reserved for them.
//
// Inside a key's CSC segment the nonzeros are in no particular order (the sort
// based path lists them by position).
//
// When the keys are not spread evenly over the key space (a bucket far above the
// average), or a bucket holds more distinct keys than its table can take, a
// device flag is raised, the remaining steps return at once, and the caller's
// gated sort-based path (psb_sort_pairs_gated + psb_localize2_gated) does the
// work instead. Every spin is bounded and reports through the status word.
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
static constexpr int kHintShift = 5;              // one row hint per 32 positions
// A bucket's table comes in two sizes. 2^11 home slots (35 KB of shared memory, six CTAs per SM) serve
// minibatches in which keys repeat, the usual case; 2^12 (55 KB, four per SM) those in which nearly
// every nonzero has its own key. The sample decides (k_bl_plan), both kernels are launched and the
// one that was not chosen returns at once.
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
static constexpr u32 kFlagAgg = 1u << 30;
static constexpr u32 kFlagIncl = 2u << 30;
static constexpr u32 kValMask = (1u << 30) - 1;

// control words
enum { kCtlNumHot = 0, kCtlTicket = 1, kCtlFallback = 2, kCtlHotElems = 3, kCtlSampleDistinct = 4, kCtlBigTables = 5,
       kCtlWords = 16 };

struct BLP {
  // input
  const void* in;
  int in_kind;            // 0 = uint64 keys, 1 = uint32 ids (hashed), 2 = uint64 ids (hashed)
  u64 seed;
  u32 n;
  int lo;                 // low key bits that are always zero (they carry the position when packed)
  int packed;
  int with_row;           // CSR rows: positions are stored with their row, as {position, row} pairs
  int nb_bits;            // log2(number of buckets)
  u32 NB, NBINS;          // buckets; NB + kHotMax
  u32 G, chunk;           // walk CTAs and elements per CTA
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
  u32* cold_base;         // [NB + 1]
  u32* pos_base;          // [NB + 1]
  u32* hot_base;          // [kHotMax + 1]
  u64* shot_key; u32* shot_h;       // hot keys sorted by key
  u32* bucket_hot_off;    // [NB + 1]
  u32* hot_u; u32* hot_seg;         // [kHotMax]
  u32* bstate;            // [NB]
  u32* row_hint;          // [n / 32 + 2], with row_ptr only: the row of every 32nd position
  u64* cold_words; u32* cold_pos; u32* hot_pos;
  // outputs
  u64* ukeys; u32* seg_off; u32* csr_col; u32* csc_row; float* csc_val;
  u32* flagbits; u32* wordbase; u32* n_unique;
  u32* status;
};

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
  return row_search(p.row_ptr, p.row_hint[b], min(p.row_hint[b + 1] + 1, p.n_rows), pos);
}

// ---------------------------------------------------------------- 0. clean scratch
// Everything that starts as zeros or ones, and the row hints, in one launch instead of one per region.
__global__ void __launch_bounds__(256) k_bl_clear(const BLP p, uint4* zero, u32 zero4, uint4* ones, u32 ones4, u32 flag_words) {
  const u32 gsize = gridDim.x * blockDim.x, gtid = blockIdx.x * blockDim.x + threadIdx.x;
  for (u32 i = gtid; i < zero4; i += gsize) zero[i] = make_uint4(0, 0, 0, 0);
  for (u32 i = gtid; i < ones4; i += gsize) ones[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
  for (u32 i = gtid; i < flag_words; i += gsize) p.flagbits[i] = 0;
  if (p.row_ptr != nullptr) {
    // row hints for steps 5 and 6, up to the block behind the last position
    const u32 nh = ((p.n - 1) >> kHintShift) + 2;
    for (u32 h = gtid; h < nh; h += gsize) p.row_hint[h] = row_search(p.row_ptr, 0, p.n_rows, h << kHintShift);
  }
}

// ---------------------------------------------------------------- 1. sample
__global__ void __launch_bounds__(256) k_bl_sample(const BLP p) {
  const u32 j = blockIdx.x * blockDim.x + threadIdx.x;
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

__global__ void __launch_bounds__(256) k_bl_hot(const BLP p) {
  const u32 s = blockIdx.x * blockDim.x + threadIdx.x;
  const u32 c = s < p.samp_slots ? p.samp_cnt[s] : 0u;
  // distinct keys of the sample (how much keys repeat decides the size of the buckets' tables)
  const u32 occ = __ballot_sync(0xffffffffu, c > 0);
  if ((threadIdx.x & 31) == 0 && occ) atomicAdd(&p.ctl[kCtlSampleDistinct], (u32)__popc(occ));
  if (c < p.hot_thresh) return;
  const u64 key = p.samp_key[s];
  const u32 h = atomicAdd(&p.ctl[kCtlNumHot], 1u);
  if (h >= kHotMax) return;                                    // more candidates than places: the rest stay cold
  p.hot_key[h] = key;
  const u32 hash = hot_hash(key), entry = ((hash & 0xFFFFFu) << 11) | h;
  u32 slot = (hash >> 20) * 4;
  for (u32 probe = 0; probe < kHotSlots; ++probe) {
    if (atomicCAS(&p.hot_tab[slot], kHotNone, entry) == kHotNone) return;
    slot = (slot + 1) & (kHotSlots - 1);
  }
}

// ---------------------------------------------------------------- 2./4. the two walks
// Shared-memory layout of a walk CTA: hot table | hot keys | one word per bin.
// kRow: CSR rows, positions are stored as {position, row} pairs (fixed-length rows do not pay for them).
// kScatter = false: count. kScatter = true: the words start as this CTA's output cursors.
template <bool kScatter, bool kRow>
__global__ void __launch_bounds__(kWalkThreads) k_bl_walk(const BLP p) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint4* s_hot = reinterpret_cast<uint4*>(smem);
  u64* s_hkey = reinterpret_cast<u64*>(smem + kHotSlots * 4);
  u32* s_bin = reinterpret_cast<u32*>(smem + kHotSlots * 4 + kHotMax * 8);
  if (kScatter && p.ctl[kCtlFallback]) return;
  const u32 nh = min(p.ctl[kCtlNumHot], kHotMax);
  const int t = threadIdx.x;
  for (u32 i = t; i < kHotBuckets; i += kWalkThreads) s_hot[i] = reinterpret_cast<const uint4*>(p.hot_tab)[i];
  for (u32 i = t; i < nh; i += kWalkThreads) s_hkey[i] = p.hot_key[i];
  u32* my_part = p.part + (size_t)blockIdx.x * p.NBINS;
  for (u32 i = t; i < p.NBINS; i += kWalkThreads) {
    u32 v = 0;
    if (kScatter) v = my_part[i] + (i < p.NB ? p.cold_base[i] : p.hot_base[i - p.NB]);
    s_bin[i] = v;
  }
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
  // Four elements: all look-ups, then all counts (when scattering: output places from the bins' cursors), then
  // all stores, so that no element waits for another's chain. Plain shared-memory atomics, also for the hot
  // keys: lanes that hit one address serialise inside the instruction, which costs far less than finding the
  // groups first.
  auto handle = [&](const u64 (&key)[4], u32 pos, u32 nvalid) {
    u32 bin[4], dst[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) bin[q] = (u32)q < nvalid ? bin_of(key[q]) : 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if ((u32)q < nvalid) dst[q] = atomicAdd(&s_bin[bin[q]], 1u);
    if constexpr (kScatter) {
      // The row of a position is found here, where neighbouring threads look at neighbouring rows, and travels
      // with it: looked up where the nonzeros arrive in key order, it is three dependent random loads each
      // (3.9 M nonzeros: bucket and hot emit kernels 130 + 51 us that way, 100 + 32 us so, this walk 49 -> 65).
      u32 row = kRow ? row_of_pos(p, pos, 0) : 0u;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if ((u32)q >= nvalid) break;
        if (kRow) {
          if (row + 1 < p.n_rows && p.row_ptr[row + 1] <= pos + q) {
            ++row;
            // behind a run of empty rows: searched, since one thread would walk all of it (20,000 nonzeros with
            // 100,000 empty rows in their midst: 7.0 ms row by row, 0.09 ms like this, as without them)
            if (row + 1 < p.n_rows && p.row_ptr[row + 1] <= pos + q) row = row_of_pos(p, pos + q, 0);
          }
          const uint2 pr = make_uint2(pos + q, row);
          if (bin[q] >= p.NB) {
            reinterpret_cast<uint2*>(p.hot_pos)[dst[q]] = pr;
          } else {
            p.cold_words[dst[q]] = key[q];
            reinterpret_cast<uint2*>(p.cold_pos)[dst[q]] = pr;
          }
        } else if (bin[q] >= p.NB) {
          p.hot_pos[dst[q]] = pos + q;
        } else if (p.packed) {
          p.cold_words[dst[q]] = key[q] | (u64)(pos + q);
        } else {
          p.cold_words[dst[q]] = key[q];
          p.cold_pos[dst[q]] = pos + q;
        }
      }
    }
  };
  // Four consecutive elements per thread and trip, the next trip's loads in flight while these are handled.
  const u32 step = 4u * kWalkThreads;
  if (p.in_kind == 1 && (((size_t)p.in) & 15) == 0) {
    // 32-bit ids: one 16-byte load per trip
    const u32* ids = (const u32*)p.in;
    u32 i = begin + 4u * t;
    uint4 cur = make_uint4(0, 0, 0, 0);
    if (i + 3 < end) cur = *reinterpret_cast<const uint4*>(ids + i);
    for (; i < end; i += step) {
      uint4 nxt = make_uint4(0, 0, 0, 0);
      if (i + step + 3 < end) nxt = *reinterpret_cast<const uint4*>(ids + i + step);
      u32 id[4] = {cur.x, cur.y, cur.z, cur.w};
      const u32 nvalid = min(4u, end - i);
      if (nvalid < 4) {
#pragma unroll
        for (int q = 0; q < 4; ++q) id[q] = (u32)q < nvalid ? ids[i + q] : 0u;
      }
      u64 key[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) key[q] = hash_id_to_key(id[q], p.seed);
      handle(key, i, nvalid);
      cur = nxt;
    }
  } else {
    u64 nxt[4];
    auto fetch = [&](u32 i) {
      if (p.in_kind == 0 && i + 3 < end && (((size_t)p.in) & 15) == 0) {
        const ulonglong2* v = reinterpret_cast<const ulonglong2*>((const u64*)p.in + i);
        const ulonglong2 a = v[0], c = v[1];
        nxt[0] = a.x; nxt[1] = a.y; nxt[2] = c.x; nxt[3] = c.y;
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) nxt[q] = (i + q < end) ? bl_key_of(p, i + q) : 0;
      }
    };
    u32 i = begin + 4u * t;
    fetch(i);
    for (; i < end; i += step) {
      const u64 key[4] = {nxt[0], nxt[1], nxt[2], nxt[3]};
      fetch(i + step);
      handle(key, i, min(4u, end - i));
    }
  }
  if (!kScatter) {
    __syncthreads();
    for (u32 i = t; i < p.NBINS; i += kWalkThreads) my_part[i] = s_bin[i];
  }
}

// ---------------------------------------------------------------- 3. scan + plan
// Per bin: exclusive prefix over the walk CTAs (in place) and the bin's total.
__global__ void __launch_bounds__(256) k_bl_scan(const BLP p) {
  const u32 bin = blockIdx.x * blockDim.x + threadIdx.x;
  if (bin >= p.NBINS) return;
  u32 run = 0;
  // sixteen CTAs' counts are fetched before the first prefix is stored
  for (u32 c0 = 0; c0 < p.G; c0 += 16) {
    u32 v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = (c0 + k < p.G) ? p.part[(size_t)(c0 + k) * p.NBINS + bin] : 0u;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      if (c0 + k < p.G) p.part[(size_t)(c0 + k) * p.NBINS + bin] = run;
      run += v[k];
    }
  }
  p.bin_total[bin] = run;
}

// One CTA: the hot keys grouped by bucket, the hot stream's offsets, and per bucket the cold stream
// offset, the final output offset and its first hot key. Every thread owns adjacent buckets and two adjacent hot
// keys, kept in registers; the four prefix sums go through one block scan, and four buckets go out in one store:
// a lone SM is bound by the number of sectors it asks for. 8192 buckets: 9 us (18 us as four scans of arrays in
// shared memory, and as long with one scan and a store per bucket), all of it on the critical path.
static constexpr int kPlanPer = kMaxBuckets / 1024;               // buckets per thread at most
__device__ __forceinline__ u32 plan_pad(u32 i) { return i + (i >> 5); }   // adjacent entries of a thread: no bank conflicts
__global__ void __launch_bounds__(1024) k_bl_plan(const BLP p) {
  extern __shared__ __align__(16) unsigned char smem[];
  u32* s_hn = reinterpret_cast<u32*>(smem);         // [NB, padded] hot nonzeros per bucket
  u32* s_hc = s_hn + plan_pad(p.NB);                // [NB, padded] hot keys per bucket, then the place of the next one
  __shared__ u32 s_tot[4][32];
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
  // {cold nonzeros, all nonzeros, hot keys, nonzeros of hot keys} before this thread's buckets and hot keys
  u32 v[4] = {0, 0, 0, ht[0] + ht[1]}, mx = 0;
#pragma unroll
  for (int k = 0; k < kPlanPer; ++k)
    if ((u32)k < per && b0 + k < p.NB) {
      const u32 b = plan_pad(b0 + k);
      v[0] += cold[k]; v[1] += cold[k] + s_hn[b]; v[2] += s_hc[b];
      mx = max(mx, cold[k]);
    }
  atomicMax(&s_max, mx);
  u32 x[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    x[q] = v[q];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(0xffffffffu, x[q], o);
      if (lane >= o) x[q] += y;
    }
    if (lane == 31) s_tot[q][w] = x[q];
  }
  __syncthreads();
  if (w < 4) {                                      // warp q turns the 32 totals of value q into prefixes
    u32 y = s_tot[w][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 z = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += z;
    }
    s_tot[w][lane] = y;
  }
  __syncthreads();
  u32 run[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) run[q] = (w ? s_tot[q][w - 1] : 0u) + x[q] - v[q];
  __align__(16) u32 out[3][kPlanPer];
#pragma unroll
  for (int k = 0; k < kPlanPer; ++k)
    if ((u32)k < per && b0 + k < p.NB) {
      const u32 b = plan_pad(b0 + k), c = s_hc[b];
      out[0][k] = run[0]; out[1][k] = run[1]; out[2][k] = run[2];
      run[0] += cold[k]; run[1] += cold[k] + s_hn[b];
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
  *reinterpret_cast<uint2*>(p.hot_base + 2 * t) = make_uint2(run[3], run[3] + ht[0]);
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
    p.hot_base[kHotMax] = s_tot[3][31];
    p.ctl[kCtlHotElems] = s_tot[3][31];
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

template <typename CK, int kBits, bool kRow>
__global__ void __launch_bounds__(kBucketThreads) k_bl_bucket(const BLP p) {
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
  __shared__ u32 s_ovf, s_b, s_ubase, s_warp[kBucketThreads / 32 + 1];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  // A CTA takes buckets by ticket until none is left (a few CTAs per SM are launched, not one per bucket).
  for (;;) {
  if (t == 0) {
    // one thread reads the flags for the whole CTA: other CTAs may raise the fallback flag at any moment
    const bool mine = (p.ctl[kCtlBigTables] != 0) == (kBits == 12);
    s_b = (!mine || ld_relaxed_gpu(&p.ctl[kCtlFallback])) ? 0xFFFFFFFFu : atomicAdd(&p.ctl[kCtlTicket], 1u);
    s_ovf = 0;
  }
  {
    // keys = all ones, counts = 0, bitmaps = 0, with 16-byte stores (while the ticket is on its way)
    uint4* k4 = reinterpret_cast<uint4*>(s_key);
    const u32 nk4 = kHsAll * sizeof(CK) / 16;
    for (u32 i = t; i < nk4; i += kBucketThreads) k4[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    uint4* c4 = reinterpret_cast<uint4*>(s_cnt);
    for (u32 i = t; i < kHsAll / 4; i += kBucketThreads) c4[i] = make_uint4(0, 0, 0, 0);
    for (u32 i = t; i < 2 * kHsWords; i += kBucketThreads) s_bits[i] = 0;
  }
  __syncthreads();
  const u32 b = s_b;
  if (b >= p.NB) return;
  const u32 cb = p.cold_base[b], nb = p.cold_base[b + 1] - cb;
  const u32 pb = p.pos_base[b];
  const u32 h0 = p.bucket_hot_off[b], h1 = p.bucket_hot_off[b + 1];
  const int sh_l = p.nb_bits, sh_r = p.nb_bits + p.lo;
  const int rem = 64 - sh_r;                    // significant bits of a compact key
  const u64 posmask = p.packed ? ((1ull << p.lo) - 1) : 0ull;
  // The first four nonzeros of every thread stay in registers for both passes over the bucket
  // (a bucket of average size has no more), the rest is read again in pass 2.
  u64 w0[4];
  uint2 p0[4];                                     // position, and with kRow its row
  auto position = [&](u32 j) -> uint2 {
    if (kRow) return reinterpret_cast<const uint2*>(p.cold_pos)[cb + j];
    return make_uint2(p.packed ? 0u : p.cold_pos[cb + j], 0u);
  };
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const u32 j = t + q * kBucketThreads;
    w0[q] = j < nb ? p.cold_words[cb + j] : 0;
    p0[q] = j < nb ? position(j) : make_uint2(0u, 0u);
  }
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
    if (t == 0) { st_relaxed_gpu(&p.ctl[kCtlFallback], 1u); st_relaxed_gpu(&p.bstate[b], kFlagIncl); }
    return;
  }
  // the bucket's number of unique keys is known: publish it for the buckets behind
  if (t == 0) st_relaxed_gpu(&p.bstate[b], (b == 0 ? kFlagIncl : kFlagAgg) | d);
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
  // unique keys in all buckets before this one: look back over the published counts
  if (w == 0) {
    u32 ex = 0;
    if (b > 0) {
      long long q = (long long)b - 1;
      u32 spins = 0;
      bool done = false;
      while (!done && q >= 0) {
        // 4 x 32 buckets are fetched per round trip to L2 and consumed from the nearest on
        u32 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const long long idx = q - 32 * k - lane;
          v[k] = kFlagIncl;
          if (idx >= 0) v[k] = ld_relaxed_gpu(p.bstate + idx);
        }
        u32 add = 0;
        int taken = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (done || taken < 32 * k) continue;    // warp-uniform
          const u32 f = v[k] & ~kValMask;
          const u32 empty = __ballot_sync(0xffffffffu, f == 0);
          const u32 incl = __ballot_sync(0xffffffffu, f == kFlagIncl);
          const int first_empty = empty ? __ffs(empty) - 1 : 32;
          const int first_incl = incl ? __ffs(incl) - 1 : 32;
          const int upto = first_incl < first_empty ? first_incl + 1 : first_empty;   // lanes [0, upto) are usable
          if (lane < upto) add += v[k] & kValMask;
          taken += upto;
          if (first_incl < first_empty) done = true;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
        ex += add;
        if (!done) {
          q -= taken;
          if (taken == 0) {
            // a bucket that gave up (or never started because of that) publishes nothing: stop waiting
            if (ld_relaxed_gpu(&p.ctl[kCtlFallback])) break;
            if (++spins > kGridWaitIters) { if (lane == 0) set_status(p.status, kLookbackTimeout); break; }
            __nanosleep(40);
          }
        }
      }
      if (lane == 0) st_relaxed_gpu(&p.bstate[b], kFlagIncl | ((ex + d) & kValMask));
    }
    if (lane == 0) {
      s_ubase = ex;
      if (b == p.NB - 1) *p.n_unique = ex + d;
    }
  }
  __syncthreads();
  if (s_ovf) {
    if (t == 0) st_relaxed_gpu(&p.ctl[kCtlFallback], 1u);
    return;
  }
  const u32 ub = s_ubase;
  const u64 bucket_bits = (u64)b << (64 - p.nb_bits);
#pragma unroll
  for (int k = 0; k < kEntriesPerThread; ++k) {
    if (my_rank[k] == 0xFFFFFFFFu) continue;
    const u32 slot = s_dense[t + k * kBucketThreads];
    const u32 c = s_cnt[slot];
    const bool is_hot = (s_hbits[slot >> 5] >> (slot & 31)) & 1u;
    const u32 hh = is_hot ? s_rank[slot] : 0u;
    const u32 start = my_start[k];
    s_cnt[slot] = start;
    s_rank[slot] = (unsigned short)my_rank[k];
    const u32 u = ub + my_rank[k], P = pb + start;
    p.ukeys[u] = bucket_bits | ((u64)s_key[slot] << p.lo);
    p.seg_off[u] = P;
    atomicOr(&p.flagbits[P >> 5], 1u << (P & 31));
    if (is_hot) {
      p.hot_u[hh] = u;          // the hot emit kernel fills this segment (and its wordbase words)
      p.hot_seg[hh] = P;
    } else {
      // number of segment heads before every 32-aligned position inside the segment
      for (u32 wd = (P + 31) >> 5; (wd << 5) < P + c; ++wd) p.wordbase[wd] = ((wd << 5) == P) ? u : u + 1;
    }
  }
  __syncthreads();
  // pass 2: every nonzero to its place
  const u32 zinv = p.fixed_z ? (u32)(0xffffffffu / p.fixed_z) : 0u;
  for (u32 j0 = t; j0 < nb; j0 += 4 * kBucketThreads) {
    u64 wd[4];
    uint2 ps[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 j = j0 + q * kBucketThreads;
      const bool first = j0 == (u32)t;
      wd[q] = first ? w0[q] : (j < nb ? p.cold_words[cb + j] : 0);
      ps[q] = first ? p0[q] : (j < nb ? position(j) : make_uint2(0u, 0u));
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 j = j0 + q * kBucketThreads;
      if (j >= nb) break;
      const CK ck = (CK)((wd[q] << sh_l) >> sh_r);
      const int slot = bucket_find<CK, kBits>(s_key, ck, rem);
      if (slot < 0) continue;                     // cannot happen: the key was inserted in pass 1
      const u32 pos = p.packed && !kRow ? (u32)(wd[q] & posmask) : ps[q].x;
      const u32 P = pb + atomicAdd(&s_cnt[slot], 1u);
      const u32 u = ub + s_rank[slot];
      p.csc_row[P] = kRow ? ps[q].y : row_of_pos(p, pos, zinv);
      p.csr_col[pos] = u;
      if (p.csc_val) p.csc_val[P] = p.vals[pos];
    }
  }
  __syncthreads();       // the tables are rebuilt for the next bucket
  }
}

// ---------------------------------------------------------------- 6. hot keys' position lists
template <bool kRow>
__global__ void __launch_bounds__(256) k_bl_hot_emit(const BLP p) {
  __shared__ u32 s_base[kHotMax + 1];
  __shared__ u32 s_u[kHotMax], s_seg[kHotMax];
  if (p.ctl[kCtlFallback]) return;
  const u32 nh = min(p.ctl[kCtlNumHot], kHotMax);
  if (nh == 0) return;
  for (u32 i = threadIdx.x; i <= nh; i += blockDim.x) s_base[i] = p.hot_base[i];
  for (u32 i = threadIdx.x; i < nh; i += blockDim.x) { s_u[i] = p.hot_u[i]; s_seg[i] = p.hot_seg[i]; }
  __syncthreads();
  const u32 total = s_base[nh];
  const u32 zinv = p.fixed_z ? (u32)(0xffffffffu / p.fixed_z) : 0u;
  // A warp walks one contiguous piece of the hot stream, 4 x 32 positions per trip. The stream is
  // grouped by hot key, so the key index only ever moves forward: one binary search at the start.
  const int lane = threadIdx.x & 31;
  const u32 nwarps = gridDim.x * (blockDim.x >> 5);
  const u32 gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const u32 piece = ((total + nwarps - 1) / nwarps + 127) & ~127u;
  const u32 begin = min(total, gw * piece), end = min(total, begin + piece);
  if (begin >= end) return;
  u32 h;
  {
    u32 lo = 0, hi = nh;                            // largest h with s_base[h] <= begin
    while (hi - lo > 1) {
      u32 mid = (lo + hi) >> 1;
      if (s_base[mid] <= begin) lo = mid; else hi = mid;
    }
    h = lo;
  }
  for (u32 j0 = begin + lane; j0 < end + lane; j0 += 128) {
    u32 pos[4], row[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 j = j0 + q * 32;
      uint2 pr = make_uint2(0u, 0u);
      if (j < end) {
        if (kRow) pr = __ldcs(&reinterpret_cast<const uint2*>(p.hot_pos)[j]);
        else pr.x = __ldcs(&p.hot_pos[j]);
      }
      pos[q] = pr.x; row[q] = pr.y;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const u32 j = j0 + q * 32;
      if (j >= end) break;
      while (h + 1 < nh && s_base[h + 1] <= j) ++h;
      const u32 u = s_u[h];
      const u32 P = s_seg[h] + (j - s_base[h]);
      p.csc_row[P] = kRow ? row[q] : row_of_pos(p, pos[q], zinv);
      p.csr_col[pos[q]] = u;
      if (p.csc_val) p.csc_val[P] = p.vals[pos[q]];
      if ((P & 31u) == 0) p.wordbase[P >> 5] = (j == s_base[h]) ? u : u + 1;
    }
  }
}

// scratch layout (bytes), shared by the size query and the launcher
struct BlLayout {
  size_t zero_begin, samp_cnt, ctl, bstate, zero_end;
  size_t ff_begin, samp_key, hot_tab, ff_end;
  size_t hot_key, part, bin_total, cold_base, pos_base, hot_base, shot_key, shot_h, bucket_hot_off,
      hot_u, hot_seg, row_hint, total;
};
static size_t al(size_t x) { return (x + 255) & ~(size_t)255; }
static BlLayout bl_layout(u32 NB, u32 G, u32 n, u32 samp_slots) {
  BlLayout L;
  size_t o = 0;
  const u32 NBINS = NB + kHotMax;
  L.zero_begin = o;
  L.samp_cnt = o; o = al(o + (size_t)samp_slots * 4);
  L.ctl = o; o = al(o + kCtlWords * 4);
  L.bstate = o; o = al(o + (size_t)NB * 4);
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
  L.hot_base = o; o = al(o + (kHotMax + 1) * 4);
  L.shot_key = o; o = al(o + kHotMax * 8);
  L.shot_h = o; o = al(o + kHotMax * 4);
  L.bucket_hot_off = o; o = al(o + (size_t)(NB + 1) * 4);
  L.hot_u = o; o = al(o + kHotMax * 4);
  L.hot_seg = o; o = al(o + kHotMax * 4);
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
static int bl_walk_ctas() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

}  // namespace psb

using namespace psb;

extern "C" size_t psb_bucket_localize_scratch_bytes(uint32_t max_n) {
  // sized for the largest bucket count; the per-nonzero buffers are the caller's
  return bl_layout(kMaxBuckets, (u32)bl_walk_ctas(), max_n, kSampSlots).total;
}

// Groups the n nonzeros of a minibatch by key. Inputs as for psb_sort_pairs (in, in_kind, seed);
// low_zero_bits = number of low key bits that are zero in every key (64 - significant bits of a
// narrow hashed key); when n - 1 fits in them the position rides in the key word (no cold_pos needed).
// cold_words (n x 8 bytes), cold_pos (n x 4 bytes, may be null when the positions fit) and hot_pos
// (n x 4 bytes) are work buffers; with row_ptr cold_pos is always needed and both are n x 8 bytes. Outputs as for psb_localize2. *gate_out (device word) is set to 1
// when the caller must run the gated sort-based path instead (its outputs then replace these).
extern "C" int psb_bucket_localize(const void* in, int in_kind, psb_u64 seed, uint32_t n, int low_zero_bits,
                                   const uint32_t* row_ptr, uint32_t n_rows, uint32_t fixed_z,
                                   const float* vals, const psb_u64* bounds, int S,
                                   psb_u64* cold_words, uint32_t* cold_pos, uint32_t* hot_pos,
                                   psb_u64* ukeys, uint32_t* seg_off, uint32_t* csr_col, uint32_t* csc_row,
                                   float* csc_val, uint32_t* flagbits, uint32_t* wordbase,
                                   uint32_t* n_unique, uint32_t* own_off, void* scratch, uint32_t* status,
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
  BLP p{};
  p.in = in; p.in_kind = in_kind; p.seed = seed; p.n = n;
  p.lo = low_zero_bits;
  p.packed = (low_zero_bits > 0 && (low_zero_bits >= 32 || ((n - 1) >> low_zero_bits) == 0)) ? 1 : 0;
  if ((!p.packed || row_ptr != nullptr) && cold_pos == nullptr) return -(int)cudaErrorInvalidValue;
  p.with_row = row_ptr != nullptr ? 1 : 0;
  p.NB = bl_num_buckets(n);
  p.nb_bits = 0;
  while ((1u << p.nb_bits) < p.NB) ++p.nb_bits;
  p.NBINS = p.NB + kHotMax;
  // walk CTAs: one per SM, and no more than get a full trip of 4096 elements (every CTA fills its shared tables
  // first, and the scan over the CTAs' counts is a serial chain)
  p.G = min((u32)bl_walk_ctas(), (n + 4 * kWalkThreads - 1) / (4 * kWalkThreads));
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
  p.hot_base = (u32*)(sc + L.hot_base); p.shot_key = (u64*)(sc + L.shot_key); p.shot_h = (u32*)(sc + L.shot_h);
  p.bucket_hot_off = (u32*)(sc + L.bucket_hot_off); p.hot_u = (u32*)(sc + L.hot_u);
  p.hot_seg = (u32*)(sc + L.hot_seg); p.row_hint = (u32*)(sc + L.row_hint); p.bstate = (u32*)(sc + L.bstate);
  p.cold_words = (u64*)cold_words; p.cold_pos = cold_pos; p.hot_pos = hot_pos;
  p.ukeys = (u64*)ukeys; p.seg_off = seg_off; p.csr_col = csr_col; p.csc_row = csc_row; p.csc_val = csc_val;
  p.flagbits = flagbits; p.wordbase = wordbase; p.n_unique = n_unique; p.status = status;

  const u32 zero4 = (u32)((L.zero_end - L.zero_begin) / 16), ones4 = (u32)((L.ff_end - L.ff_begin) / 16);
  k_bl_clear<<<psb_device_sm_count() * 2, 256, 0, stream>>>(p, (uint4*)(sc + L.zero_begin), zero4, (uint4*)(sc + L.ff_begin),
                                                            ones4, (n + 31) / 32);
  k_bl_sample<<<(p.samp_m + 255) / 256, 256, 0, stream>>>(p);
  k_bl_hot<<<(p.samp_slots + 255) / 256, 256, 0, stream>>>(p);
  const size_t walk_smem = kHotSlots * 4 + kHotMax * 8 + (size_t)p.NBINS * 4;
  static bool attr_set = false;
  const int remaining = 64 - p.nb_bits - p.lo;      // key bits that distinguish keys inside a bucket
  const bool ck32 = remaining <= 31;
  const size_t plan_smem = (size_t)(p.NB + p.NB / 32) * 8;
  if (!attr_set) {
    const size_t walk_max = kHotSlots * 4 + kHotMax * 8 + (size_t)(kMaxBuckets + kHotMax) * 4;
    cudaFuncSetAttribute((const void*)k_bl_plan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)((kMaxBuckets + kMaxBuckets / 32) * 8));
    cudaFuncSetAttribute((const void*)k_bl_walk<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_max);
    cudaFuncSetAttribute((const void*)k_bl_walk<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_max);
    cudaFuncSetAttribute((const void*)k_bl_walk<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_max);
    cudaFuncSetAttribute((const void*)k_bl_bucket<u32, 11, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BucketShape<11>::smem_bytes(4));
    cudaFuncSetAttribute((const void*)k_bl_bucket<u32, 11, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BucketShape<11>::smem_bytes(4));
    cudaFuncSetAttribute((const void*)k_bl_bucket<u32, 12, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BucketShape<12>::smem_bytes(4));
    cudaFuncSetAttribute((const void*)k_bl_bucket<u32, 12, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BucketShape<12>::smem_bytes(4));
    cudaFuncSetAttribute((const void*)k_bl_bucket<u64, 11, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BucketShape<11>::smem_bytes(8));
    cudaFuncSetAttribute((const void*)k_bl_bucket<u64, 11, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BucketShape<11>::smem_bytes(8));
    cudaFuncSetAttribute((const void*)k_bl_bucket<u64, 12, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BucketShape<12>::smem_bytes(8));
    cudaFuncSetAttribute((const void*)k_bl_bucket<u64, 12, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BucketShape<12>::smem_bytes(8));
    attr_set = true;
  }
  k_bl_walk<false, false><<<p.G, kWalkThreads, walk_smem, stream>>>(p);
  k_bl_scan<<<(p.NBINS + 255) / 256, 256, 0, stream>>>(p);
  k_bl_plan<<<1, 1024, plan_smem, stream>>>(p);
  if (p.with_row) k_bl_walk<true, true><<<p.G, kWalkThreads, walk_smem, stream>>>(p);
  else k_bl_walk<true, false><<<p.G, kWalkThreads, walk_smem, stream>>>(p);
  const u32 sms = (u32)bl_walk_ctas(), g11 = min(p.NB, sms * 6), g12 = min(p.NB, sms * 4);
  auto buckets = [&](auto row) {
    constexpr bool kRow = decltype(row)::value;
    if (ck32) {
      k_bl_bucket<u32, 11, kRow><<<g11, kBucketThreads, BucketShape<11>::smem_bytes(4), stream>>>(p);
      k_bl_bucket<u32, 12, kRow><<<g12, kBucketThreads, BucketShape<12>::smem_bytes(4), stream>>>(p);
    } else {
      k_bl_bucket<u64, 11, kRow><<<g11, kBucketThreads, BucketShape<11>::smem_bytes(8), stream>>>(p);
      k_bl_bucket<u64, 12, kRow><<<g12, kBucketThreads, BucketShape<12>::smem_bytes(8), stream>>>(p);
    }
    k_bl_hot_emit<kRow><<<min(sms * 8, (n + 1023) / 1024), 256, 0, stream>>>(p);
  };
  if (p.with_row) buckets(std::true_type()); else buckets(std::false_type());
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return -(int)e;
  return psb_owner_offsets_n(ukeys, n_unique, bounds, S, n, seg_off, own_off, p.ctl + kCtlFallback, gate_out, stream);
}
