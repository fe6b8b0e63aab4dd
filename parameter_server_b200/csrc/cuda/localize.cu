// Minibatch localisation on the device: from the sorted (key, position) pairs
// produce the sorted unique key list, the CSC segment offsets, the CSR column
// remap and the per-owner slice offsets.
//
// Reference behaviour: Localizer::CountUniqIndex + RemapIndex
// (util/localizer.h:97-221) and the key-range slicing of
// SliceKOFVMessage (system/message.h:107-147). Here the sort already groups
// equal keys, so "unique + counts" is a head-flag scan, the remap is a scatter
// of the unique index back to each nonzero's original position, and slicing
// is S+1 binary searches over the unique keys.
//
// Kernels: k_uniq_count (heads per tile) -> k_uniq_scan (tile bases, U) ->
// k_uniq_emit (everything else) -> k_owner_offsets.
#include "psb_common.cuh"
#include "psb_cuda.h"

namespace psb {

static constexpr int kLocThreads = 256;
static constexpr int kLocItems = 16;
static constexpr int kLocTile = kLocThreads * kLocItems;  // 4096 = 128 flag words

// Loads the warp's 16 x 32 consecutive keys starting at `base` (all requested
// before the first is used) and returns, per item, the ballot of segment heads.
// kmask selects the key bits (all ones, or without the packed position bits).
__device__ __forceinline__ void warp_heads(const u64* __restrict__ keys, u32 n, u32 base, int lane, u64 kmask,
                                           u64 (&k)[kLocItems], u32 (&bal)[kLocItems]) {
#pragma unroll
  for (int i = 0; i < kLocItems; ++i) {
    u32 g = base + i * 32 + lane;
    k[i] = g < n ? keys[g] : 0;
  }
  u64 before = (lane == 0 && base > 0 && base < n) ? keys[base - 1] : 0;   // last key before the warp's span
#pragma unroll
  for (int i = 0; i < kLocItems; ++i) {
    u32 g = base + i * 32 + lane;
    u64 prev = __shfl_up_sync(0xffffffffu, k[i], 1);
    u64 carry = __shfl_sync(0xffffffffu, i ? k[i ? i - 1 : 0] : before, i ? 31 : 0);
    if (lane == 0) prev = carry;
    bool head = g < n && (g == 0 || (k[i] & kmask) != (prev & kmask));
    bal[i] = __ballot_sync(0xffffffffu, head);
  }
}

__device__ __forceinline__ void uniq_count_tile(const u64* keys, u32 n, u32 tile, u32* __restrict__ tile_heads, u64 kmask) {
  __shared__ u32 s_w[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const u32 base = tile * (u32)kLocTile + w * (32 * kLocItems);
  u64 k[kLocItems];
  u32 bal[kLocItems];
  warp_heads(keys, n, base, lane, kmask, k, bal);
  u32 cnt = 0;
#pragma unroll
  for (int i = 0; i < kLocItems; ++i) cnt += __popc(bal[i]);
  if (lane == 0) s_w[w] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    u32 t = 0;
    for (int i = 0; i < 8; ++i) t += s_w[i];
    tile_heads[tile] = t;
  }
}
__global__ void __launch_bounds__(kLocThreads) k_uniq_count(const u64* __restrict__ keys_a,
                                                            const u64* __restrict__ keys_b,
                                                            const u32* __restrict__ where, u32 n,
                                                            u32* __restrict__ tile_heads, u64 kmask) {
  uniq_count_tile((where && *where) ? keys_b : keys_a, n, blockIdx.x, tile_heads, kmask);
}

// One CTA (any number of whole warps): exclusive scan of tile_heads in place; writes U.
__device__ __forceinline__ void uniq_scan(u32* tile_heads, u32 ntiles, u32* __restrict__ n_unique) {
  __shared__ u32 s_warp[32];
  __shared__ u32 s_carry;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (u32 base = 0; base < ntiles; base += blockDim.x) {
    u32 i = base + threadIdx.x;
    u32 v = i < ntiles ? __ldcg(&tile_heads[i]) : 0;
    u32 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      u32 y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {
      u32 t = lane < nw ? s_warp[lane] : 0u;
      u32 xs = t;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        u32 y = __shfl_up_sync(0xffffffffu, xs, o);
        if (lane >= o) xs += y;
      }
      s_warp[lane] = xs - t;
    }
    __syncthreads();
    u32 carry = s_carry;
    if (i < ntiles) tile_heads[i] = carry + s_warp[w] + x - v;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) s_carry = carry + s_warp[w] + x;
    __syncthreads();
  }
  if (threadIdx.x == 0) *n_unique = s_carry;
}
__global__ void __launch_bounds__(1024) k_uniq_scan(u32* __restrict__ tile_heads, u32 ntiles, u32* __restrict__ n_unique) {
  uniq_scan(tile_heads, ntiles, n_unique);
}

// Emits, for the sorted pairs (keys[i], pos[i]) held in buffer A or B (*where):
//   ukeys[u], seg_off[u] at segment heads (seg_off[U] = n),
//   csr_col[pos[i]] = u            (CSR remap to local column ids),
//   csc_row[i] = row of pos[i]     (the CSC row index),
//   csc_val[i] = vals[pos[i]]      (only when vals != null),
//   flagbits[i/32], wordbase[i/32] (head bitmap and heads before each word).
// Row of a position: pos / fixed_z when row_ptr is null, else the row whose
// [row_ptr[r], row_ptr[r+1]) contains it.
__device__ __forceinline__ void uniq_emit_tile(
    const u64* keys, const u32* pos, u32* csc_row /* may alias pos */, u32 n, u32 tile, const u32* tile_base,
    const u32* __restrict__ row_ptr, u32 n_rows, u32 fixed_z, const float* __restrict__ vals,
    u64* __restrict__ ukeys, u32* __restrict__ seg_off, u32* __restrict__ csr_col,
    float* __restrict__ csc_val, u32* __restrict__ flagbits, u32* __restrict__ wordbase, u64 kmask) {
  __shared__ u32 s_w[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const u32 base = tile * (u32)kLocTile + w * (32 * kLocItems);
  u64 key[kLocItems];
  u32 bal[kLocItems];
  warp_heads(keys, n, base, lane, kmask, key, bal);
  u32 cnt = 0;
#pragma unroll
  for (int i = 0; i < kLocItems; ++i) cnt += __popc(bal[i]);
  if (lane == 0) s_w[w] = cnt;
  __syncthreads();
  u32 run = __ldcg(&tile_base[tile]);
  for (int i = 0; i < w; ++i) run += s_w[i];
  const u32 zinv = fixed_z ? (u32)(0xffffffffu / fixed_z) : 0u;   // umulhi(p, zinv) <= p / fixed_z, short by at most 2
  const u32 le = 0xffffffffu >> (31 - lane);
#pragma unroll
  for (int i = 0; i < kLocItems; ++i) {
    u32 g = base + i * 32 + lane;
    if (g - lane < n && lane == 0) {
      flagbits[g >> 5] = bal[i];
      wordbase[g >> 5] = run;
    }
    if (g < n) {
      u32 u = run + __popc(bal[i] & le) - 1;
      if ((bal[i] >> lane) & 1u) {
        ukeys[u] = key[i] & kmask;
        seg_off[u] = g;
      }
      u32 p = pos ? pos[g] : (u32)(key[i] & ~kmask);   // packed: the position rides in the key's low bits
      csr_col[p] = u;
      if (csc_val) csc_val[g] = vals[p];
      u32 r;
      if (row_ptr == nullptr) {
        r = __umulhi(p, zinv);
        while (p - r * fixed_z >= fixed_z) ++r;   // the estimate is at most two short
      } else {
        u32 lo = 0, hi = n_rows;  // largest r with row_ptr[r] <= p
        while (hi - lo > 1) {
          u32 mid = (lo + hi) >> 1;
          if (row_ptr[mid] <= p) lo = mid; else hi = mid;
        }
        r = lo;
      }
      csc_row[g] = r;
    }
    run += __popc(bal[i]);
  }
}
__global__ void __launch_bounds__(kLocThreads) k_uniq_emit(
    const u64* __restrict__ keys_a, const u64* __restrict__ keys_b, const u32* pos_a,
    const u32* pos_b, const u32* __restrict__ where, u32* csc_row /* may alias pos */, u32 n,
    const u32* __restrict__ tile_base,
    const u32* __restrict__ row_ptr, u32 n_rows, u32 fixed_z, const float* __restrict__ vals,
    u64* __restrict__ ukeys, u32* __restrict__ seg_off, u32* __restrict__ csr_col,
    float* __restrict__ csc_val, u32* __restrict__ flagbits, u32* __restrict__ wordbase, u64 kmask) {
  const bool in_b = where && *where;
  uniq_emit_tile(in_b ? keys_b : keys_a, in_b ? pos_b : pos_a, csc_row, n, blockIdx.x, tile_base, row_ptr, n_rows, fixed_z,
                 vals, ukeys, seg_off, csr_col, csc_val, flagbits, wordbase, kmask);
}

// own_off[s] = lower_bound(ukeys[0..U), bounds[s]) for s in 0..S; own_off[S] = U.
// Also closes the CSC offsets with seg_off[U] = n.
// One warp per boundary: 32 probes side by side cut the range by 33 per trip, where a lone thread would wait
// for log2(U) dependent loads (6 us with 2.7 M keys).
__device__ __forceinline__ void owner_offsets(const u64* ukeys, u32 U, const u64* __restrict__ bounds, int S, u32 n,
                                              u32* seg_off, u32* __restrict__ own_off) {
  const u32 lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    if (seg_off) seg_off[U] = n;
    own_off[S] = U;
  }
  for (int s = threadIdx.x >> 5; s < S; s += blockDim.x >> 5) {
    const u64 b = bounds[s];
    u32 lo = 0, hi = U;                            // the answer lies in [lo, hi]
    while (lo < hi) {
      const u32 step = (hi - lo + 32) / 33;        // probes at lo + step - 1, lo + 2 * step - 1, ..
      const u64 at = (u64)lo + (u64)(lane + 1) * step - 1;
      const bool below = at < hi && __ldcg(&ukeys[at]) < b;
      const u32 k = (u32)__popc(__ballot_sync(0xffffffffu, below));
      const u64 end = (u64)lo + (u64)(k + 1) * step - 1;    // the first probe that is not below (k < 32)
      lo += k * step;
      if (k < 32 && end < hi) hi = (u32)end;
    }
    if (lane == 0) own_off[s] = lo;
  }
}
__global__ void __launch_bounds__(256) k_owner_offsets(const u64* __restrict__ ukeys, const u32* __restrict__ n_unique,
                                                       const u64* __restrict__ bounds, int S, u32 n,
                                                       u32* __restrict__ seg_off, u32* __restrict__ own_off) {
  owner_offsets(ukeys, *n_unique, bounds, S, n, seg_off, own_off);
}

// A key list handed in by the caller: into the request's own buffer, with its length and owner offsets.
__global__ void __launch_bounds__(256) k_set_keys(const u64* __restrict__ keys, u32 n, u64* __restrict__ ukeys,
                                                  u32* __restrict__ n_unique, const u64* __restrict__ bounds, int S,
                                                  u32* __restrict__ own_off) {
  const u32 gsize = gridDim.x * blockDim.x;
  for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += 4 * gsize) {
    u64 k[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) k[q] = i + q * gsize < n ? keys[i + q * gsize] : 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (i + q * gsize < n) ukeys[i + q * gsize] = k[q];
  }
  if (blockIdx.x != gridDim.x - 1) return;
  if (threadIdx.x == 0) *n_unique = n;
  owner_offsets(keys, n, bounds, S, n, nullptr, own_off);
}

// The four steps behind a device word, in one cooperative launch (see k_sort_gated).
struct GatedLocalize {
  const u64 *keys_a, *keys_b; const u32 *pos_a, *pos_b; const u32* where; u32* csc_row; u32 n;
  const u32* row_ptr; u32 n_rows, fixed_z; const float* vals; const u64* bounds; int S;
  u64* ukeys; u32 *seg_off, *csr_col; float* csc_val; u32 *flagbits, *wordbase, *n_unique, *own_off;
  u32* tile_heads; u32* bar; u64 kmask; const u32* gate; u32* status;
};
__global__ void __launch_bounds__(kLocThreads) k_localize_gated(const GatedLocalize a) {
  if (*a.gate == 0) return;
  const u32 ntiles = (a.n + kLocTile - 1) / kLocTile;
  const bool in_b = a.where && *a.where;
  const u64* keys = in_b ? a.keys_b : a.keys_a;
  for (u32 tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    uniq_count_tile(keys, a.n, tile, a.tile_heads, a.kmask);
    __syncthreads();
  }
  if (!grid_barrier(a.bar, a.status)) return;
  if (blockIdx.x == 0) uniq_scan(a.tile_heads, ntiles, a.n_unique);
  if (!grid_barrier(a.bar, a.status)) return;
  for (u32 tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    uniq_emit_tile(keys, in_b ? a.pos_b : a.pos_a, a.csc_row, a.n, tile, a.tile_heads, a.row_ptr, a.n_rows, a.fixed_z, a.vals,
                   a.ukeys, a.seg_off, a.csr_col, a.csc_val, a.flagbits, a.wordbase, a.kmask);
    __syncthreads();
  }
  if (!grid_barrier(a.bar, a.status)) return;
  if (blockIdx.x == 0) owner_offsets(a.ukeys, __ldcg(a.n_unique), a.bounds, a.S, a.n, a.seg_off, a.own_off);
}

}  // namespace psb

using namespace psb;

// Owner slice offsets of an already sorted unique key list (generic Push/Pull
// path): own_off[s] = lower_bound(ukeys, bounds[s]), own_off[S] = *n_unique.
extern "C" int psb_owner_offsets(const psb_u64* ukeys, const uint32_t* n_unique, const psb_u64* bounds, int S,
                                 uint32_t* own_off, cudaStream_t stream) {
  if (S < 1 || S > 64) return -(int)cudaErrorInvalidValue;
  k_owner_offsets<<<1, 256, 0, stream>>>((const u64*)ukeys, n_unique, (const u64*)bounds, S, 0, nullptr, own_off);
  return -(int)cudaGetLastError();
}

extern "C" int psb_set_keys(const psb_u64* keys, uint32_t n, psb_u64* ukeys, uint32_t* n_unique, const psb_u64* bounds,
                            int S, uint32_t* own_off, cudaStream_t stream) {
  if (S < 1 || S > 64) return -(int)cudaErrorInvalidValue;
  const u32 blocks = (n + 1023) / 1024, most = (u32)psb_device_sm_count() * 8;
  k_set_keys<<<min(most, max(1u, blocks)), 256, 0, stream>>>((const u64*)keys, n, (u64*)ukeys, n_unique, (const u64*)bounds, S,
                                                             own_off);
  return -(int)cudaGetLastError();
}

extern "C" size_t psb_localize_scratch_bytes(uint32_t n) {
  size_t ntiles = (n + kLocTile - 1) / kLocTile;
  return sizeof(u32) * (ntiles + 16);
}

// The sorted pairs are in (keys_a, pos_a) when *where == 0 (or where is null) and
// in (keys_b, pos_b) otherwise. csc_row may alias the selected pos buffer.
static int localize2_impl(const psb_u64* keys_a, const psb_u64* keys_b, const uint32_t* pos_a,
                          const uint32_t* pos_b, const uint32_t* where, uint32_t* csc_row, uint32_t n,
                          const uint32_t* row_ptr, uint32_t n_rows, uint32_t fixed_z,
                          const float* vals, const psb_u64* bounds, int S, psb_u64* ukeys,
                          uint32_t* seg_off, uint32_t* csr_col, float* csc_val,
                          uint32_t* flagbits, uint32_t* wordbase, uint32_t* n_unique,
                          uint32_t* own_off, void* scratch, int pack_pos_bits, const uint32_t* gate,
                          uint32_t* status, cudaStream_t stream) {
  if (S < 1 || S > 64) return -(int)cudaErrorInvalidValue;
  if (row_ptr == nullptr && fixed_z == 0) return -(int)cudaErrorInvalidValue;
  if (pack_pos_bits < 0 || pack_pos_bits > 32) return -(int)cudaErrorInvalidValue;
  const u64 kmask = pack_pos_bits ? ~((1ull << pack_pos_bits) - 1) : ~0ull;
  if (pack_pos_bits) pos_a = pos_b = nullptr;
  u32 ntiles = (n + kLocTile - 1) / kLocTile;
  u32* tile_heads = (u32*)scratch;
  if (n == 0) {
    cudaMemsetAsync(n_unique, 0, sizeof(u32), stream);
    cudaMemsetAsync(own_off, 0, sizeof(u32) * (S + 1), stream);
    cudaMemsetAsync(seg_off, 0, sizeof(u32), stream);
    return -(int)cudaGetLastError();
  }
  if (gate != nullptr) {
    u32* bar = const_cast<u32*>(gate) + 3;             // see psb_sort_pairs_gated
    static int per_sm = 0;
    if (per_sm == 0) {
      int per = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)k_localize_gated, kLocThreads, 0);
      per_sm = per < 1 ? 1 : (per > 4 ? 4 : per);
    }
    GatedLocalize a{(const u64*)keys_a, (const u64*)keys_b, pos_a, pos_b, where, csc_row, n, row_ptr, n_rows, fixed_z, vals,
                    (const u64*)bounds, S, (u64*)ukeys, seg_off, csr_col, csc_val, flagbits, wordbase, n_unique, own_off,
                    tile_heads, bar, kmask, gate, status};
    void* args[] = {&a};
    return -(int)cudaLaunchCooperativeKernel((const void*)k_localize_gated,
                                             dim3(min(ntiles, (u32)(psb_device_sm_count() * per_sm))), dim3(kLocThreads),
                                             args, 0, stream);
  }
  k_uniq_count<<<ntiles, kLocThreads, 0, stream>>>((const u64*)keys_a, (const u64*)keys_b, where, n, tile_heads, kmask);
  k_uniq_scan<<<1, 1024, 0, stream>>>(tile_heads, ntiles, n_unique);
  k_uniq_emit<<<ntiles, kLocThreads, 0, stream>>>((const u64*)keys_a, (const u64*)keys_b, pos_a, pos_b, where, csc_row,
                                                  n, tile_heads, row_ptr, n_rows, fixed_z, vals, (u64*)ukeys, seg_off,
                                                  csr_col, csc_val, flagbits, wordbase, kmask);
  k_owner_offsets<<<1, 256, 0, stream>>>((const u64*)ukeys, n_unique, (const u64*)bounds, S, n, seg_off, own_off);
  return -(int)cudaGetLastError();
}

extern "C" int psb_localize2(const psb_u64* keys_a, const psb_u64* keys_b, const uint32_t* pos_a,
                             const uint32_t* pos_b, const uint32_t* where, uint32_t* csc_row, uint32_t n,
                             const uint32_t* row_ptr, uint32_t n_rows, uint32_t fixed_z,
                             const float* vals, const psb_u64* bounds, int S, psb_u64* ukeys,
                             uint32_t* seg_off, uint32_t* csr_col, float* csc_val,
                             uint32_t* flagbits, uint32_t* wordbase, uint32_t* n_unique,
                             uint32_t* own_off, void* scratch, int pack_pos_bits, cudaStream_t stream) {
  return localize2_impl(keys_a, keys_b, pos_a, pos_b, where, csc_row, n, row_ptr, n_rows, fixed_z, vals, bounds, S,
                        ukeys, seg_off, csr_col, csc_val, flagbits, wordbase, n_unique, own_off, scratch,
                        pack_pos_bits, nullptr, nullptr, stream);
}

// Same, but nothing happens unless the device word *gate is non-zero (null: always; see k_localize_gated).
extern "C" int psb_localize2_gated(const psb_u64* keys_a, const psb_u64* keys_b, const uint32_t* pos_a,
                                   const uint32_t* pos_b, const uint32_t* where, uint32_t* csc_row, uint32_t n,
                                   const uint32_t* row_ptr, uint32_t n_rows, uint32_t fixed_z,
                                   const float* vals, const psb_u64* bounds, int S, psb_u64* ukeys,
                                   uint32_t* seg_off, uint32_t* csr_col, float* csc_val,
                                   uint32_t* flagbits, uint32_t* wordbase, uint32_t* n_unique,
                                   uint32_t* own_off, void* scratch, int pack_pos_bits, const uint32_t* gate,
                                   uint32_t* status, cudaStream_t stream) {
  return localize2_impl(keys_a, keys_b, pos_a, pos_b, where, csc_row, n, row_ptr, n_rows, fixed_z, vals, bounds, S,
                        ukeys, seg_off, csr_col, csc_val, flagbits, wordbase, n_unique, own_off, scratch,
                        pack_pos_bits, gate, status, stream);
}

// Sorted pairs in one buffer; sorted_pos is rewritten in place with the CSC row index.
extern "C" int psb_localize(const psb_u64* sorted_keys, uint32_t* sorted_pos, uint32_t n,
                            const uint32_t* row_ptr, uint32_t n_rows, uint32_t fixed_z,
                            const float* vals, const psb_u64* bounds, int S, psb_u64* ukeys,
                            uint32_t* seg_off, uint32_t* csr_col, float* csc_val,
                            uint32_t* flagbits, uint32_t* wordbase, uint32_t* n_unique,
                            uint32_t* own_off, void* scratch, cudaStream_t stream) {
  if (S < 1 || S > 64) return -(int)cudaErrorInvalidValue;
  if (row_ptr == nullptr && fixed_z == 0) return -(int)cudaErrorInvalidValue;
  u32 ntiles = (n + kLocTile - 1) / kLocTile;
  u32* tile_heads = (u32*)scratch;
  if (n == 0) {
    cudaMemsetAsync(n_unique, 0, sizeof(u32), stream);
    cudaMemsetAsync(own_off, 0, sizeof(u32) * (S + 1), stream);
    cudaMemsetAsync(seg_off, 0, sizeof(u32), stream);
    return -(int)cudaGetLastError();
  }
  k_uniq_count<<<ntiles, kLocThreads, 0, stream>>>((const u64*)sorted_keys, nullptr, nullptr, n, tile_heads, ~0ull);
  k_uniq_scan<<<1, 1024, 0, stream>>>(tile_heads, ntiles, n_unique);
  k_uniq_emit<<<ntiles, kLocThreads, 0, stream>>>((const u64*)sorted_keys, nullptr, sorted_pos, nullptr, nullptr,
                                                  sorted_pos, n, tile_heads, row_ptr, n_rows, fixed_z, vals,
                                                  (u64*)ukeys, seg_off, csr_col, csc_val, flagbits, wordbase, ~0ull);
  k_owner_offsets<<<1, 256, 0, stream>>>((const u64*)ukeys, n_unique, (const u64*)bounds, S, n, seg_off, own_off);
  return -(int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Allocation-free variant (declared in psb_noalloc.h; nothing like it exists in
// the reference). The per-tile head counts, which psb_localize keeps in a
// caller-provided scratch buffer, live in this fixed device array instead.
#include <mutex>
#include "psb_noalloc.h"

static __device__ __align__(256) unsigned int g_localize_static_scratch[PSB_LOCALIZE_STATIC_SCRATCH_WORDS];

namespace {
// In host code the array's name is only a handle for the runtime, not an
// address a kernel can use; the device address is looked up once per device,
// with that device current.
constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
void* g_static_ptr[kMaxDevices] = {nullptr};

int localize_static_scratch(void** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return -(int)e;
  if (dev < 0 || dev >= kMaxDevices) return -(int)cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (g_static_ptr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_localize_static_scratch);
    if (e != cudaSuccess) return -(int)e;
    g_static_ptr[dev] = p;
  }
  *out = g_static_ptr[dev];
  return 0;
}
}  // namespace

extern "C" int psb_localize_static(const psb_u64* sorted_keys, uint32_t* sorted_pos, uint32_t n,
                                   const uint32_t* row_ptr, uint32_t n_rows, uint32_t fixed_z,
                                   const float* vals, const psb_u64* bounds, int S, psb_u64* ukeys,
                                   uint32_t* seg_off, uint32_t* csr_col, float* csc_val,
                                   uint32_t* flagbits, uint32_t* wordbase, uint32_t* n_unique,
                                   uint32_t* own_off, cudaStream_t stream) {
  if (n > PSB_LOCALIZE_STATIC_MAX_N) return -(int)cudaErrorInvalidValue;  // beyond the built-in scratch
  if (S < 1 || S > 64) return -(int)cudaErrorInvalidValue;
  if (row_ptr == nullptr && fixed_z == 0) return -(int)cudaErrorInvalidValue;
  void* scratch = nullptr;
  int rc = localize_static_scratch(&scratch);
  if (rc != 0) return rc;
  u32* tile_heads = (u32*)scratch;
  if (n == 0) {
    cudaMemsetAsync(n_unique, 0, sizeof(u32), stream);
    cudaMemsetAsync(own_off, 0, sizeof(u32) * (S + 1), stream);
    cudaMemsetAsync(seg_off, 0, sizeof(u32), stream);
    return -(int)cudaGetLastError();
  }
  const u32 ntiles = (n + kLocTile - 1) / kLocTile;
  // every tile_heads word that the scan and the emit kernel read is written by
  // k_uniq_count first, so the array needs no clearing between calls
  k_uniq_count<<<ntiles, kLocThreads, 0, stream>>>((const u64*)sorted_keys, nullptr, nullptr, n, tile_heads, ~0ull);
  k_uniq_scan<<<1, 1024, 0, stream>>>(tile_heads, ntiles, n_unique);
  k_uniq_emit<<<ntiles, kLocThreads, 0, stream>>>((const u64*)sorted_keys, nullptr, sorted_pos, nullptr, nullptr,
                                                  sorted_pos, n, tile_heads, row_ptr, n_rows, fixed_z, vals,
                                                  (u64*)ukeys, seg_off, csr_col, csc_val, flagbits, wordbase, ~0ull);
  k_owner_offsets<<<1, 256, 0, stream>>>((const u64*)ukeys, n_unique, (const u64*)bounds, S, n, seg_off,
                                         own_off);
  return -(int)cudaGetLastError();
}
