// KV store: variable-size byte values over the map, the way a key-value
// store uses a slab hash (the reference's KVCG tests keep pointers to values
// in the map, test/slabunified_test.cu:360-380).  Values live in one device
// byte heap; the map holds key -> handle, handle = heap offset << 24 | length
// (offsets below 2^40, values of at most 2^24 - 1 bytes).
//
//   put     the batch's values arrive packed in one device buffer with n + 1
//           offsets (op i's bytes are vals[off[i] .. off[i+1])); they are
//           copied to the heap in one piece, each op gets its handle, and the
//           map takes the handles as a put batch (ops in index order, so the
//           last put of a key wins).  Space of replaced values becomes
//           garbage until lsb_kvs_compact.
//   get     handles by a read batch; lengths out; then the bytes of the found
//           values are copied to the caller's buffer at offsets that are the
//           exclusive prefix sums of the lengths (computed on the device).
//   remove  a map remove; the value's space becomes garbage.
//
// No counterpart in the reference's library itself (lslab maps fixed-size
// values only).
#include <cuda_runtime.h>

#include <algorithm>
#include <new>

#include "lsb.h"
#include "lsb_core.cuh"
#include "lsb_internal.h"

namespace {

constexpr uint64_t kLenBits = 24;
constexpr uint64_t kMaxLen = (1ull << kLenBits) - 1;
constexpr uint64_t kMaxHeap = 1ull << 40;

__device__ __forceinline__ uint32_t h_len(uint64_t h) { return (uint32_t)(h & kMaxLen); }
__device__ __forceinline__ uint64_t h_off(uint64_t h) { return h >> kLenBits; }

// What the host reads of a call, in pinned host memory that the kernels write
// to directly: one wait for the stream gives it all, where copies of single
// words each cost a transfer and a wait (three in a put: 75-100 us of host
// time a call, 30-40 this way).
struct HostWords {
  uint64_t first, last;  // put: the batch's first and last offset
  uint64_t total;        // get, compact: bytes of all found (live) values
  uint64_t count;        // compact: live entries
  uint64_t end;          // compact: the largest end of a live value in the heap
  uint32_t bad;          // put: a value longer than kMaxLen or offsets that fall
  uint32_t pad;
};

// handle[i] = (base + off[i] - off[0]) << 24 | (off[i+1] - off[i]); a length
// over the limit raises words->bad.
__global__ void k_handles(const uint64_t* off, uint64_t base, uint64_t* handle, uint32_t n,
                          HostWords* words) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t a = off[i], b = off[i + 1];
  if (i == 0) words->first = a;
  if (i == n - 1) words->last = b;
  if (b < a || b - a > kMaxLen) {
    *(volatile uint32_t*)&words->bad = 1u;
    handle[i] = 0;
    return;
  }
  handle[i] = ((base + a - off[0]) << kLenBits) | (b - a);
}

// Garbage accounting: bytes of the values that a put or remove replaced.
__global__ void k_dead_bytes(const lsb_result* res, const uint64_t* old, uint32_t n,
                             unsigned long long* dead) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint64_t v = 0;
  if (i < n) {
    if (res) v = res[i].found ? h_len(res[i].value) : 0;
    else v = h_len(old[i]);  // a put's old handle (0 when the key was absent)
  }
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, d);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(dead, (unsigned long long)v);
}

// Prefix sums over up to 2^32 items in two launches: each of at most kParts
// blocks sums its part of them (k_*_sums), then each adds up the sums of the
// parts before its own and walks its part again in tiles of one item a thread.
// No block waits for another.  (One block of 1024 threads, each walking n /
// 1024 consecutive items twice, took 151 us for 32768 lengths; the two launches
// take 7.)
constexpr uint32_t kParts = 1024;
constexpr uint32_t kSums = 5;  // words behind the parts, of k_live
constexpr uint32_t kPartThreads = 256;

inline uint32_t part_size(uint64_t n) {  // a multiple of the block, at least 4 tiles
  const uint64_t per = (n + kParts - 1) / kParts;
  return (uint32_t)std::max<uint64_t>(4 * kPartThreads,
                                      (per + kPartThreads - 1) / kPartThreads * kPartThreads);
}
inline uint32_t part_count(uint64_t n) { return (uint32_t)((n + part_size(n) - 1) / part_size(n)); }

// Sum of one value per thread over the block (kPartThreads); every thread gets it.
__device__ __forceinline__ uint64_t block_sum(uint64_t v) {
  __shared__ uint64_t s_sum[kPartThreads / 32];
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
  __syncthreads();  // the previous call's readers
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = v;
  __syncthreads();
  uint64_t t = 0;
  for (uint32_t k = 0; k < kPartThreads / 32; ++k) t += s_sum[k];
  return t;
}

// Sum of the parts before this block's.
__device__ __forceinline__ uint64_t parts_before(const uint64_t* parts) {
  uint64_t v = 0;
  for (uint32_t k = threadIdx.x; k < blockIdx.x; k += kPartThreads) v += parts[k];
  return block_sum(v);
}

// Exclusive prefix of one length per thread (below 2^24 each, so a tile's sum
// fits 32 bits); *total receives the tile's sum.
__device__ __forceinline__ uint32_t tile_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t s_warp[kPartThreads / 32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
    if (lane >= d) x += y;
  }
  __syncthreads();
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  uint32_t before = 0, all = 0;
  for (uint32_t k = 0; k < kPartThreads / 32; ++k) {
    if (k < warp) before += s_warp[k];
    all += s_warp[k];
  }
  *total = all;
  return before + x - v;
}

__device__ __forceinline__ uint32_t found_len(const lsb_result* res, uint32_t j, bool* found) {
  const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(res + j);  // our own array: 16-aligned
  *found = (r.x & 0xFFu) != 0;
  return *found ? h_len(r.y) : 0u;
}

__global__ void __launch_bounds__(kPartThreads)
    k_length_sums(const lsb_result* res, uint32_t n, uint32_t part, uint64_t* parts) {
  const uint64_t j0 = (uint64_t)blockIdx.x * part, j1 = j0 + part < n ? j0 + part : n;
  uint64_t v = 0;
  bool found;
  for (uint64_t j = j0 + threadIdx.x; j < j1; j += kPartThreads)
    v += found_len(res, (uint32_t)j, &found);
  v = block_sum(v);
  if (threadIdx.x == 0) parts[blockIdx.x] = v;
}

// Lengths of the looked-up values (0 when absent) and their exclusive prefix
// sums; the last block knows the total.
__global__ void __launch_bounds__(kPartThreads)
    k_length_offsets(const lsb_result* res, uint32_t n, uint32_t part, const uint64_t* parts,
                     uint32_t* len, uint64_t* dst_off, uint8_t* found_out, HostWords* words) {
  uint64_t run = parts_before(parts);
  const uint64_t j0 = (uint64_t)blockIdx.x * part, j1 = j0 + part < n ? j0 + part : n;
  for (uint64_t t0 = j0; t0 < j1; t0 += kPartThreads) {
    const uint64_t j = t0 + threadIdx.x;
    bool found = false;
    const uint32_t l = j < j1 ? found_len(res, (uint32_t)j, &found) : 0u;
    uint32_t total;
    const uint32_t before = tile_scan(l, &total);
    if (j < j1) {
      len[j] = l;
      dst_off[j] = run + before;
      if (found_out) found_out[j] = found;
    }
    run += total;
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) words->total = run;
}

// Copy len bytes by kCopyLanes lanes of a warp (lane l of them): aligned
// 32-bit stores, each from the one or two aligned source words that hold its
// bytes, kCopyBatch words a lane loaded before any is stored, so that a value
// of 2 KB takes four round trips and not one per word.  Source words are read
// only where they hold at least one of the bytes; the source array's size is
// rounded up to whole words.  (A whole warp a value, a byte a lane, moved 32768
// values of 210 bytes in 24 us; 8.7 this way.)
constexpr uint32_t kCopyLanes = 16;
constexpr uint32_t kCopyBatch = 8;

__device__ __forceinline__ void copy_value(uint8_t* dst, const uint8_t* src, uint32_t len,
                                           uint32_t l) {
  const uint32_t to_word = (uint32_t)(-(uintptr_t)dst) & 3u;
  const uint32_t head = to_word < len ? to_word : len;
  const uint32_t words = (len - head) / 4;
  const uint8_t* from = src + head;
  const uint32_t shift = 8 * ((uint32_t)(uintptr_t)from & 3u);
  const uint32_t* sw = reinterpret_cast<const uint32_t*>((uintptr_t)from & ~(uintptr_t)3);
  uint32_t* dw = reinterpret_cast<uint32_t*>(dst + head);
  const uint32_t done = head + 4 * words;
  // the ragged ends: at most 3 bytes each
  const uint32_t e = l < head ? l : done + l - head;
  const bool end = e < len && l < head + (len - done);
  const uint8_t byte = end ? src[e] : (uint8_t)0;
  for (uint32_t w0 = l; w0 < words; w0 += kCopyLanes * kCopyBatch) {
    uint32_t lo[kCopyBatch], hi[kCopyBatch];
#pragma unroll
    for (uint32_t k = 0; k < kCopyBatch; ++k) {
      const uint32_t w = w0 + k * kCopyLanes;
      lo[k] = w < words ? sw[w] : 0u;
      hi[k] = w < words && shift ? sw[w + 1] : 0u;
    }
#pragma unroll
    for (uint32_t k = 0; k < kCopyBatch; ++k) {
      const uint32_t w = w0 + k * kCopyLanes;
      if (w < words) dw[w] = __funnelshift_r(lo[k], hi[k], shift);
    }
  }
  if (end) dst[e] = byte;
}

// Copy each found value's bytes from the heap to dst + dst_off[i]; values that
// would end past cap are skipped.
__global__ void __launch_bounds__(256)
    k_gather(const lsb_result* res, const uint64_t* dst_off, const uint8_t* heap, uint8_t* dst,
             uint64_t cap, uint32_t n) {
  const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / kCopyLanes;
  if (i >= n || !res[i].found) return;
  const uint64_t h = res[i].value, o = dst_off[i];
  const uint32_t l = h_len(h);
  if (o + l > cap) return;
  copy_value(dst + o, heap + h_off(h), l, threadIdx.x % kCopyLanes);
}

// ------------------------------------------------------- heap compaction
// The live entries of a table as (key, address of the slot's value): a warp
// per bucket, a lane per slot.  With keys == nullptr only counts them, their
// values' bytes and where the last of these ends into *words (through
// sums[0..1] and sums[4], cleared by the caller, of which sums[2] blocks are
// done).
__global__ void __launch_bounds__(256)
    k_live(lsb::TableView t, uint32_t buckets, uint64_t* keys, uint64_t** slots, uint64_t cap,
           unsigned long long* sums, HostWords* words) {
  using Tr = lsb::MapTraits;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  uint64_t count = 0, bytes = 0, end = 0;
  for (uint64_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < buckets; b += nw) {
    uint32_t s = (uint32_t)b;
    for (uint32_t hop = 0; hop < lsb::kMaxHops; ++hop) {
      uint8_t* slab = lsb::slab_ptr(t.slabs, s, Tr::kSlabBytes);
      const lsb::Meta m = lsb::load_meta(slab);
      const uint32_t live = lsb::live_mask(m);
      const bool mine = (live >> lane) & 1u;  // lanes 28..31 have no slot
      const uint8_t* sp = slab + lsb::kMetaBytes + lane * Tr::kSlotBytes;
      if (keys == nullptr) {
        if (mine) {
          const uint64_t h = lsb::ld_cg_u64(sp + 8);
          ++count;
          bytes += h_len(h);
          end = max(end, h_off(h) + h_len(h));
        }
      } else if (live) {
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&sums[3], (unsigned long long)__popc(live));
        at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(live & ((1u << lane) - 1u));
        if (mine && at < cap) {
          keys[at] = lsb::ld_cg_u64(sp);
          slots[at] = (uint64_t*)(sp + 8);
        }
      }
      if (m.next == 0) break;
      s = m.next;
    }
  }
  if (keys != nullptr) return;
  __shared__ int last;
  for (int d = 16; d > 0; d >>= 1) end = max(end, __shfl_xor_sync(0xFFFFFFFFu, end, d));
  if (lane == 0 && end) atomicMax(&sums[4], (unsigned long long)end);
  count = block_sum(count);
  bytes = block_sum(bytes);
  if (threadIdx.x == 0) {
    atomicAdd(&sums[0], (unsigned long long)count);
    atomicAdd(&sums[1], (unsigned long long)bytes);
    __threadfence();
    last = atomicAdd(&sums[2], 1ull) == gridDim.x - 1;
    if (last) {
      __threadfence();
      words->count = atomicAdd(&sums[0], 0ull);
      words->total = atomicAdd(&sums[1], 0ull);
      words->end = atomicMax(&sums[4], 0ull);
    }
  }
}

// One pass of a stable radix sort of (key, slot) pairs by an 8-bit digit of the
// key: digit counts per block, then each block places its pairs behind those
// of smaller digits and of earlier blocks.  Eight passes order the entries by
// key on the device; copying them out, sorting on the host and copying back
// was most of a compaction's 3.1 ms at 32768 entries (about 0.2 now, 75 us of
// it the eight passes).
constexpr uint32_t kDigits = 256;
constexpr uint32_t kSortTile = 2048;  // pairs a block ranks at a time, 8 a thread

inline uint32_t sort_part(uint64_t n) {
  const uint64_t per = (n + kParts - 1) / kParts;
  return (uint32_t)std::max<uint64_t>(kSortTile, (per + kSortTile - 1) / kSortTile * kSortTile);
}

__global__ void __launch_bounds__(kDigits)
    k_digit_counts(const uint64_t* keys, uint64_t n, uint32_t part, uint32_t shift,
                   uint32_t* counts) {
  __shared__ uint32_t c[kDigits];
  c[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t j0 = (uint64_t)blockIdx.x * part, j1 = j0 + part < n ? j0 + part : n;
  for (uint64_t j = j0 + threadIdx.x; j < j1; j += kDigits)
    atomicAdd(&c[(keys[j] >> shift) & (kDigits - 1)], 1u);
  __syncthreads();
  counts[(size_t)blockIdx.x * kDigits + threadIdx.x] = c[threadIdx.x];
}

__global__ void __launch_bounds__(kDigits)
    k_digit_place(const uint64_t* keys, uint64_t* const* slots, uint64_t n, uint32_t part,
                  uint32_t shift, const uint32_t* counts, uint64_t* keys_out, uint64_t** slots_out) {
  constexpr uint32_t kWarps = kDigits / 32, kPer = kSortTile / kDigits;
  __shared__ uint64_t s_base[kDigits];        // next place of a digit
  __shared__ uint64_t s_place[kWarps][kDigits];
  __shared__ uint32_t s_count[kWarps][kDigits];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this digit's pairs in earlier blocks, and in all
  uint64_t before = 0, all = 0;
  for (uint32_t b = 0; b < gridDim.x; ++b) {
    const uint32_t c = counts[(size_t)b * kDigits + tid];
    if (b < blockIdx.x) before += c;
    all += c;
  }
  uint64_t x = all;  // inclusive prefix over the digits
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) s_place[0][warp] = x;
  __syncthreads();
  uint64_t smaller = x - all;  // pairs of smaller digits
  for (uint32_t w = 0; w < warp; ++w) smaller += s_place[0][w];
  s_base[tid] = smaller + before;
  const uint64_t j0 = (uint64_t)blockIdx.x * part, j1 = j0 + part < n ? j0 + part : n;
  for (uint64_t t0 = j0; t0 < j1; t0 += kSortTile) {
    for (uint32_t w = 0; w < kWarps; ++w) s_count[w][tid] = 0;
    __syncthreads();
    // a warp ranks its kPer * 32 consecutive pairs in order
    const uint64_t w0 = t0 + (uint64_t)warp * kPer * 32;
    uint64_t key[kPer];
    uint64_t* slot[kPer];
    uint32_t rank[kPer];
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
      const uint64_t j = w0 + k * 32 + lane;
      key[k] = j < j1 ? keys[j] : 0;
      slot[k] = j < j1 ? slots[j] : nullptr;
    }
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
      const bool in = w0 + k * 32 + lane < j1;
      const uint32_t d = in ? (uint32_t)(key[k] >> shift) & (kDigits - 1) : kDigits;
      const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
      rank[k] = (in ? s_count[warp][d] : 0u) + __popc(peers & ((1u << lane) - 1u));
      __syncwarp();
      if (in && lane == (uint32_t)__ffs(peers) - 1) s_count[warp][d] += __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    uint64_t at = s_base[tid];
    for (uint32_t w = 0; w < kWarps; ++w) {
      s_place[w][tid] = at;
      at += s_count[w][tid];
    }
    s_base[tid] = at;
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
      const uint64_t j = w0 + k * 32 + lane;
      if (j < j1) {
        const uint64_t p = s_place[warp][(key[k] >> shift) & (kDigits - 1)] + rank[k];
        if (p < n) {
          keys_out[p] = key[k];
          slots_out[p] = slot[k];
        }
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kPartThreads)
    k_slot_sums(uint64_t* const* slots, uint64_t n, uint32_t part, uint64_t* parts) {
  const uint64_t j0 = (uint64_t)blockIdx.x * part, j1 = j0 + part < n ? j0 + part : n;
  uint64_t v = 0;
  for (uint64_t j = j0 + threadIdx.x; j < j1; j += kPartThreads)
    v += h_len(lsb::ld_cg_u64(slots[j]));
  v = block_sum(v);
  if (threadIdx.x == 0) parts[blockIdx.x] = v;
}

// New handles (the values packed in the order of `slots`) into the slots; the
// old ones to old_handles.
__global__ void __launch_bounds__(kPartThreads)
    k_new_handles(uint64_t* const* slots, uint64_t n, uint32_t part, const uint64_t* parts,
                  uint64_t* old_handles) {
  uint64_t run = parts_before(parts);
  const uint64_t j0 = (uint64_t)blockIdx.x * part, j1 = j0 + part < n ? j0 + part : n;
  for (uint64_t t0 = j0; t0 < j1; t0 += kPartThreads) {
    const uint64_t j = t0 + threadIdx.x;
    uint64_t* slot = j < j1 ? slots[j] : nullptr;
    const uint64_t h = slot ? lsb::ld_cg_u64(slot) : 0ull;
    uint32_t total;
    const uint64_t at = run + tile_scan(h_len(h), &total);
    if (slot) {
      lsb::st_cg_u64(slot, (at << kLenBits) | h_len(h));
      old_handles[j] = h;
    }
    run += total;
  }
}

// The values to the staging copy: value j from its old place to its new one.
__global__ void __launch_bounds__(256)
    k_move(uint64_t* const* slots, const uint64_t* old_handles, uint64_t n, const uint8_t* heap,
           uint8_t* stage, uint64_t stage_bytes) {
  const uint64_t j = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / kCopyLanes;
  if (j >= n) return;
  const uint64_t h = old_handles[j], at = h_off(lsb::ld_cg_u64(slots[j]));
  if (at + h_len(h) <= stage_bytes)
    copy_value(stage + at, heap + h_off(h), h_len(h), threadIdx.x % kCopyLanes);
}

}  // namespace

struct lsb_kvs {
  lsb_map* map = nullptr;
  uint8_t* heap = nullptr;
  uint64_t heap_cap = 0;
  uint64_t heap_used = 0;      // bump cursor (host-side: every allocation goes through put)
  unsigned long long* dead = nullptr;  // device: bytes of replaced values
  HostWords* words = nullptr;  // pinned, mapped
  HostWords* d_words = nullptr;  // the same for the device
  uint64_t* parts = nullptr;   // device: kParts partial sums, then k_live's sums
  uint64_t* tmp = nullptr;     // device scratch: handles / old handles
  lsb_result* res = nullptr;   // device scratch: lookup results
  uint32_t tmp_cap = 0;
  uint8_t* work = nullptr;     // device scratch of compact, kept while small
  uint64_t work_bytes = 0;
};

namespace {

// scratch of compact that is kept for the next call
constexpr uint64_t kWorkKept = 64ull << 20;

int ensure_tmp(lsb_kvs* s, size_t n) {
  if (n <= s->tmp_cap) return LSB_OK;
  cudaFree(s->tmp);
  cudaFree(s->res);
  s->tmp = nullptr;
  s->res = nullptr;
  s->tmp_cap = 0;
  if (cudaMalloc(&s->tmp, sizeof(uint64_t) * 2 * (n + 1)) != cudaSuccess ||
      cudaMalloc(&s->res, sizeof(lsb_result) * n) != cudaSuccess) {
    cudaGetLastError();
    return LSB_ERR_OOM;
  }
  s->tmp_cap = (uint32_t)n;
  return LSB_OK;
}

int ensure_work(lsb_kvs* s, uint64_t bytes) {
  if (bytes <= s->work_bytes) return LSB_OK;
  cudaFree(s->work);
  s->work = nullptr;
  s->work_bytes = 0;
  if (cudaMalloc(&s->work, bytes) != cudaSuccess) {
    cudaGetLastError();
    return LSB_ERR_OOM;
  }
  s->work_bytes = bytes;
  return LSB_OK;
}

}  // namespace

extern "C" {

int lsb_kvs_create(unsigned log2_buckets, uint64_t heap_bytes, const lsb_options* opt,
                   lsb_kvs** out) {
  if (!out || heap_bytes == 0 || heap_bytes > kMaxHeap) return LSB_ERR_ARG;
  *out = nullptr;
  lsb_kvs* s = new (std::nothrow) lsb_kvs();
  if (!s) return LSB_ERR_OOM;
  lsb_options o{};
  if (opt) {
    o = *opt;
  } else {
    o.device = -1;
  }
  int rc = lsb_map_create_ex(log2_buckets, &o, &s->map);
  if (rc == LSB_OK &&
      (cudaMalloc(&s->heap, (heap_bytes + 3) / 4 * 4) != cudaSuccess ||  // whole words
       cudaMalloc(&s->dead, sizeof(unsigned long long)) != cudaSuccess ||
       cudaMalloc(&s->parts, sizeof(uint64_t) * (kParts + kSums)) != cudaSuccess ||
       cudaHostAlloc((void**)&s->words, sizeof(HostWords), cudaHostAllocMapped) != cudaSuccess ||
       cudaHostGetDevicePointer((void**)&s->d_words, s->words, 0) != cudaSuccess ||
       cudaMemset(s->dead, 0, sizeof(unsigned long long)) != cudaSuccess)) {
    cudaGetLastError();
    rc = LSB_ERR_OOM;
  }
  if (rc != LSB_OK) {
    lsb_kvs_destroy(s);
    return rc;
  }
  s->heap_cap = heap_bytes;
  *out = s;
  return LSB_OK;
}

int lsb_kvs_destroy(lsb_kvs* s) {
  if (!s) return LSB_ERR_ARG;
  if (s->map) lsb_map_destroy(s->map);
  cudaFree(s->heap);
  cudaFree(s->dead);
  cudaFreeHost(s->words);
  cudaFree(s->parts);
  cudaFree(s->tmp);
  cudaFree(s->res);
  cudaFree(s->work);
  delete s;
  return LSB_OK;
}

lsb_map* lsb_kvs_map(lsb_kvs* s) { return s ? s->map : nullptr; }

int lsb_kvs_put(lsb_kvs* s, const uint64_t* keys, const uint8_t* vals, const uint64_t* val_off,
                size_t n, cudaStream_t stream) {
  if (!s || (n && (!keys || !val_off))) return LSB_ERR_ARG;
  if (n == 0) return LSB_OK;
  if (n > 0xFFFFFFFFull) return LSB_ERR_ARG;
  int rc = ensure_tmp(s, n);
  if (rc) return rc;
  const uint64_t base = s->heap_used;
  uint64_t* handle = s->tmp;
  uint64_t* old = s->tmp + (n + 1);
  // handles first (they need only the batch's offsets and the heap cursor), so
  // that one wait returns everything the host has to check
  s->words->bad = 0;
  k_handles<<<(uint32_t)((n + 255) / 256), 256, 0, stream>>>(val_off, base, handle, (uint32_t)n,
                                                             s->d_words);
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(stream) != cudaSuccess)
    return LSB_ERR_CUDA;
  const uint64_t first = s->words->first, last = s->words->last;
  if (last < first) return LSB_ERR_ARG;
  const uint64_t bytes = last - first;
  if (bytes && !vals) return LSB_ERR_ARG;
  if (bytes > s->heap_cap - s->heap_used) return LSB_ERR_OOM;  // no effect
  if (s->words->bad) return LSB_ERR_ARG;  // a value longer than 2^24 - 1 bytes: nothing stored
  if (bytes && cudaMemcpyAsync(s->heap + base, vals + first, bytes, cudaMemcpyDeviceToDevice,
                               stream) != cudaSuccess)
    return LSB_ERR_CUDA;
  rc = lsb_map_put(s->map, keys, handle, old, n, stream);
  if (rc) return rc;
  k_dead_bytes<<<(uint32_t)((n + 255) / 256), 256, 0, stream>>>(nullptr, old, (uint32_t)n,
                                                                s->dead);
  s->heap_used += bytes;
  return cudaGetLastError() == cudaSuccess ? LSB_OK : LSB_ERR_CUDA;
}

int lsb_kvs_get(lsb_kvs* s, const uint64_t* keys, uint8_t* found_out, uint32_t* len_out,
                uint64_t* dst_off_out, uint8_t* dst, uint64_t dst_cap, size_t n,
                uint64_t* total_out, cudaStream_t stream) {
  if (!s || (n && (!keys || !len_out || !dst_off_out))) return LSB_ERR_ARG;
  if (n == 0) {
    if (total_out) *total_out = 0;
    return LSB_OK;
  }
  if (n > 0xFFFFFFFFull) return LSB_ERR_ARG;
  int rc = ensure_tmp(s, n);
  if (rc) return rc;
  rc = lsb_map_get(s->map, keys, s->res, n, stream);
  if (rc) return rc;
  const uint32_t part = part_size(n), nparts = part_count(n);
  k_length_sums<<<nparts, kPartThreads, 0, stream>>>(s->res, (uint32_t)n, part, s->parts);
  k_length_offsets<<<nparts, kPartThreads, 0, stream>>>(s->res, (uint32_t)n, part, s->parts, len_out,
                                                        dst_off_out, found_out, s->d_words);
  if (dst && dst_cap) {
    const uint64_t threads = (uint64_t)kCopyLanes * n;
    k_gather<<<(uint32_t)((threads + 255) / 256), 256, 0, stream>>>(s->res, dst_off_out, s->heap,
                                                                   dst, dst_cap, (uint32_t)n);
  }
  if (total_out) {
    if (cudaStreamSynchronize(stream) != cudaSuccess) return LSB_ERR_CUDA;
    *total_out = s->words->total;
  }
  return cudaGetLastError() == cudaSuccess ? LSB_OK : LSB_ERR_CUDA;
}

int lsb_kvs_remove(lsb_kvs* s, const uint64_t* keys, uint8_t* found_out, size_t n,
                   cudaStream_t stream) {
  if (!s || (n && !keys)) return LSB_ERR_ARG;
  if (n == 0) return LSB_OK;
  if (n > 0xFFFFFFFFull) return LSB_ERR_ARG;
  int rc = ensure_tmp(s, n);
  if (rc) return rc;
  rc = lsb_map_remove(s->map, keys, s->res, n, stream);
  if (rc) return rc;
  k_dead_bytes<<<(uint32_t)((n + 255) / 256), 256, 0, stream>>>(s->res, nullptr, (uint32_t)n,
                                                                s->dead);
  if (found_out) {
    // found bytes are the first byte of each 16-byte result
    if (cudaMemcpy2DAsync(found_out, 1, s->res, sizeof(lsb_result), 1, n,
                          cudaMemcpyDeviceToDevice, stream) != cudaSuccess)
      return LSB_ERR_CUDA;
  }
  return cudaGetLastError() == cudaSuccess ? LSB_OK : LSB_ERR_CUDA;
}

int lsb_kvs_usage(lsb_kvs* s, uint64_t* heap_used, uint64_t* heap_dead, uint64_t* heap_cap,
                  cudaStream_t stream) {
  if (!s) return LSB_ERR_ARG;
  unsigned long long dead = 0;
  if (cudaMemcpyAsync(&dead, s->dead, 8, cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
      cudaStreamSynchronize(stream) != cudaSuccess)
    return LSB_ERR_CUDA;
  if (heap_used) *heap_used = s->heap_used;
  if (heap_dead) *heap_dead = dead;
  if (heap_cap) *heap_cap = s->heap_cap;
  return LSB_OK;
}

// Heap compaction: the live values move, in key order, to the front of the
// heap (through a staging copy), their slots take the new handles, and the
// garbage count restarts at zero.  All of it on the device; the host waits
// once for the number of live entries and their bytes, which size the scratch,
// and once at the end.
int lsb_kvs_compact(lsb_kvs* s, cudaStream_t stream) {
  if (!s) return LSB_ERR_ARG;
  lsb::TableView view;
  uint32_t buckets = 0;
  lsb_internal_map_view(s->map, &view, &buckets);
  unsigned long long* sums = reinterpret_cast<unsigned long long*>(s->parts + kParts);
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount,
                             lsb_internal_map_device(s->map)) != cudaSuccess)
    return LSB_ERR_CUDA;
  const uint32_t scan_blocks =
      (uint32_t)std::min<uint64_t>(((uint64_t)buckets + 7) / 8, (uint64_t)sms * 8);
  if (cudaMemsetAsync(sums, 0, kSums * sizeof(*sums), stream) != cudaSuccess) return LSB_ERR_CUDA;
  k_live<<<scan_blocks, 256, 0, stream>>>(view, buckets, nullptr, nullptr, 0, sums, s->d_words);
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(stream) != cudaSuccess)
    return LSB_ERR_CUDA;
  const uint64_t n = s->words->count, live = s->words->total;
  // The map may hold more entries than the store put (lsb_kvs_map): a handle
  // under a second key is a value of its own from here on.  Refused: handles
  // that reach past the heap, and more bytes than it takes.
  if (s->words->end > s->heap_cap || live > s->heap_cap) return LSB_ERR_STATE;
  int rc = LSB_OK;
  if (n) {
    const uint32_t part = sort_part(n), blocks = (uint32_t)((n + part - 1) / part);
    const uint64_t stage_bytes = (live + 15) / 16 * 16;
    rc = ensure_work(s, stage_bytes + 4 * 8 * n + sizeof(uint32_t) * kDigits * blocks);
    if (rc) return rc;
    uint64_t* keys[2] = {reinterpret_cast<uint64_t*>(s->work + stage_bytes), nullptr};
    keys[1] = keys[0] + n;
    uint64_t** slots[2] = {reinterpret_cast<uint64_t**>(keys[1] + n), nullptr};
    slots[1] = slots[0] + n;
    uint32_t* counts = reinterpret_cast<uint32_t*>(slots[1] + n);
    k_live<<<scan_blocks, 256, 0, stream>>>(view, buckets, keys[0], slots[0], n, sums, s->d_words);
    for (uint32_t pass = 0; pass < 8; ++pass) {
      const int a = pass & 1, b = a ^ 1;
      k_digit_counts<<<blocks, kDigits, 0, stream>>>(keys[a], n, part, 8 * pass, counts);
      k_digit_place<<<blocks, kDigits, 0, stream>>>(keys[a], slots[a], n, part, 8 * pass, counts,
                                                   keys[b], slots[b]);
    }
    const uint32_t mpart = part_size(n), mparts = part_count(n);
    k_slot_sums<<<mparts, kPartThreads, 0, stream>>>(slots[0], n, mpart, s->parts);
    k_new_handles<<<mparts, kPartThreads, 0, stream>>>(slots[0], n, mpart, s->parts, keys[1]);
    k_move<<<(uint32_t)((kCopyLanes * n + 255) / 256), 256, 0, stream>>>(slots[0], keys[1], n,
                                                                       s->heap, s->work, live);
    if (cudaGetLastError() != cudaSuccess) rc = LSB_ERR_CUDA;
    if (rc == LSB_OK && live &&
        cudaMemcpyAsync(s->heap, s->work, live, cudaMemcpyDeviceToDevice, stream) != cudaSuccess)
      rc = LSB_ERR_CUDA;
  }
  if (rc == LSB_OK && cudaMemsetAsync(s->dead, 0, 8, stream) != cudaSuccess) rc = LSB_ERR_CUDA;
  if (rc == LSB_OK && cudaStreamSynchronize(stream) != cudaSuccess) rc = LSB_ERR_CUDA;
  if (s->work_bytes > kWorkKept) {
    cudaStreamSynchronize(stream);
    cudaFree(s->work);
    s->work = nullptr;
    s->work_bytes = 0;
  }
  if (rc == LSB_OK) s->heap_used = live;
  return rc;
}

}  // extern "C"
