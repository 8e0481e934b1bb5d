// Forward phase 2: binning — the list of (tile, Gaussian) instances in the order the
// compositing reads them: by tile, within a tile by depth, equal depths by Gaussian id.
//
// Upstream emits K 64-bit keys (tile << 32 | depth bits) in Gaussian order and runs
// one global stable radix sort over 32 + log2(tiles) bits. Here the depth part is
// sorted once per Gaussian instead of once per instance:
//   1. depth sort: stable LSD radix sort of the N depth keys (4 passes of 8 bits), so
//      the Gaussians come out by (depth, id), and the prefix of their tile counts in that
//      order: an instance's index is its position in the list of all Gaussians' tiles
//      (row-major in the tile rectangle) in depth order;
//   2. tile keys: that list's tile indices, written in order (the list's other columns
//      are not: its Gaussian is found again from the prefix, its index is its position);
//   3. tile sort: stable LSD radix sort of the instances by tile index alone
//      (ceil(log2 tiles) bits, at most 8 per pass: 2 passes at 1080p). The first pass's
//      scatter reads the keys and finds the Gaussians.
// A stable sort by tile of a list ordered by (depth, id) is ordered by (tile, depth,
// id): exactly the stable sort of upstream's keys over instances emitted by id. The
// last tile pass also counts the instances of every tile (runs of equal tiles), and a
// scan turns the counts into tile ranges.
//
// Every radix pass is three launches over chunks of elements (two where the chunks are
// few): count (digit histogram per chunk), scan (per digit, over chunks: the chunk's first
// global slot), scatter (rank inside the chunk, exchange through shared memory by digit,
// then write each digit's run to its global slots). Ranking inside a chunk is stable: a warp
// owns a contiguous slice and walks it 64 elements per round; lanes with equal digits meet
// in a mask in shared memory.
//
// The scatters are bound by shared memory (84 to 87 % of its wavefronts), the rest by latency
// per block, so a thread holds its keys in registers, all loads in flight at once, an element
// goes through shared memory once, as one 8-byte value beside or with its key, and the first
// tile pass carries positions only. 1,000,000 Gaussians, 12.4 million instances, 8160 tiles:
// the depth order 114 us, tile keys 48, tile sort 172, ranges 5; with the list written out
// first, chunks staged through shared memory and a ballot per digit bit, 130, 84, 250 and 10.


#include "cfgs_internal.cuh"
#include "kernels.cuh"

namespace cfgs {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;

// Elements per thread of a radix chunk: 8 for long lists, whose digit runs get longer (12.4
// million instances, two passes: keys 41, counts 14, scatters 72 and 72 us; with 4 elements
// 42, 20, 83 and 86), 4 where the wide chunks would fill the GPU only a few times (1,000,000
// depths: scatters 12.4 us each, with 8 elements 13.3): from 16 of those blocks per SM.
constexpr int64_t kWideListMin = 16 * 152 * 4 * kSortThreads;
inline int radix_items(int64_t n) { return n >= kWideListMin ? 8 : 4; }

// Few chunks are added up by every scatter block itself, from counts stored chunk by chunk;
// more by the scan kernel, from counts stored digit by digit. (Forward of 16,384 Gaussians at
// 256x256, chunks 16 and below 128: 154 -> 141 us, with the line at 64 chunks 145. At 225
// chunks the sums cost what the launch did: 12.64 against 12.58 ms for 25 pose iterations.)
constexpr int64_t kFoldMaxChunks = 128;
constexpr int kFoldUnroll = 6;  // loads in flight per thread
inline bool fold_counts(int64_t num_chunks) { return num_chunks <= kFoldMaxChunks; }

// What a radix pass carries beside the key.
enum Payload {
  kValue,      // one value: val_in, or the element's own index when that is NULL
  kFirstPair,  // Gaussian and position of an instance, found from the list (InstanceList)
  kPair,       // the same, from pair_in
};

// One radix pass over elements [0, n).
struct SortPass {
  const uint32_t* depth_touched;  // first depth pass: the count forms the keys from these (key_form)
  const float4* depth_rgbd;
  uint32_t* key_form;
  const uint32_t* key_in;
  const uint32_t* val_in;
  const uint2* pair_in;
  uint32_t* key_out;           // NULL: keys are not written (last pass)
  uint32_t* val_out;
  uint32_t* aux_out;           // last tile pass: the pairs' positions (val_out: the Gaussians)
  uint2* pair_out;             // tile passes before the last
  uint32_t* tile_count;        // last tile pass: instances per tile
  int shift, bits;
  int items;                   // elements per thread (radix_items): chunks of kSortThreads * items
  int64_t n;                   // element count, when counts is NULL
  const CfgsCounts* counts;    // element count = num_rendered (nothing to do above cap)
  int64_t cap;
  int64_t num_chunks;          // chunks covered by the grid
  bool fold;                   // no scan launch: the scatter adds up the counts (fold_counts)
  uint32_t* chunk_counts;      // [1 << bits][num_chunks]; with fold [num_chunks][kSortDigits]
  uint32_t* digit_totals;      // [1 << bits], written by the scan
};

// Shared memory of a block of any stage.
constexpr int kScanItems = 8;
template <int ITEMS>
struct CountShared {
  uint32_t whist[kSortWarps][kSortDigits];  // per-warp digit counters, then first positions
  uint32_t mark[kSortWarps * ITEMS];        // bit i set where a Gaussian's instances begin
  uint32_t mark_before[kSortWarps * ITEMS]; // marks in earlier words
  uint32_t scan[kScanItems * 32 + 4];
};
template <int ITEMS>
struct BinShared : CountShared<ITEMS> {
  union {
    uint32_t same[2][kSortWarps][kSortDigits];  // ranking: the lanes that hold a digit, for two elements per lane
    uint2 buf[kSortThreads * ITEMS];            // a chunk in digit order
  };
  uint32_t keys[kSortThreads * ITEMS];      // its keys, where buf holds pairs
  uint32_t slot[kSortDigits];               // global slot minus position of a digit's first element
};

__device__ __forceinline__ uint32_t pass_elements(const SortPass& p) {
  if (!p.counts) return (uint32_t)p.n;
  const int64_t k = (int64_t)p.counts->num_rendered;
  return k > p.cap ? 0u : (uint32_t)k;
}

// Block-wide inclusive scan of one value per thread (blockDim.x <= 1024); returns the
// inclusive prefix and writes the block total to *total.
__device__ __forceinline__ uint32_t block_inclusive_scan(uint32_t v, uint32_t* sh, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < nw ? sh[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    sh[32 + lane] = w;
  }
  __syncthreads();
  const uint32_t r = x + (warp > 0 ? sh[32 + warp - 1] : 0u);
  *total = sh[32 + nw - 1];
  __syncthreads();
  return r;
}

// Exclusive scan of load(0 .. n) by one block into store(i, prefix); returns the total.
// IT values per thread and round, so that a few thousand take one round; blockDim.x is a
// multiple of 128. sh holds IT * 32 + 1 values.
template <int IT, class Load, class Store>
__device__ __forceinline__ uint32_t block_exclusive_scan(int64_t n, uint32_t* sh, Load load, Store store) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  uint32_t carry = 0;
  for (int64_t base = 0; base < n; base += IT * (int64_t)blockDim.x) {
    uint32_t v[IT], x[IT];
#pragma unroll
    for (int k = 0; k < IT; ++k) {
      const int64_t i = base + k * (int64_t)blockDim.x + threadIdx.x;
      v[k] = i < n ? load(i) : 0u;
    }
#pragma unroll
    for (int k = 0; k < IT; ++k) {
      x[k] = v[k];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x[k], o);
        if (lane >= o) x[k] += y;
      }
      if (lane == 31) sh[k * nw + warp] = x[k];
    }
    __syncthreads();
    if (warp == 0) {  // the IT * nw warp totals, a multiple of 32: consecutive ones per lane
      const int per = IT * nw / 32;
      uint32_t sum = 0;
      for (int k = 0; k < per; ++k) sum += sh[lane * per + k];
      uint32_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      uint32_t before = incl - sum;
      for (int k = 0; k < per; ++k) {
        const uint32_t t = sh[lane * per + k];
        sh[lane * per + k] = before;
        before += t;
      }
      if (lane == 31) sh[IT * nw] = incl;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IT; ++k) {
      const int64_t i = base + k * (int64_t)blockDim.x + threadIdx.x;
      if (i < n) store(i, carry + sh[k * nw + warp] + x[k] - v[k]);
    }
    carry += sh[IT * nw];
    __syncthreads();
  }
  return carry;
}

// Adds up a block's per-warp digit counters and writes them to chunk_counts[d][chunk].
template <int ITEMS>
__device__ __forceinline__ void write_chunk_counts(const SortPass& p, CountShared<ITEMS>& sh, uint32_t bid) {
  __syncthreads();
  for (int d = threadIdx.x; d < (1 << p.bits); d += kSortThreads) {
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) s += sh.whist[w][d];
    p.chunk_counts[p.fold ? (size_t)bid * kSortDigits + d : (size_t)d * p.num_chunks + bid] = s;
  }
}

// Clears n tables of per-warp digit counters.
__device__ __forceinline__ void clear_digits(uint32_t* tables, int n) {
  uint4* w = reinterpret_cast<uint4*>(tables);
#pragma unroll
  for (int i = 0; i < n * (kSortWarps * kSortDigits / 4 / kSortThreads); ++i)
    w[i * kSortThreads + threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
}

// Digit histogram of one chunk. FORM: the first depth pass, whose keys (depth bits; Gaussians
// that touch no tile sort last) are written here as well.
template <int ITEMS, bool FORM>
__device__ __forceinline__ void sort_count_block(const SortPass& p, CountShared<ITEMS>& sh, uint32_t bid) {
  constexpr uint32_t kChunk = kSortThreads * ITEMS;
  const uint32_t n = pass_elements(p);
  const uint32_t c0 = bid * kChunk;
  if (c0 >= n) return;
  const uint32_t mask = (1u << p.bits) - 1u;
  const int warp = threadIdx.x >> 5;
  clear_digits(&sh.whist[0][0], 1);
  uint4 k[ITEMS / 4];
#pragma unroll
  for (int q = 0; q < ITEMS / 4; ++q) {
    const uint32_t i = c0 + 4u * (q * kSortThreads + threadIdx.x);
    if (FORM) {
      uint32_t e[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
        e[c] = i + c < n && p.depth_touched[i + c] ? __float_as_uint(p.depth_rgbd[i + c].w) : 0xffffffffu;
      k[q] = make_uint4(e[0], e[1], e[2], e[3]);
      if (i < n) *reinterpret_cast<uint4*>(p.key_form + i) = k[q];  // the buffer's stride is a multiple of 4
    } else if (i + 3 < n) {
      k[q] = *reinterpret_cast<const uint4*>(p.key_in + i);
    } else {
      k[q].x = i < n ? p.key_in[i] : 0u;
      k[q].y = i + 1 < n ? p.key_in[i + 1] : 0u;
      k[q].z = i + 2 < n ? p.key_in[i + 2] : 0u;
      k[q].w = 0u;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < ITEMS / 4; ++q) {
    const uint32_t i = c0 + 4u * (q * kSortThreads + threadIdx.x);
    if (i < n) atomicAdd(&sh.whist[warp][(k[q].x >> p.shift) & mask], 1u);
    if (i + 1 < n) atomicAdd(&sh.whist[warp][(k[q].y >> p.shift) & mask], 1u);
    if (i + 2 < n) atomicAdd(&sh.whist[warp][(k[q].z >> p.shift) & mask], 1u);
    if (i + 3 < n) atomicAdd(&sh.whist[warp][(k[q].w >> p.shift) & mask], 1u);
  }
  write_chunk_counts(p, sh, bid);
}
template <int ITEMS, bool FORM>
__global__ void __launch_bounds__(kSortThreads) k_sort_count(SortPass p) {
  __shared__ __align__(16) CountShared<ITEMS> sh;
  sort_count_block<ITEMS, FORM>(p, sh, blockIdx.x);
}

// One block per digit d: chunk_counts[d][c] becomes the number of digit-d elements in
// earlier chunks, and digit_totals[d] the digit's count. The scatter adds the counts of
// the smaller digits.
__device__ __forceinline__ void sort_scan_block(const SortPass& p, uint32_t* sh, int d) {
  const uint32_t n = pass_elements(p);
  const int64_t chunk = (int64_t)kSortThreads * p.items, nc = ((int64_t)n + chunk - 1) / chunk;
  uint32_t* col = p.chunk_counts + (size_t)d * p.num_chunks;
  const uint32_t total = block_exclusive_scan<kScanItems>(
      nc, sh, [&](int64_t c) { return col[c]; }, [&](int64_t c, uint32_t v) { col[c] = v; });
  if (threadIdx.x == 0) p.digit_totals[d] = total;
}
__global__ void __launch_bounds__(1024) k_sort_scan(SortPass p) {
  __shared__ uint32_t sh[kScanItems * 32 + 1];
  sort_scan_block(p, sh, blockIdx.x);
}

// ---- the instance list -------------------------------------------------------------------
// A chunk [c0, c0 + cnt) of the list of instances in depth order: starts[bid] is the depth
// rank whose instances cover position c0, starts[bid + 1] the one that covers the next
// chunk's first position (or the last instance). A mark at every position where a
// Gaussian's instances begin gives an instance's rank as starts[bid] plus the marks up to
// it: one shared word, one population count.
template <int ITEMS>
__device__ __forceinline__ void mark_chunk(const InstanceList& a, CountShared<ITEMS>& sh, uint32_t bid, uint32_t c0,
                                           uint32_t cnt) {
  constexpr int kWords = kSortWarps * ITEMS;
  if (threadIdx.x < kWords) sh.mark[threadIdx.x] = 0u;
  __syncthreads();
  const uint32_t r0 = a.starts[bid], r1 = a.starts[bid + 1];
  for (uint32_t r = r0 + 1 + threadIdx.x; r <= r1; r += kSortThreads) {
    const uint32_t at = a.prefix[r] - c0;
    if (at < cnt) atomicOr(&sh.mark[at >> 5], 1u << (at & 31));
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    constexpr int kPer = kWords / 32;
    uint32_t own[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      own[k] = (uint32_t)__popc(sh.mark[threadIdx.x * kPer + k]);
      sum += own[k];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)threadIdx.x >= o) incl += y;
    }
    uint32_t before = incl - sum;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      sh.mark_before[threadIdx.x * kPer + k] = before;
      before += own[k];
    }
  }
  __syncthreads();
}

// Depth rank of the instance at chunk position i.
template <int ITEMS>
__device__ __forceinline__ uint32_t instance_rank(const CountShared<ITEMS>& sh, uint32_t r0, uint32_t i) {
  const uint32_t w = i >> 5;
  return r0 + sh.mark_before[w] + (uint32_t)__popc(sh.mark[w] & (0xffffffffu >> (31 - (i & 31))));
}

// Tile of instance j of a rectangle: row j / w, column j % w of the rectangle's w columns.
// The quotient is estimated with a reciprocal of 1 ulp (off by at most one for j < 2^22) and
// corrected exactly.
__device__ __forceinline__ uint32_t instance_tile(uint2 rc, uint32_t j, uint32_t tile_base, uint32_t grid_x) {
  const uint32_t x0 = rc.x & 0xffffu, y0 = rc.x >> 16, w = (rc.y & 0xffffu) - x0;
  uint32_t ty, tx;
  if (j < (1u << 22)) {
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"((float)w));
    ty = (uint32_t)((float)j * inv);
    tx = j - ty * w;
    if ((int32_t)tx < 0) {
      --ty;
      tx += w;
    } else if (tx >= w) {
      ++ty;
      tx -= w;
    }
  } else {
    ty = j / w;
    tx = j - ty * w;
  }
  return tile_base + (y0 + ty) * grid_x + x0 + tx;
}

// One chunk's tile keys, and its digit histogram for the first tile pass p.
template <class Scenes, int ITEMS>
__device__ __forceinline__ void emit_keys_block(const EmitArgs<Scenes>& a, const SortPass& p, CountShared<ITEMS>& sh,
                                                uint32_t bid) {
  constexpr uint32_t kChunk = kSortThreads * ITEMS;
  const uint32_t n = pass_elements(p);
  const uint32_t c0 = bid * kChunk;
  if (c0 >= n) return;
  const uint32_t cnt = min(kChunk, n - c0);
  const uint32_t mask = (1u << p.bits) - 1u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  clear_digits(&sh.whist[0][0], 1);
  mark_chunk(a.list, sh, bid, c0, cnt);
  const uint32_t r0 = a.list.starts[bid];
  uint32_t g[ITEMS], j[ITEMS];
  uint2 rc[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const uint32_t i = (uint32_t)(warp * 32 * ITEMS + k * 32 + lane);
    if (i < cnt) {
      const uint32_t r = instance_rank(sh, r0, i);
      g[k] = a.list.order[r];
      j[k] = c0 + i - a.list.prefix[r];
    }
  }
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const uint32_t i = (uint32_t)(warp * 32 * ITEMS + k * 32 + lane);
    if (i < cnt) rc[k] = a.geom.rect[g[k]];
  }
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const uint32_t i = (uint32_t)(warp * 32 * ITEMS + k * 32 + lane);
    if (i < cnt) {
      const SceneDesc& sd = a.scenes.for_gaussian(g[k]);
      const uint32_t key = instance_tile(rc[k], j[k], (uint32_t)sd.tile_base, (uint32_t)sd.grid_x);
      a.keys[c0 + i] = key;
      atomicAdd(&sh.whist[warp][(key >> p.shift) & mask], 1u);
    }
  }
  write_chunk_counts(p, sh, bid);
}
template <class Scenes, int ITEMS>
__global__ void __launch_bounds__(kSortThreads) k_emit_keys(EmitArgs<Scenes> a, SortPass p) {
  __shared__ __align__(16) CountShared<ITEMS> sh;
  emit_keys_block<Scenes, ITEMS>(a, p, sh, blockIdx.x);
}

// ---- scatter -----------------------------------------------------------------------------
template <int ITEMS, Payload P, bool FULL>
__device__ __forceinline__ void scatter_chunk(const SortPass& p, const InstanceList& a, BinShared<ITEMS>& sh,
                                              uint32_t bid, int cnt) {
  constexpr uint32_t kChunk = kSortThreads * ITEMS;
  static_assert(ITEMS % 2 == 0, "elements are ranked two at a time");
  const uint32_t c0 = bid * kChunk;
  const int ndig = 1 << p.bits;
  const uint32_t mask = (uint32_t)ndig - 1u;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int i0 = warp * 32 * ITEMS + lane;  // this thread's elements: i0 + 32 k

  uint32_t key[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) key[k] = FULL || i0 + 32 * k < cnt ? p.key_in[c0 + i0 + 32 * k] : 0u;
  // digit t: elements in all chunks and in earlier chunks; folded, digits 4 (t % 64) ... + 3
  // over every fourth chunk first
  uint32_t dtot = 0, earlier = 0;
  uint4 tot4 = make_uint4(0u, 0u, 0u, 0u), earlier4 = tot4;
  const bool fold = ITEMS == 4 && p.fold;
  if (fold) {
    const uint32_t nc = (pass_elements(p) + kChunk - 1) / kChunk;
    const uint4* counts = reinterpret_cast<const uint4*>(p.chunk_counts) + (t & 63);
    if (4 * (t & 63) < ndig) {
      for (uint32_t c = t >> 6; c < nc; c += 4 * kFoldUnroll) {
        uint4 v[kFoldUnroll];
#pragma unroll
        for (int k = 0; k < kFoldUnroll; ++k)
          v[k] = c + 4 * k < nc ? counts[(c + 4 * k) * (kSortDigits / 4)] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int k = 0; k < kFoldUnroll; ++k) {
          const uint32_t use = c + 4 * k < bid ? 0xffffffffu : 0u;
          tot4.x += v[k].x;
          tot4.y += v[k].y;
          tot4.z += v[k].z;
          tot4.w += v[k].w;
          earlier4.x += v[k].x & use;
          earlier4.y += v[k].y & use;
          earlier4.z += v[k].z & use;
          earlier4.w += v[k].w & use;
        }
      }
    }
  } else if (t < ndig) {
    dtot = p.digit_totals[t];
    earlier = p.chunk_counts[(size_t)t * p.num_chunks + bid];
  }
  clear_digits(&sh.whist[0][0], 1);
  clear_digits(&sh.same[0][0][0], 2);
  if (P == kFirstPair) mark_chunk(a, sh, bid, c0, (uint32_t)cnt);
  __syncthreads();

  // Rank of every element among the equal digits of its warp's slice, two elements per lane
  // at a time: the lanes of a digit meet in a mask in shared memory. (First tile pass of the
  // size above, before the pairs: 85 us and 53 million instructions; with a ballot per digit
  // bit 116 and 90 million, with match.any 139 us.)
  uint32_t pos[ITEMS];
  const unsigned lt = (1u << lane) - 1u;
  uint32_t* hist = sh.whist[warp];
  uint32_t* m0 = sh.same[0][warp];
  uint32_t* m1 = sh.same[1][warp];
#pragma unroll
  for (int k = 0; k < ITEMS; k += 2) {
    const bool act0 = FULL || i0 + 32 * k < cnt, act1 = FULL || i0 + 32 * (k + 1) < cnt;
    const uint32_t d0 = (key[k] >> p.shift) & mask, d1 = (key[k + 1] >> p.shift) & mask;
    if (act0) atomicOr(&m0[d0], 1u << lane);
    if (act1) atomicOr(&m1[d1], 1u << lane);
    __syncwarp();
    const uint32_t peers0 = m0[d0], peers1 = m1[d1];
    const uint32_t before0 = hist[d0];
    const uint32_t before1 = hist[d1] + (uint32_t)__popc(m0[d1]);
    pos[k] = before0 + (uint32_t)__popc(peers0 & lt);
    pos[k + 1] = before1 + (uint32_t)__popc(peers1 & lt);
    __syncwarp();
    if (act0 && (peers0 & lt) == 0) {
      hist[d0] = before0 + (uint32_t)__popc(peers0);
      m0[d0] = 0u;
    }
    __syncwarp();
    if (act1 && (peers1 & lt) == 0) {
      hist[d1] = before1 + (uint32_t)__popc(peers1);
      m1[d1] = 0u;
    }
    __syncwarp();
  }
  __syncthreads();
  if (fold) {
    uint4* parts = reinterpret_cast<uint4*>(&sh.same[0][0][0]);  // [2][4][kSortDigits]
    parts[t] = tot4;
    parts[kSortThreads + t] = earlier4;
    __syncthreads();
    const uint32_t* part = &sh.same[0][0][0];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      dtot += part[g * kSortDigits + t];
      earlier += part[(4 + g) * kSortDigits + t];
    }
  }

  // digit t: the warps' first positions, the digit's global slot
  uint32_t dsum = 0, first[kSortWarps];
  if (t < ndig) {
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      first[w] = dsum;
      dsum += sh.whist[w][t];
    }
  }
  uint32_t start = dsum, below = dtot;  // elements of smaller digits, in the chunk and in all
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, start, o), y = __shfl_up_sync(0xffffffffu, below, o);
    if (lane >= o) {
      start += x;
      below += y;
    }
  }
  if (lane == 31) {
    sh.scan[warp] = start;
    sh.scan[32 + warp] = below;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kSortWarps - 1; ++w)
    if (w < warp) {
      start += sh.scan[w];
      below += sh.scan[32 + w];
    }
  start -= dsum;
  below -= dtot;
  if (t < ndig) {
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) sh.whist[w][t] = start + first[w];
    sh.slot[t] = below + earlier - start;
  }
  __syncthreads();

  // into digit order
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int i = i0 + 32 * k;
    if (FULL || i < cnt) {
      const uint32_t q = pos[k] + hist[(key[k] >> p.shift) & mask];
      if (P == kPair) {
        sh.keys[q] = key[k];
        sh.buf[q] = p.pair_in[c0 + i];
      } else {
        sh.buf[q] = make_uint2(key[k], P == kFirstPair ? (uint32_t)i : p.val_in ? p.val_in[c0 + i] : c0 + i);
      }
    }
  }
  __syncthreads();
  const uint32_t r0 = P == kFirstPair ? a.starts[bid] : 0u;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int q = t + kSortThreads * k;
    if (FULL || q < cnt) {
      uint2 e = sh.buf[q];
      const uint32_t kk = P == kPair ? sh.keys[q] : e.x;
      const uint32_t out = sh.slot[(kk >> p.shift) & mask] + (uint32_t)q;
      if (P == kFirstPair) e = make_uint2(a.order[instance_rank(sh, r0, e.y)], c0 + e.y);
      if (p.key_out) p.key_out[out] = kk;
      if (P == kValue) {
        p.val_out[out] = e.y;
      } else if (p.pair_out) {
        p.pair_out[out] = e;
      } else {
        p.val_out[out] = e.x;
        p.aux_out[out] = e.y;
        // The chunk is fully sorted now (its input was sorted by the lower digits), so
        // equal tiles form runs: a run [b, e) adds e - b.
        const uint32_t before = q == 0 ? kk : P == kPair ? sh.keys[q - 1] : sh.buf[q - 1].x;
        if (before != kk) {
          atomicSub(&p.tile_count[kk], (uint32_t)q);
          atomicAdd(&p.tile_count[before], (uint32_t)q);
        }
        if (q == cnt - 1) atomicAdd(&p.tile_count[kk], (uint32_t)cnt);
      }
    }
  }
}

template <int ITEMS, Payload P>
__device__ __forceinline__ void sort_scatter_block(const SortPass& p, const InstanceList& a, BinShared<ITEMS>& sh,
                                                   uint32_t bid) {
  constexpr uint32_t kChunk = kSortThreads * ITEMS;
  const uint32_t n = pass_elements(p);
  const uint32_t c0 = bid * kChunk;
  if (c0 >= n) return;
  if (n - c0 >= kChunk) scatter_chunk<ITEMS, P, true>(p, a, sh, bid, (int)kChunk);
  else scatter_chunk<ITEMS, P, false>(p, a, sh, bid, (int)(n - c0));
}
// Resident blocks: pairs read from memory want the registers of 4 (72 us; with 5: 77), the
// others 5 (first tile pass 72 us; with 4: 74).
template <int ITEMS, Payload P>
__global__ void __launch_bounds__(kSortThreads, P == kPair ? 4 : 5) k_sort_scatter(SortPass p, InstanceList a) {
  __shared__ __align__(16) BinShared<ITEMS> sh;
  sort_scatter_block<ITEMS, P>(p, a, sh, blockIdx.x);
}

// ---- the depth order's prefix ------------------------------------------------------------
constexpr int kRankItems = 4;  // depth ranks per thread
constexpr int kRankBlock = kPreprocessBlock * kRankItems;

// Instances of every kRankBlock depth-ordered Gaussians; the instances of each go to the
// first depth-key buffer (free by now).
__device__ __forceinline__ void rank_sums_block(const GeomView& gv, int64_t slots, uint32_t* sh, int bid) {
  const int64_t r = (int64_t)bid * kRankBlock + kRankItems * threadIdx.x;
  uint4 n = make_uint4(0u, 0u, 0u, 0u);
  if (r < slots) {
    const uint4 g = *reinterpret_cast<const uint4*>(gv.depth_val[1] + r);
    n.x = gv.touched[g.x];
    if (r + 1 < slots) n.y = gv.touched[g.y];
    if (r + 2 < slots) n.z = gv.touched[g.z];
    if (r + 3 < slots) n.w = gv.touched[g.w];
    *reinterpret_cast<uint4*>(gv.depth_key[0] + r) = n;
  }
  uint32_t tot;
  block_inclusive_scan(n.x + n.y + n.z + n.w, sh, &tot);
  if (threadIdx.x == 0) gv.rank_sums[bid] = tot;
}
__global__ void __launch_bounds__(kPreprocessBlock) k_rank_sums(GeomView gv, int64_t slots) {
  __shared__ uint32_t sh[64];
  rank_sums_block(gv, slots, sh, blockIdx.x);
}

// The per-block instance counts become their exclusive prefix, in place (one block). Run for
// large batches only: below kRankScanMinBlocks blocks each block sums its predecessors
// itself (cheaper than a launch; quadratic in the block count above it).
constexpr int kRankScanMinBlocks = 2048;
inline bool rank_scan_needed(int rank_blocks) { return rank_blocks > kRankScanMinBlocks; }
__device__ __forceinline__ void rank_scan_block(uint32_t* rank_sums, int n, uint32_t* sh) {
  block_exclusive_scan<kScanItems>(
      n, sh, [&](int64_t c) { return rank_sums[c]; }, [&](int64_t c, uint32_t v) { rank_sums[c] = v; });
}
__global__ void __launch_bounds__(1024) k_rank_scan(uint32_t* rank_sums, int n) {
  __shared__ uint32_t sh[kScanItems * 32 + 1];
  rank_scan_block(rank_sums, n, sh);
}

// First instance index of every depth rank (the prefix, over its instance counts) and of
// every Gaussian (offset).
__device__ __forceinline__ void rank_place_block(const GeomView& gv, int64_t slots, bool scanned, uint32_t* sh, int bid) {
  uint32_t tot, block_first;
  if (scanned) {
    block_first = gv.rank_sums[bid];
  } else {
    uint32_t pre = 0;
    for (int b = threadIdx.x; b < bid; b += blockDim.x) pre += gv.rank_sums[b];
    block_inclusive_scan(pre, sh, &tot);
    block_first = tot;
  }
  const int64_t r = (int64_t)bid * kRankBlock + kRankItems * threadIdx.x;
  uint4 g = make_uint4(0u, 0u, 0u, 0u), n = g;
  if (r < slots) {
    g = *reinterpret_cast<const uint4*>(gv.depth_val[1] + r);
    n = *reinterpret_cast<const uint4*>(gv.depth_key[0] + r);
  }
  const uint32_t own = n.x + n.y + n.z + n.w;
  uint4 at;
  at.x = block_first + block_inclusive_scan(own, sh, &tot) - own;
  at.y = at.x + n.x;
  at.z = at.y + n.y;
  at.w = at.z + n.z;
  if (r < slots) *reinterpret_cast<uint4*>(gv.depth_key[0] + r) = at;
  if (n.x) gv.offset[g.x] = at.x;
  if (n.y) gv.offset[g.y] = at.y;
  if (n.z) gv.offset[g.z] = at.z;
  if (n.w) gv.offset[g.w] = at.w;
}
__global__ void __launch_bounds__(kPreprocessBlock) k_rank_place(GeomView gv, int64_t slots, bool scanned) {
  __shared__ uint32_t sh[64];
  rank_place_block(gv, slots, scanned, sh, blockIdx.x);
}

// starts[c] = the depth rank whose instances cover position c * chunk, starts[last + 1] the
// rank of the last instance. Raises the overflow flag when the instances exceed the
// capacity.
template <class Scenes>
__device__ __forceinline__ void emit_starts_block(const EmitArgs<Scenes>& a, uint32_t chunk, int bid) {
  const int64_t K = (int64_t)a.counts->num_rendered;
  if (K > a.cap) {
    if (bid == 0 && threadIdx.x == 0) atomicOr(&a.counts->flags, CFGS_FLAG_CAPACITY_OVERFLOW);
    return;
  }
  const int64_t r = (int64_t)bid * blockDim.x + threadIdx.x;
  if (r >= a.total_slots) return;
  const uint32_t b = a.list.prefix[r], e = r + 1 < a.total_slots ? a.list.prefix[r + 1] : (uint32_t)K;
  if (b == e) return;
  for (uint32_t c = (b + chunk - 1) / chunk; (int64_t)c * chunk < e; ++c) a.list.starts[c] = (uint32_t)r;
  if (e == (uint32_t)K) a.list.starts[(uint32_t)((K + chunk - 1) / chunk)] = (uint32_t)r;
}
template <class Scenes>
__global__ void __launch_bounds__(kPreprocessBlock) k_emit_starts(EmitArgs<Scenes> a, uint32_t chunk) {
  emit_starts_block<Scenes>(a, chunk, blockIdx.x);
}

// Tile ranges from the per-tile instance counts (one block).
template <int IT>
__device__ __forceinline__ void tile_ranges_block(const uint32_t* tile_count, uint32_t* tile_range, int num_tiles,
                                                  uint32_t* sh) {
  const uint32_t total = block_exclusive_scan<IT>(
      num_tiles, sh, [&](int64_t i) { return tile_count[i]; }, [&](int64_t i, uint32_t v) { tile_range[i] = v; });
  if (threadIdx.x == 0) tile_range[num_tiles] = total;
}
__global__ void __launch_bounds__(1024) k_tile_ranges(const uint32_t* tile_count, uint32_t* tile_range, int num_tiles) {
  __shared__ uint32_t sh[kScanItems * 32 + 1];
  tile_ranges_block<kScanItems>(tile_count, tile_range, num_tiles, sh);
}

namespace {

// The scan's block: a digit's chunks in one round where they are few.
void launch_scan(const SortPass& p, cudaStream_t st) {
  if (p.fold) return;
  k_sort_scan<<<1 << p.bits, p.num_chunks <= 256 * kScanItems ? 256 : 1024, 0, st>>>(p);
}

template <int ITEMS>
void launch_pass_items(const SortPass& p, cudaStream_t st) {
  const int grid = (int)p.num_chunks;
  if (p.key_form) k_sort_count<ITEMS, true><<<grid, kSortThreads, 0, st>>>(p);
  else k_sort_count<ITEMS, false><<<grid, kSortThreads, 0, st>>>(p);
  launch_scan(p, st);
  if (p.pair_in) k_sort_scatter<ITEMS, kPair><<<grid, kSortThreads, 0, st>>>(p, InstanceList{});
  else k_sort_scatter<ITEMS, kValue><<<grid, kSortThreads, 0, st>>>(p, InstanceList{});
}

void launch_pass(const SortPass& p, cudaStream_t st) {
  if (p.items == 8) launch_pass_items<8>(p, st);
  else launch_pass_items<4>(p, st);
}

// The first tile pass, keys included.
template <class Scenes, int ITEMS>
void launch_emit_items(const EmitArgs<Scenes>& a, const SortPass& p, cudaStream_t st) {
  const int grid = (int)p.num_chunks;
  k_emit_keys<Scenes, ITEMS><<<grid, kSortThreads, 0, st>>>(a, p);
  launch_scan(p, st);
  k_sort_scatter<ITEMS, kFirstPair><<<grid, kSortThreads, 0, st>>>(p, a.list);
}

}  // namespace

// Tile-key digits: the fewest passes of at most 8 bits that cover the tile index, split
// evenly.
void tile_sort_plan(int64_t num_tiles, int* passes, int* width) {
  int bits = 1;
  while (bits < 31 && ((int64_t)1 << bits) < num_tiles) ++bits;
  *passes = (bits + 7) / 8;
  *width = (bits + *passes - 1) / *passes;
}

namespace {

void set_chunks(SortPass& p, int64_t n) {
  p.items = radix_items(n);
  p.num_chunks = sort_chunks(n, kSortThreads * p.items);
  p.fold = p.items == 4 && fold_counts(p.num_chunks);
}

// Pass `pass` of the depth sort: the depths (keys formed in depth_key[1]) -> 0 -> 1 -> 0 ->
// depth_val[1].
SortPass depth_pass(const GeomView& gv, int64_t slots, int pass) {
  SortPass p{};
  const bool last = pass == kDepthPasses - 1;
  const int src = pass & 1 ? 0 : 1, dst = src ^ 1;
  if (pass == 0) {
    p.depth_touched = gv.touched;
    p.depth_rgbd = gv.rgbd;
    p.key_form = gv.depth_key[src];
  }
  p.key_in = gv.depth_key[src];
  p.val_in = pass == 0 ? nullptr : gv.depth_val[src];
  p.key_out = last ? nullptr : gv.depth_key[dst];
  p.val_out = gv.depth_val[dst];
  p.shift = 8 * pass;
  p.bits = 8;
  p.n = slots;
  p.cap = slots;
  set_chunks(p, slots);
  p.chunk_counts = gv.depth_counts;
  p.digit_totals = gv.depth_totals + kSortDigits * pass;
  return p;
}

// Pass `pass` of the tile sort: keys 0 (and the list itself) -> keys and pairs 1 -> 0 ... ->
// sorted.
template <class Scenes>
SortPass tile_pass(const BinArgs<Scenes>& a, int pass, int passes, int width) {
  const BinningView& bv = a.bin;
  SortPass p{};
  const bool last = pass == passes - 1;
  const int src = pass & 1, dst = src ^ 1;
  p.key_in = bv.key[src];
  p.pair_in = pass == 0 ? nullptr : bv.pair[src];
  if (last) {
    p.val_out = bv.sorted_gid;
    p.aux_out = bv.sorted_pidx;
    p.tile_count = a.tile_count;
  } else {
    p.key_out = bv.key[dst];
    p.pair_out = bv.pair[dst];
  }
  p.shift = width * pass;
  p.bits = width;
  p.counts = a.counts;
  p.cap = a.cap;
  set_chunks(p, a.cap);
  p.chunk_counts = bv.chunk_counts;
  p.digit_totals = bv.totals + kSortDigits * pass;
  return p;
}

template <class Scenes>
EmitArgs<Scenes> emit_args(const BinArgs<Scenes>& a) {
  EmitArgs<Scenes> e;
  e.scenes = a.scenes;
  e.total_slots = a.total_slots;
  e.list.order = a.geom.depth_val[1];
  e.list.prefix = a.geom.depth_key[0];
  e.list.starts = a.bin.starts;
  e.keys = a.bin.key[0];
  e.geom = a.geom;
  e.cap = a.cap;
  e.counts = a.counts;
  return e;
}

int slot_blocks(int64_t slots) { return (int)((slots + kPreprocessBlock - 1) / kPreprocessBlock); }
int rank_blocks_of(int64_t slots) { return (int)((slots + kRankBlock - 1) / kRankBlock); }

}  // namespace

// Step 1 of the binning, which needs no instance capacity: the depth order of the
// Gaussians and the prefix of their instance counts in that order.
int launch_depth_order(const GeomView& gv, int64_t slots, cudaStream_t st) {
  if (slots <= 0) return CFGS_OK;
  for (int pass = 0; pass < kDepthPasses; ++pass) launch_pass(depth_pass(gv, slots, pass), st);
  const int blocks = rank_blocks_of(slots);
  k_rank_sums<<<blocks, kPreprocessBlock, 0, st>>>(gv, slots);
  const bool scan = rank_scan_needed(blocks);
  if (scan) k_rank_scan<<<1, 1024, 0, st>>>(gv.rank_sums, blocks);
  k_rank_place<<<blocks, kPreprocessBlock, 0, st>>>(gv, slots, scan);
  return CFGS_OK;
}

// Steps 2-3, after launch_depth_order: tile keys, tile sort, tile ranges.
template <class Scenes>
int launch_instances(const BinArgs<Scenes>& a, cudaStream_t st) {
  if (a.total_slots > 0) {
    const EmitArgs<Scenes> e = emit_args(a);
    int passes, width;
    tile_sort_plan(a.num_tiles, &passes, &width);
    const SortPass first = tile_pass(a, 0, passes, width);
    k_emit_starts<Scenes><<<slot_blocks(a.total_slots), kPreprocessBlock, 0, st>>>(
        e, (uint32_t)(kSortThreads * first.items));
    if (first.items == 8) launch_emit_items<Scenes, 8>(e, first, st);
    else launch_emit_items<Scenes, 4>(e, first, st);
    for (int pass = 1; pass < passes; ++pass) launch_pass(tile_pass(a, pass, passes, width), st);
  }
  k_tile_ranges<<<1, 1024, 0, st>>>(a.tile_count, a.tile_range, (int)a.num_tiles);
  return CFGS_OK;
}

// ---- the binning as one persistent launch ----------------------------------------------
// The same block functions as the per-stage kernels above, run by a cooperative grid of
// resident 256-thread blocks: each stage's blocks are dealt out over the grid, and a
// bounded grid-wide wait separates the stages (each reads what the previous one wrote).
// The outputs are the per-stage launches' outputs (integer work, same order).
template <class Scenes>
struct PersistentBinArgs {
  SortPass depth[kDepthPasses];
  GeomView geom;
  int64_t slots;
  int rank_blocks, start_blocks;
  bool rank_scanned;
  EmitArgs<Scenes> emit;
  SortPass tile[kMaxTilePasses];
  int tile_passes;
  const uint32_t* tile_count;
  uint32_t* tile_range;
  int num_tiles;
  GridBarrier* barrier;
  uint32_t* flags;
};

template <class Scenes>
__global__ void __launch_bounds__(kSortThreads, 3) k_binning_persistent(PersistentBinArgs<Scenes> a) {
  static_assert(kSortThreads == kPreprocessBlock, "one block shape for every stage");
  constexpr int kItems = 4;  // every pass's chunks (launch_binning_persistent)
  __shared__ __align__(16) BinShared<kItems> sh;
  auto each = [&](int64_t blocks, auto&& block_fn) {
    for (int64_t b = blockIdx.x; b < blocks; b += gridDim.x) {
      block_fn((uint32_t)b);
      __syncthreads();  // the block's shared memory is reused by its next virtual block
    }
  };
  for (int pass = 0; pass < kDepthPasses; ++pass) {
    const SortPass& p = a.depth[pass];
    if (pass == 0) each(p.num_chunks, [&](uint32_t b) { sort_count_block<kItems, true>(p, sh, b); });
    else each(p.num_chunks, [&](uint32_t b) { sort_count_block<kItems, false>(p, sh, b); });
    if (!grid_barrier(a.barrier, a.flags)) return;
    if (!p.fold) {
      each(1 << p.bits, [&](uint32_t b) { sort_scan_block(p, sh.scan, (int)b); });
      if (!grid_barrier(a.barrier, a.flags)) return;
    }
    each(p.num_chunks, [&](uint32_t b) { sort_scatter_block<kItems, kValue>(p, a.emit.list, sh, b); });
    if (!grid_barrier(a.barrier, a.flags)) return;
  }
  each(a.rank_blocks, [&](uint32_t b) { rank_sums_block(a.geom, a.slots, sh.scan, (int)b); });
  if (!grid_barrier(a.barrier, a.flags)) return;
  if (a.rank_scanned) {
    if (blockIdx.x == 0) rank_scan_block(a.geom.rank_sums, a.rank_blocks, sh.scan);
    if (!grid_barrier(a.barrier, a.flags)) return;
  }
  each(a.rank_blocks, [&](uint32_t b) { rank_place_block(a.geom, a.slots, a.rank_scanned, sh.scan, (int)b); });
  if (!grid_barrier(a.barrier, a.flags)) return;
  each(a.start_blocks, [&](uint32_t b) { emit_starts_block<Scenes>(a.emit, kSortThreads * kItems, (int)b); });
  if (!grid_barrier(a.barrier, a.flags)) return;
  for (int pass = 0; pass < a.tile_passes; ++pass) {
    const SortPass& p = a.tile[pass];
    if (pass == 0) each(p.num_chunks, [&](uint32_t b) { emit_keys_block<Scenes, kItems>(a.emit, p, sh, b); });
    else each(p.num_chunks, [&](uint32_t b) { sort_count_block<kItems, false>(p, sh, b); });
    if (!grid_barrier(a.barrier, a.flags)) return;
    if (!p.fold) {
      each(1 << p.bits, [&](uint32_t b) { sort_scan_block(p, sh.scan, (int)b); });
      if (!grid_barrier(a.barrier, a.flags)) return;
    }
    if (pass == 0) each(p.num_chunks, [&](uint32_t b) { sort_scatter_block<kItems, kFirstPair>(p, a.emit.list, sh, b); });
    else each(p.num_chunks, [&](uint32_t b) { sort_scatter_block<kItems, kPair>(p, a.emit.list, sh, b); });
    if (!grid_barrier(a.barrier, a.flags)) return;
  }
  if (blockIdx.x == 0) tile_ranges_block<kScanItems>(a.tile_count, a.tile_range, a.num_tiles, sh.scan);
}

// The pass descriptions of launch_depth_order and launch_instances, for one launch.
template <class Scenes>
int launch_binning_persistent(const BinArgs<Scenes>& a, GridBarrier* barrier, cudaStream_t st) {
  if (a.total_slots <= 0) return launch_instances(a, st);
  PersistentBinArgs<Scenes> pa{};
  auto narrow = [](SortPass p, int64_t n) {
    p.items = 4;
    p.num_chunks = sort_chunks(n, kSortThreads * 4);
    p.fold = fold_counts(p.num_chunks);
    return p;
  };
  for (int pass = 0; pass < kDepthPasses; ++pass)
    pa.depth[pass] = narrow(depth_pass(a.geom, a.total_slots, pass), a.total_slots);
  pa.geom = a.geom;
  pa.slots = a.total_slots;
  pa.rank_blocks = rank_blocks_of(a.total_slots);
  pa.start_blocks = slot_blocks(a.total_slots);
  pa.rank_scanned = rank_scan_needed(pa.rank_blocks);
  pa.emit = emit_args(a);
  int passes, width;
  tile_sort_plan(a.num_tiles, &passes, &width);
  if (passes > kMaxTilePasses) return CFGS_ERR_TOO_LARGE;
  pa.tile_passes = passes;
  for (int pass = 0; pass < passes; ++pass) pa.tile[pass] = narrow(tile_pass(a, pass, passes, width), a.cap);
  pa.tile_count = a.tile_count;
  pa.tile_range = a.tile_range;
  pa.num_tiles = (int)a.num_tiles;
  pa.barrier = barrier;
  pa.flags = &a.counts->flags;

  // every block resident: the grid is the kernel's occupancy times the SM count (per device)
  static std::atomic<int> grid_of_device[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return CFGS_ERR_LAUNCH;
  int grid = dev < 64 ? grid_of_device[dev].load(std::memory_order_acquire) : 0;
  if (grid <= 0) {
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_binning_persistent<Scenes>, kSortThreads, 0) !=
            cudaSuccess ||
        sms <= 0 || per_sm <= 0)
      return CFGS_ERR_LAUNCH;
    grid = sms * per_sm;
    if (dev < 64) grid_of_device[dev].store(grid, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kSortThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, k_binning_persistent<Scenes>, pa) != cudaSuccess) return CFGS_ERR_LAUNCH;
  return CFGS_OK;
}
template int launch_binning_persistent<SceneTable>(const BinArgs<SceneTable>&, GridBarrier*, cudaStream_t);

template <class Scenes>
int launch_binning(const BinArgs<Scenes>& a, cudaStream_t st) {
  const int s = launch_depth_order(a.geom, a.total_slots, st);
  return s != CFGS_OK ? s : launch_instances(a, st);
}
template int launch_binning<SingleScene>(const BinArgs<SingleScene>&, cudaStream_t);

// Stable LSD radix sort of n (key, value) pairs by the low `bits` key bits, passes of at
// most 8 bits, ping-ponging between (keys[0], vals[0]) and (keys[1], vals[1]); returns
// the index (0 or 1) of the buffers holding the result. chunk_counts holds
// 256 x sort_chunks(n, kTileChunk) values, totals 256 x kMaxTilePasses.
int sort_pairs(uint32_t* keys[2], uint32_t* vals[2], int64_t n, int bits, uint32_t* chunk_counts, uint32_t* totals,
               cudaStream_t st, int* result) {
  if (bits < 1 || bits > 32 || n < 0 || n > 0x7fffffffll) return CFGS_ERR_INVALID_ARGUMENT;
  const int passes = (bits + 7) / 8;
  const int width = (bits + passes - 1) / passes;
  int src = 0;
  for (int pass = 0; pass < passes; ++pass) {
    SortPass p{};
    const int dst = src ^ 1;
    p.key_in = keys[src];
    p.val_in = vals[src];
    p.key_out = keys[dst];
    p.val_out = vals[dst];
    p.shift = width * pass;
    p.bits = min(width, bits - width * pass);
    p.n = n;
    p.cap = n;
    set_chunks(p, n);
    p.chunk_counts = chunk_counts;
    p.digit_totals = totals + kSortDigits * pass;
    if (n > 0) launch_pass(p, st);
    src = dst;
  }
  *result = src;
  return CFGS_OK;
}

template int launch_binning<SceneTable>(const BinArgs<SceneTable>&, cudaStream_t);

}  // namespace cfgs

using namespace cfgs;

namespace {

// The single-scene binning arguments of the drop-in path.
int single_bin_args(const CfgsSettings* s, const CfgsGaussians* g, void* geom, void* image, void* binning,
                    int64_t capacity, BinArgs<SingleScene>* a) {
  if (!s || !g || !geom || !image || !binning || capacity < 0) return CFGS_ERR_INVALID_ARGUMENT;
  if (s->image_width <= 0 || s->image_height <= 0 || g->num_gaussians < 0) return CFGS_ERR_INVALID_ARGUMENT;
  if (capacity > 0x7fffffffll) return CFGS_ERR_TOO_LARGE;
  ImageLayout IL(s->image_width, s->image_height);
  ImageView iv(image, s->image_width, s->image_height);
  a->scenes.d = single_scene_desc(s, g->num_gaussians, g->sh_coeffs);
  a->total_slots = g->num_gaussians;
  a->geom = GeomView(geom, g->num_gaussians);
  a->bin = BinningView(binning, capacity);
  a->cap = capacity;
  a->counts = iv.counts;
  a->num_tiles = IL.num_tiles;
  a->tile_count = iv.tile_count;
  a->tile_range = iv.tile_range;
  return CFGS_OK;
}

}  // namespace

extern "C" int cfgs_bin_forward(const CfgsSettings* s, const CfgsGaussians* g, void* geom, void* image, void* binning,
                                int64_t capacity, void* stream) {
  BinArgs<SingleScene> a;
  int status = single_bin_args(s, g, geom, image, binning, capacity, &a);
  if (status != CFGS_OK) return status;
  cudaStream_t st = (cudaStream_t)stream;
  status = launch_binning(a, st);
  if (status != CFGS_OK) return status;
  CFGS_CHECK_LAUNCH(s->debug, st);
  return CFGS_OK;
}

extern "C" int cfgs_depth_order(int32_t num_gaussians, void* geom, void* stream) {
  if (num_gaussians < 0 || (num_gaussians > 0 && !geom)) return CFGS_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  const int status = launch_depth_order(GeomView(geom, num_gaussians), num_gaussians, st);
  if (status != CFGS_OK) return status;
  CFGS_CHECK_LAUNCH(0, st);
  return CFGS_OK;
}

extern "C" int cfgs_bin_instances(const CfgsSettings* s, const CfgsGaussians* g, void* geom, void* image,
                                  void* binning, int64_t capacity, void* stream) {
  BinArgs<SingleScene> a;
  int status = single_bin_args(s, g, geom, image, binning, capacity, &a);
  if (status != CFGS_OK) return status;
  cudaStream_t st = (cudaStream_t)stream;
  status = launch_instances(a, st);
  if (status != CFGS_OK) return status;
  CFGS_CHECK_LAUNCH(s->debug, st);
  return CFGS_OK;
}

extern "C" void cfgs_binning_layout(int64_t cap, size_t o[8]) {
  BinningLayout L(cap);
  size_t v[8] = {L.key, L.gid, L.pidx, L.sorted_gid, L.sorted_pidx, L.chunk_counts, L.totals, L.total};
  for (int i = 0; i < 8; ++i) o[i] = v[i];
}
