// rt_sort.cu -- stable LSD radix sort of 32-bit keys with optional 32-bit
// values, 8-bit digits, a count and a scatter launch per digit pass.
//
// Replaces the reference's sort family (CUDA_radixSortGeneral, CUDA_radixSort,
// CUDA_bitonicSort*, CUDA_bubbleSort512; kernels/CUDA_radixSortGeneral.cu:397-482
// etc.), which serialises its shared histogram 256 ways and ranks keys with
// warp-synchronous code that is undefined on Volta and later. Here:
//   * the keys are cut into chunks of whole tiles, about two chunks per SM; a
//     pass is two launches. k_sort_count reads its chunk's keys and writes the
//     chunk's 256 digit counts (and adds them to a sum per 16 chunks);
//     k_sort_scatter adds up the counts before its chunk, then takes the
//     chunk's tiles one after another (with few chunks it counts the keys
//     itself, and the pass is one launch): ranks the keys stably (the lanes of
//     equal digit, plus per-warp counters),
//     stages the tile in shared memory in sorted order and writes it out so
//     that consecutive threads write consecutive addresses of each digit run,
//     while the next tile's keys are on their way. No CTA waits for another.
//   * segments (the meshes of a batched build) are sorted side by side: every
//     chunk belongs to one segment, and counts are added up inside it, so the
//     segment number is not a sort key of those passes. Where segments are short
//     on average, the short ones go several to a CTA, which does every pass of
//     both of a build's sorts in shared memory (k_sort_segments); so does a
//     whole build of at most 4096 faces.
//   * n <= 4096, one segment: a single CTA does every pass in shared memory
//     (one launch).
// Traffic per pass: keys (and values) read once and written once, and the keys
// once more for the counts (from L2 when the keys fit there). One launch per
// pass with a decoupled look-back over the earlier tiles' counts (which this
// replaces) moved 4 bytes per pair less, but a pass over 2^24 pairs took
// 166 us of which the look-back's L2 round trips were most.
#include "rt_common.cuh"

namespace rt {
namespace {

// single-CTA sort of up to one tile
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 16;
constexpr int kTile = kThreads * kItems;  // 4096
constexpr int kRadix = 256;

// chunked passes
constexpr int kScThreads = 512;
constexpr int kScWarps = kScThreads / 32;
constexpr int kCountThreads = 1024;
constexpr int kMaskRows = 3;  // of every four rows of a warp, those ranked by masks in shared memory (the fourth by ballots)
constexpr int kGroup = 16;  // chunks whose counts are also kept as one sum
constexpr int kMaxPasses = 4;
constexpr uint32_t kMaxKeys = (1u << 30) - 1u;

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Block-wide exclusive scan of one value per thread (NT threads).
template <int NT>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_warp, uint32_t& total) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < NW ? s_warp[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < NW) s_warp[lane] = w;
  }
  __syncthreads();
  uint32_t warp_prefix = warp ? s_warp[warp - 1] : 0u;
  total = s_warp[NW - 1];
  __syncthreads();
  return warp_prefix + x - v;
}

// The lanes of the warp whose 9-bit digit equals this lane's (digits 0..255, 256 for a lane without a key): one
// ballot per bit, each lane keeping the lanes that agree with it on that bit -- the mask __match_any_sync gives.
__device__ __forceinline__ uint32_t match_digit(uint32_t d) {
  uint32_t m = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    const bool bit = (d >> b) & 1u;
    const uint32_t v = __ballot_sync(0xffffffffu, bit);
    m &= bit ? v : ~v;
  }
  return m;
}

// First chunk of segment m, whose keys start at F, among chunks of per_chunk keys (chunks never span segments). Where
// short segments have no chunks, a segment has more than kSegWindow keys, and the windows before it serve as well as the
// segments before it to keep one segment's chunks apart from the next one's, however many segments there are.
constexpr uint32_t kSegWindow = 2048;
__host__ __device__ __forceinline__ uint32_t chunk_base(uint32_t F, uint32_t m, uint32_t per_chunk, uint32_t short_segs) {
  return F / per_chunk + (short_segs ? F / kSegWindow : m);
}

// One pass over chunked keys. kMode 0: keys_in are the keys; 1: the key of position i is the split level of the sorted
// Morton codes in keys_in, clz(code[i] ^ code[i + 1]) (32 for equal codes and for a segment's last position).
struct PassArgs {
  const uint32_t* keys_in;
  const uint32_t* vals_in;  // null: value i is val_base + i
  uint32_t* keys_out;       // null: the sorted keys are not needed
  uint32_t* vals_out;
  uint32_t n, shift, val_base;
  uint32_t per_chunk;        // keys of a whole chunk
  const uint32_t* seg_off;   // null: one segment, 0 .. n
  const uint32_t* chunk_seg; // segment of each chunk (~0: no chunk); with seg_off
  uint32_t short_segs;       // segments of at most kSegWindow keys have no chunks
  uint32_t* rows;            // [chunks][256]; null: few chunks of one segment, whose CTAs count the keys themselves
  uint32_t* groups;          // [chunks / kGroup + 1][256], zero before the pass
  uint32_t* totals;          // optional: [segments][totals_stride] digit counts
  uint32_t totals_stride;
};
struct Chunk {
  uint32_t seg_begin, seg_end;    // keys of the segment
  uint32_t first_chunk, n_chunks; // its chunks
  uint32_t begin, end;            // keys of this chunk
  uint32_t seg;
};
__device__ __forceinline__ bool chunk_of(const PassArgs& P, uint32_t c, Chunk& C) {
  if (!P.seg_off) {
    C.seg = 0; C.seg_begin = 0; C.seg_end = P.n; C.first_chunk = 0;
  } else {
    C.seg = __ldg(P.chunk_seg + c);
    if (C.seg == ~0u) return false;
    C.seg_begin = __ldg(P.seg_off + C.seg);
    C.seg_end = __ldg(P.seg_off + C.seg + 1);
    C.first_chunk = chunk_base(C.seg_begin, C.seg, P.per_chunk, P.short_segs);
  }
  C.n_chunks = (C.seg_end - C.seg_begin + P.per_chunk - 1) / P.per_chunk;
  C.begin = C.seg_begin + (c - C.first_chunk) * P.per_chunk;
  C.end = C.seg_end - C.begin <= P.per_chunk ? C.seg_end : C.begin + P.per_chunk;
  return true;
}
template <int kMode>
__device__ __forceinline__ uint32_t load_key(const PassArgs& P, const Chunk& C, uint32_t i) {
  const uint32_t k = __ldg(P.keys_in + i);
  if (kMode == 0) return k;
  if (i + 1 >= C.seg_end) return 32u;
  const uint32_t x = k ^ __ldg(P.keys_in + i + 1);
  return x ? (uint32_t)__clz(x) : 32u;
}

// Digit counts of one chunk. Sixteen counters per digit, picked by lane, keep equal digits of a warp apart (Morton
// codes and split levels come in long runs of equal digits).
template <int kBits, int kMode>
__global__ __launch_bounds__(kCountThreads) void k_sort_count(PassArgs P) {
  constexpr uint32_t D = 1u << kBits;
  __shared__ uint32_t h[D * 16];
  Chunk C;
  if (!chunk_of(P, blockIdx.x, C)) return;
  for (uint32_t i = threadIdx.x; i < D * 16; i += kCountThreads) h[i] = 0;
  __syncthreads();
  const uint32_t copy = threadIdx.x & 15u;
  for (uint32_t base = C.begin + threadIdx.x; base < C.end; base += 8 * kCountThreads) {
    uint32_t k[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t i = base + q * kCountThreads;  // below 2^31: positions are below 2^30
      k[q] = i < C.end ? load_key<kMode>(P, C, i) : 0u;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (base + q * kCountThreads < C.end) atomicAdd(&h[((k[q] >> P.shift) & (D - 1u)) * 16u + copy], 1u);
  }
  __syncthreads();
  const uint32_t d = threadIdx.x;
  if (d < kRadix) {
    uint32_t sum = 0;
    if (d < D) {
#pragma unroll
      for (uint32_t q = 0; q < 16; ++q) sum += h[d * 16u + ((q + d) & 15u)];
    }
    P.rows[(size_t)blockIdx.x * kRadix + d] = sum;
    if (sum) atomicAdd(P.groups + (size_t)(blockIdx.x / kGroup) * kRadix + d, sum);
  }
}

// Sum of the 256-word rows [from, to) at one digit, eight loads in flight; `upto` (from <= upto): the part below it.
__device__ __forceinline__ void sum_rows(const uint32_t* __restrict__ rows, uint32_t d, uint32_t from, uint32_t to, uint32_t upto,
                                         uint32_t& all, uint32_t& part) {
  for (uint32_t x = from; x < to; x += 8) {
    uint32_t v[8];
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) v[q] = x + q < to ? __ldg(rows + (size_t)(x + q) * kRadix + d) : 0u;
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
      all += v[q];
      if (x + q < upto) part += v[q];
    }
  }
}

// The tiles of one chunk, in order. What bounds it: the shared-memory pipe (ranking, and the move of the tile into
// sorted order: about 30 wavefronts per 32 keys) beside the integer pipe, at two CTAs per SM. 2^24 pairs, whole
// sort: ballots alone 561 us (60% of the integer pipe), masks alone 463 (equal digits everywhere: 523), three rows of
// masks to one of ballots 461 (467); __match_any_sync 750; the look-back sort that this replaced 694.
template <bool kVals, int kItems, int kBits, int kMode>
__global__ __launch_bounds__(kScThreads, kItems == 16 ? 2 : 3) void k_sort_scatter(PassArgs P) {
  constexpr uint32_t T = kScThreads * kItems, D = 1u << kBits;
  extern __shared__ uint32_t s_dyn[];
  uint32_t* s_keys = s_dyn;
  uint32_t* s_vals = s_dyn + T;                  // kVals only
  uint32_t* s_mask = s_dyn + T * (kVals ? 2 : 1) + (threadIdx.x >> 5) * D;  // the warp's masks
  __shared__ __align__(16) uint16_t s_cnt[kScWarps][kRadix];  // per warp and digit: count, then the place of its first key in the tile
  __shared__ uint32_t s_out[kRadix];             // where the tile's run of a digit goes, less where it starts in the tile
  __shared__ uint32_t s_half[2 * kRadix];
  __shared__ uint32_t s_scan[8];
  Chunk C;
  if (!chunk_of(P, blockIdx.x, C)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t lt = lanemask_lt();
  const uint32_t lane0 = (uint32_t)warp * (kItems * 32) + lane;  // the warp's keys of a tile: kItems rows of 32

  uint32_t key[kItems];
  auto load_tile = [&](uint32_t base) {
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const uint32_t i = base + lane0 + r * 32;
      key[r] = i < C.end ? load_key<kMode>(P, C, i) : 0u;
    }
  };
  load_tile(C.begin);

  // where this chunk's keys of each digit start: the segment's keys of smaller digits, then the digit's keys in
  // earlier chunks. Threads 0 .. 255 add up whole groups, threads 256 .. 511 the rows beside them.
  uint32_t next = 0;  // thread d < 256: where the next tile's keys of digit d go
  {
    const uint32_t c = blockIdx.x, cs = C.first_chunk, ce = cs + C.n_chunks, d = tid & 255u;
    const uint32_t g0 = (cs + kGroup - 1) / kGroup, g1 = max(g0, ce / kGroup);  // whole groups of the segment
    uint32_t all = 0, part = 0;
    if (!P.rows) {
      uint32_t* const s_own = s_dyn;  // keys before the chunk, then the others: four counters per digit each, picked by lane
      for (uint32_t i = tid; i < 8 * D; i += kScThreads) s_own[i] = 0;
      __syncthreads();
      for (uint32_t i0 = tid; i0 < P.n; i0 += 8 * kScThreads) {
        uint32_t k[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) k[q] = i0 + q * kScThreads < P.n ? load_key<kMode>(P, C, i0 + q * kScThreads) : 0u;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const uint32_t i = i0 + q * kScThreads;
          if (i < P.n) atomicAdd(&s_own[(i < C.begin ? 0u : 4u * D) + ((k[q] >> P.shift) & (D - 1u)) * 4u + (lane & 3u)], 1u);
        }
      }
      __syncthreads();
      if (tid < (int)D) {
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
          part += s_own[4 * d + q];
          all += s_own[4 * (D + d) + q];
        }
        all += part;
      }
    } else if (d < D) {
      if (tid < kRadix) {
        sum_rows(P.groups, d, g0, g1, c / kGroup, all, part);
      } else {
        const uint32_t h1 = min(ce, g0 * kGroup), t0 = max(h1, g1 * kGroup);
        sum_rows(P.rows, d, cs, h1, c, all, part);
        sum_rows(P.rows, d, t0, ce, c, all, part);
        const uint32_t own = c / kGroup;
        uint32_t unused = 0;
        if (own >= g0 && own < g1) sum_rows(P.rows, d, own * kGroup, c, c, unused, part);  // earlier chunks of its own group
      }
    }
    if (tid >= kRadix) { s_half[d] = all; s_half[kRadix + d] = part; }
    __syncthreads();
    uint32_t x = 0;
    if (tid < kRadix) {
      all += s_half[d];
      part += s_half[kRadix + d];
      x = all;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) s_scan[warp] = x;
    }
    __syncthreads();
    if (tid < kRadix) {
      uint32_t before = 0;
      for (int w = 0; w < warp; ++w) before += s_scan[w];
      next = C.seg_begin + before + x - all + part;
      if (P.totals && c == cs && d < P.totals_stride) P.totals[(size_t)C.seg * P.totals_stride + d] = all;
    }
  }

  for (uint32_t q = lane; q < D; q += 32) s_mask[q] = 0;
  for (uint32_t base = C.begin; base < C.end; base += T) {
    const uint32_t tile_n = min(T, C.end - base);
    // stable ranks inside the tile, the warp's counters in its own row of s_cnt. The lanes of equal digit come from a
    // mask per digit in shared memory that every lane sets its bit in (and the first of them clears), or from one
    // ballot per digit bit: masks load the shared-memory pipe, ballots the integer pipe, so a warp uses both.
    *reinterpret_cast<uint4*>(&s_cnt[warp][8 * lane]) = make_uint4(0, 0, 0, 0);
    __syncwarp();
    uint32_t rank[kItems / 2] = {};  // two 16-bit ranks per word
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      if ((uint32_t)warp * (kItems * 32) + r * 32 >= tile_n) continue;  // a row without keys (the same for the warp)
      const bool valid = lane0 + r * 32 < tile_n;
      const uint32_t d = (key[r] >> P.shift) & (D - 1u);
      uint32_t peers;
      const bool by_mask = r % 4 < kMaskRows;
      if (by_mask) {
        if (valid) atomicOr(&s_mask[d], 1u << lane);
        __syncwarp();
        peers = s_mask[d];
      } else {
        peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < kBits; ++b) {
          const bool bit = (d >> b) & 1u;
          const uint32_t v = __ballot_sync(0xffffffffu, bit);
          peers &= bit ? v : ~v;
        }
      }
      const uint32_t pre = s_cnt[warp][d];
      rank[r / 2] |= (pre + __popc(peers & lt)) << (16 * (r & 1));
      __syncwarp();
      if (valid && (peers & lt) == 0) {
        s_cnt[warp][d] = (uint16_t)(pre + __popc(peers));
        if (by_mask) s_mask[d] = 0;
      }
      __syncwarp();
    }
    uint32_t val[kVals ? kItems : 1];
    if (kVals) {
#pragma unroll
      for (int r = 0; r < kItems; ++r) {
        const uint32_t i = base + lane0 + r * 32;
        val[r] = P.vals_in ? (i < C.end ? __ldg(P.vals_in + i) : 0u) : P.val_base + i;
      }
    }
    __syncthreads();
    // threads 0 .. 255, one digit each: the tile's run of the digit and where each warp's keys start in it
    uint32_t x = 0, tile_count = 0;
    if (tid < kRadix) {
#pragma unroll
      for (int w = 0; w < kScWarps; ++w) tile_count += s_cnt[w][tid];
      x = tile_count;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) s_scan[warp] = x;
    }
    __syncthreads();
    if (tid < kRadix) {
      uint32_t start = x - tile_count;
      for (int w = 0; w < warp; ++w) start += s_scan[w];
      s_out[tid] = next - start;
      next += tile_count;
#pragma unroll
      for (int w = 0; w < kScWarps; ++w) {
        const uint32_t c = s_cnt[w][tid];
        s_cnt[w][tid] = (uint16_t)start;
        start += c;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      if (lane0 + r * 32 < tile_n) {
        const uint32_t pos = s_cnt[warp][(key[r] >> P.shift) & (D - 1u)] + ((rank[r / 2] >> (16 * (r & 1))) & 0xffffu);
        s_keys[pos] = key[r];
        if (kVals) s_vals[pos] = val[r];
      }
    }
    if (base + T < C.end) load_tile(base + T);  // on its way while this tile is written out
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const uint32_t i = tid + r * kScThreads;
      if (i < tile_n) {
        const uint32_t k = s_keys[i];
        const uint32_t out = s_out[(k >> P.shift) & (D - 1u)] + i;
        if (P.keys_out) P.keys_out[out] = k;
        if (kVals) P.vals_out[out] = s_vals[i];
      }
    }
  }
}

// The segment of every chunk (~0 for a gap of the chunk numbering).
__global__ __launch_bounds__(256) void k_chunk_segs(const uint32_t* __restrict__ off, uint32_t M, uint32_t per_chunk, uint32_t short_segs,
                                                    uint32_t chunks, uint32_t* __restrict__ chunk_seg) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= chunks) return;
  uint32_t lo = 0, hi = M - 1;  // largest m with chunk_base(off[m], m) <= c
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (chunk_base(__ldg(off + mid), mid, per_chunk, short_segs) <= c) lo = mid; else hi = mid - 1;
  }
  const uint32_t F = __ldg(off + lo), n = __ldg(off + lo + 1) - F, j = c - chunk_base(F, lo, per_chunk, short_segs);
  const bool has = (uint64_t)j * per_chunk < n && !(short_segs && n <= kSegWindow);
  chunk_seg[c] = has ? lo : ~0u;
}

// Both sorts of a build for short segments: a CTA takes the segments of at most `window` keys that start in its window of
// so many positions (a longer one is the window's last, and left out), at most 4096 keys in all, and does every pass in
// shared memory: by code (four digits), by segment where there are several; then the split levels by level and by
// segment. The threads' rows of a pass are as many as the keys need. Bound by the latency of its eight to ten passes. What
// it replaces at these sizes is a chain of eleven launches, with a CTA of its own for every segment in ten of them; whole
// builds of 65,536 meshes of 10 faces 8.65 -> 3.06 ms, 20,000 of 100 3.92 -> 1.54, 1024 of 200 284 -> 216 us, 16 of 64
// 128 -> 81, one mesh of 4096 124 -> 106, of 17 75 -> 56.
constexpr int kSegThreads = 512;
constexpr int kSegWarps = kSegThreads / 32;
constexpr int kSegItems = kTile / kSegThreads;
constexpr size_t kSegSmem = kTile * (2 * 4 + 3 * 2);
__global__ __launch_bounds__(kSegThreads) void k_sort_segments(uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n,
                                                               const uint32_t* __restrict__ off, uint32_t M, uint32_t window,
                                                               uint32_t* __restrict__ splits, uint32_t* __restrict__ level_counts,
                                                               uint32_t stride) {
  extern __shared__ uint32_t dyn[];
  uint32_t *k0 = dyn, *k1 = dyn + kTile;  // keys, and where the pass puts them
  uint16_t *v0 = (uint16_t*)(dyn + 2 * kTile), *v1 = v0 + kTile;
  uint16_t* const seg = v0 + 2 * kTile;  // segment of each input position, counted from the CTA's first
  __shared__ __align__(16) uint16_t s_cnt[kSegWarps][kRadix];
  __shared__ uint32_t s_start[kRadix];
  __shared__ uint32_t s_warp[kRadix / 32];
  __shared__ uint32_t s_m[2];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, lt = lanemask_lt();
  uint32_t m0 = 0, m1 = 1, a = 0, e = n;
  if (off) {
    if (warp < 2) {  // the segments that start before the window (warp 0) and before its end (warp 1), 32 places at a time
      const uint64_t x = (uint64_t)(blockIdx.x + warp) * window;
      uint32_t lo = 0, len = M;  // the answer is in lo .. lo + len
      while (len > 0) {
        const uint32_t step = (len + 31) / 32, at = lane * step;
        const uint32_t c = (uint32_t)__popc(__ballot_sync(0xffffffffu, at < len && __ldg(off + lo + at) < x));
        if (c == 0) break;
        lo += (c - 1) * step + 1;
        len = min(step, len - (c - 1) * step) - 1;
      }
      if (lane == 0) s_m[warp] = lo;
    }
    __syncthreads();
    m0 = s_m[0];
    m1 = s_m[1];
    if (m0 >= m1) return;
    a = __ldg(off + m0);
    e = __ldg(off + m1);
    const uint32_t last = __ldg(off + m1 - 1);
    if (e - last > window) { e = last; --m1; }
  }
  const uint32_t count = e - a, segs = m1 - m0, items = (count + kSegThreads - 1) / kSegThreads;
  if (count == 0 || items > (uint32_t)kSegItems) return;
  for (uint32_t i = tid; i < count; i += kSegThreads) {
    k0[i] = keys[a + i];
    v0[i] = (uint16_t)i;
    uint32_t lo = 0, hi = segs - 1;
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (__ldg(off + m0 + mid) <= a + i) lo = mid; else hi = mid - 1;
    }
    seg[i] = (uint16_t)lo;
  }
  for (uint32_t i = tid; i < segs * 64u; i += kSegThreads)
    if ((i & 63u) < stride) level_counts[(size_t)(m0 + (i >> 6)) * stride + (i & 63u)] = 0;

  // one stable pass by eight bits of the keys, or of the values' segments
  auto pass = [&](uint32_t shift, bool by_seg) {
    *reinterpret_cast<uint4*>(&s_cnt[warp][8 * lane]) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    uint32_t place[kSegItems], digit[kSegItems];
#pragma unroll
    for (int r = 0; r < kSegItems; ++r) {
      if ((uint32_t)r >= items) break;
      const uint32_t p = (warp * items + r) * 32 + lane;
      const bool valid = p < count;
      const uint32_t w = !valid ? 0u : by_seg ? seg[v0[p]] : k0[p], d = (w >> shift) & 255u;
      uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t v = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? v : ~v;
      }
      const uint32_t pre = s_cnt[warp][d];
      digit[r] = d;
      place[r] = pre + __popc(peers & lt);
      __syncwarp();
      if (valid && (peers & lt) == 0) s_cnt[warp][d] = (uint16_t)(pre + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    uint32_t x = 0, total = 0;
    if (tid < kRadix) {
#pragma unroll
      for (int w = 0; w < kSegWarps; ++w) {
        const uint32_t c = s_cnt[w][tid];
        s_cnt[w][tid] = (uint16_t)total;
        total += c;
      }
      x = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
      }
      if (lane == 31) s_warp[warp] = x;
    }
    __syncthreads();
    if (tid < kRadix) {
      uint32_t start = x - total;
      for (uint32_t w = 0; w < warp; ++w) start += s_warp[w];
      s_start[tid] = start;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSegItems; ++r) {
      if ((uint32_t)r >= items) break;
      const uint32_t p = (warp * items + r) * 32 + lane;
      if (p < count) {
        const uint32_t to = s_start[digit[r]] + s_cnt[warp][digit[r]] + place[r];
        k1[to] = k0[p];
        v1[to] = v0[p];
      }
    }
    __syncthreads();
    uint32_t* const k = k0; k0 = k1; k1 = k;
    uint16_t* const v = v0; v0 = v1; v1 = v;
  };
  __syncthreads();
  for (uint32_t shift = 0; shift < 32; shift += 8) pass(shift, false);
  if (segs > 1) pass(0, true);
  if (segs > 256) pass(8, true);
  for (uint32_t i = tid; i < count; i += kSegThreads) {
    const uint32_t code = k0[i], s = seg[v0[i]];
    keys[a + i] = code;
    vals[a + i] = a + v0[i];
    uint32_t level = 32;
    if (i + 1 < count && seg[v0[i + 1]] == s) {
      const uint32_t x = code ^ k0[i + 1];
      if (x) level = (uint32_t)__clz(x);
    }
    k1[i] = s << 8 | level;
    v1[i] = (uint16_t)i;
  }
  __syncthreads();
  uint32_t* const k = k0; k0 = k1; k1 = k;
  uint16_t* const v = v0; v0 = v1; v1 = v;
  pass(0, false);
  if (segs > 1) pass(8, false);
  if (segs > 256) pass(16, false);
  for (uint32_t base = warp * 32; base < count; base += kSegThreads) {
    const uint32_t i = base + lane;
    const bool valid = i < count;
    const uint32_t key = valid ? k0[i] : ~0u, before = __shfl_up_sync(0xffffffffu, key, 1);
    if (valid) splits[a + i] = a + v0[i] + 1;
    // the first lane of a run of one segment and level counts it
    const bool head = lane == 0 || key != before;
    const uint32_t heads = __ballot_sync(0xffffffffu, head) & ~(lt | 1u << lane);
    if (valid && head && (key & 255u) < stride)
      atomicAdd(level_counts + (size_t)(m0 + (key >> 8)) * stride + (key & 255u), (heads ? (uint32_t)__ffs((int)heads) - 1u : 32u) - lane);
  }
}

// n <= kTile: every pass in shared memory, one CTA. Dynamic shared memory:
// 2 x kTile keys (+ 2 x kTile values).
template <bool kVals>
__global__ __launch_bounds__(kThreads) void k_radix_small(uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n,
                                                         uint32_t begin_bit, uint32_t passes, int init_vals) {
  extern __shared__ uint32_t dyn[];
  uint32_t* kbuf[2] = {dyn, dyn + kTile};
  uint32_t* vbuf[2] = {dyn + 2 * kTile, dyn + 3 * kTile};
  __shared__ uint32_t s_cnt[kWarps][kRadix + 1];
  __shared__ uint32_t s_tile_start[kRadix];
  __shared__ uint32_t s_warp[kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t lt = lanemask_lt();
  for (uint32_t i = threadIdx.x; i < n; i += kThreads) {
    kbuf[0][i] = keys[i];
    if (kVals) vbuf[0][i] = init_vals ? i : vals[i];
  }
  __syncthreads();
  int cur = 0;
  for (uint32_t p = 0; p < passes; ++p) {
    const uint32_t shift = begin_bit + 8 * p;
    for (int i = threadIdx.x; i < kWarps * (kRadix + 1); i += kThreads) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    uint32_t rank[kItems];
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      uint32_t idx = warp * (kItems * 32) + r * 32 + lane;
      uint32_t d = idx < n ? ((kbuf[cur][idx] >> shift) & 255u) : (uint32_t)kRadix;
      uint32_t peers = match_digit(d);
      uint32_t pre = s_cnt[warp][d];
      rank[r] = pre + __popc(peers & lt);
      __syncwarp();
      if ((peers & lt) == 0) s_cnt[warp][d] = pre + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      uint32_t c = s_cnt[w][threadIdx.x];
      s_cnt[w][threadIdx.x] = run;
      run += c;
    }
    uint32_t total;
    s_tile_start[threadIdx.x] = block_excl_scan<kThreads>(run, s_warp, total);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      uint32_t idx = warp * (kItems * 32) + r * 32 + lane;
      if (idx < n) {
        uint32_t k = kbuf[cur][idx];
        uint32_t d = (k >> shift) & 255u;
        uint32_t pos = s_tile_start[d] + s_cnt[warp][d] + rank[r];
        kbuf[cur ^ 1][pos] = k;
        if (kVals) vbuf[cur ^ 1][pos] = vbuf[cur][idx];
      }
    }
    __syncthreads();
    cur ^= 1;
  }
  for (uint32_t i = threadIdx.x; i < n; i += kThreads) {
    keys[i] = kbuf[cur][i];
    if (kVals) vals[i] = vbuf[cur][i];
  }
}

__global__ void k_iota(uint32_t* v, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = i;
}

constexpr size_t kSmallSmem = 4 * kTile * sizeof(uint32_t);

// The single-block sort's 64 KB of dynamic shared memory, allowed once per device.
bool small_smem_ready() {
  static PerDeviceOnce once;
  return once.run([] {
    cudaError_t a = cudaFuncSetAttribute(k_radix_small<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem);
    cudaError_t b = cudaFuncSetAttribute(k_radix_small<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem);
    return a == cudaSuccess && b == cudaSuccess;
  });
}

// Tiles and chunks of an n-key sort with M segments. Tiles of 2048, 4096 or 8192 keys (4, 8 or 16 per thread): the
// smallest that leaves every SM's two (three for 4096) resident CTAs at most one tile each, so that small sorts
// spread over the chip and large ones have long digit runs; chunks of as many whole tiles as give two CTAs per SM.
// 2^24 pairs: 8192-key tiles take 461 us, 6144 about 480, 4096 (three CTAs per SM) 610. The plan takes 148 SMs whatever the
// device has: the scratch that a caller sized by it must not depend on the device that is current then and later (with
// fewer SMs the chunks run in more than one wave, with the same results).
struct SortPlan {
  uint32_t items, per_chunk, chunks;
  uint32_t short_segs;  // segments of at most kSegWindow keys go to k_sort_segments
};
SortPlan sort_plan(uint32_t n, uint32_t M) {
  constexpr uint32_t kSms = 148;
  SortPlan P;
  P.items = n <= 2 * kSms * kScThreads * 4 ? 4 : (n <= 3 * kSms * kScThreads * 8 ? 8 : 16);
  const uint32_t T = kScThreads * P.items, tiles = (uint32_t)(((uint64_t)n + T - 1) / T);
  const uint32_t per = P.items == 16 ? (tiles + 2 * kSms - 1) / (2 * kSms) : 1;
  P.per_chunk = per * T;
  // With fewer than kSegWindow keys a segment on average, a chunk of its own for each would be mostly set-up (and 1 KB of
  // counts each: 90 MB for 65,536 meshes of 10 faces, now 6): the short ones go to k_sort_segments, one CTA for every
  // kSegWindow keys. 4096 meshes of 2000 faces: whole build 2.03 -> 1.81 ms; with more faces a mesh on average most
  // segments are longer than a window anyway.
  P.short_segs = M > 1 && M > n / kSegWindow ? 1u : 0u;
  P.chunks = M > 1 ? chunk_base(n, M, P.per_chunk, P.short_segs) + P.short_segs : (tiles + per - 1) / per;
  return P;
}
// Scratch regions, in carve order: the other key and value buffers, the chunks' digit counts, the groups' (zeroed, one
// set per pass), and with segments the chunks' segments.
struct SortLayout {
  uint32_t *kalt, *valt, *rows, *groups, *chunk_seg;
  size_t group_words;  // of one pass
};
SortLayout carve_sort(Carve& c, uint32_t n, uint32_t M, const SortPlan& P) {
  SortLayout L;
  L.kalt = c.take<uint32_t>(n);
  L.valt = c.take<uint32_t>(n);
  L.rows = c.take<uint32_t>((size_t)P.chunks * kRadix);
  L.group_words = ((size_t)P.chunks / kGroup + 1) * kRadix;
  L.groups = c.take<uint32_t>(kMaxPasses * L.group_words);
  L.chunk_seg = M > 1 ? c.take<uint32_t>(P.chunks) : nullptr;
  return L;
}

template <bool kVals, int kItems, int kBits, int kMode>
rt_status launch_pass_of(const PassArgs& P, uint32_t chunks, cudaStream_t st) {
  constexpr size_t smem = (size_t)kScThreads * kItems * 4 * (kVals ? 2 : 1) + (size_t)kScWarps * (1u << kBits) * 4;
  if (smem + 12 * 1024 > 48 * 1024) {  // above what a launch may use unasked, with the static arrays
    static PerDeviceOnce once;
    if (!once.run([] {
          return cudaFuncSetAttribute(k_sort_scatter<kVals, kItems, kBits, kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem) == cudaSuccess;
        }))
      return RT_ERR_CUDA;
  }
  if (P.rows) k_sort_count<kBits, kMode><<<chunks, kCountThreads, 0, st>>>(P);
  k_sort_scatter<kVals, kItems, kBits, kMode><<<chunks, kScThreads, smem, st>>>(P);
  note_launch(P.rows ? 2 : 1);
  RT_CHECK_LAUNCH();
  return RT_OK;
}
template <bool kVals, int kBits, int kMode>
rt_status launch_pass(const PassArgs& P, const SortPlan& S, cudaStream_t st) {
  if (S.items == 4) return launch_pass_of<kVals, 4, kBits, kMode>(P, S.chunks, st);
  if (S.items == 8) return launch_pass_of<kVals, 8, kBits, kMode>(P, S.chunks, st);
  return launch_pass_of<kVals, 16, kBits, kMode>(P, S.chunks, st);
}

// k_sort_segments over windows of `window` positions; fails where its shared memory is refused.
rt_status launch_segments(uint32_t* codes, uint32_t* idx, uint32_t n, uint32_t* splits, uint32_t* level_counts, uint32_t count_stride,
                          const uint32_t* seg_off, uint32_t M, uint32_t window, cudaStream_t st) {
  static PerDeviceOnce once;
  if (!once.run([] {
        return cudaFuncSetAttribute(k_sort_segments, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSegSmem) == cudaSuccess;
      }))
    return RT_ERR_CUDA;
  k_sort_segments<<<(n - 1) / window + 1, kSegThreads, kSegSmem, st>>>(codes, idx, n, seg_off, M, window, splits, level_counts, count_stride);
  note_launch();
  RT_CHECK_LAUNCH();
  return RT_OK;
}

// Few chunks of one segment: each CTA of a scatter launch counts all the keys for itself, and the count launch and its
// zeroed sums go. 32-bit keys alone: 4097 30.6 -> 19.8 us, 16,384 31.0 -> 24.8, 20,481 32.0 -> 26.7, 30,000 34.1 -> 36.0 (one
// launch per pass with a look-back took 31.2, 33.3, 33.6 and 35.1). The split levels read two codes per key: builds of
// 16,384 faces 153 -> 147 us, of 30,000 163 -> 172 with both.
constexpr uint32_t kSelfCount = 12, kSelfCountLevels = 8;

// The digit passes over chunked keys [0, 8 * passes) from begin_bit; the result is in keys and vals.
rt_status chunked_passes(uint32_t* keys, uint32_t* vals, uint32_t n, uint32_t begin_bit, uint32_t passes, int init_vals, const SortPlan& S,
                         const SortLayout& L, const uint32_t* seg_off, cudaStream_t stream) {
  const bool self_count = !L.chunk_seg && S.chunks <= kSelfCount;
  if (!self_count && cudaMemsetAsync(L.groups, 0, passes * L.group_words * 4, stream) != cudaSuccess) return RT_ERR_CUDA;
  uint32_t *ks = keys, *vs = vals, *kd = L.kalt, *vd = L.valt;
  for (uint32_t p = 0; p < passes; ++p) {
    PassArgs P = {};
    P.keys_in = ks; P.keys_out = kd;
    P.vals_in = (p == 0 && init_vals) ? nullptr : vs; P.vals_out = vd;
    P.n = n; P.shift = begin_bit + 8 * p; P.per_chunk = S.per_chunk; P.short_segs = S.short_segs;
    if (L.chunk_seg) { P.seg_off = seg_off; P.chunk_seg = L.chunk_seg; }
    P.rows = self_count ? nullptr : L.rows; P.groups = L.groups + p * L.group_words;
    const rt_status s = vals ? launch_pass<true, 8, 0>(P, S, stream) : launch_pass<false, 8, 0>(P, S, stream);
    if (s != RT_OK) return s;
    uint32_t* t;
    t = ks; ks = kd; kd = t;
    t = vs; vs = vd; vd = t;
  }
  if (ks != keys) {
    if (cudaMemcpyAsync(keys, ks, (size_t)n * 4, cudaMemcpyDeviceToDevice, stream) != cudaSuccess) return RT_ERR_CUDA;
    if (vals && cudaMemcpyAsync(vals, vs, (size_t)n * 4, cudaMemcpyDeviceToDevice, stream) != cudaSuccess) return RT_ERR_CUDA;
  }
  return RT_OK;
}

}  // namespace

size_t radix_scratch_bytes(uint32_t n) {
  if (n <= (uint32_t)kTile) return 256;
  return radix_scratch_bytes_of(n);
}

size_t segment_sort_scratch_bytes(uint32_t n, uint32_t M) {
  Carve c(nullptr, 0);
  carve_sort(c, n, M, sort_plan(n, M));
  return c.off + 256;
}

rt_status radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t n, uint32_t begin_bit, uint32_t end_bit, int init_vals,
                           void* scratch, size_t scratch_bytes, cudaStream_t stream) {
  if (n == 0) return RT_OK;
  if (end_bit <= begin_bit || end_bit > 32) return RT_ERR_INVALID_ARGUMENT;
  if (n > kMaxKeys) return RT_ERR_INVALID_ARGUMENT;
  const uint32_t passes = (end_bit - begin_bit + 7) / 8;
  if (n <= (uint32_t)kTile) {
    if (!small_smem_ready()) return RT_ERR_CUDA;
    if (vals) k_radix_small<true><<<1, kThreads, kSmallSmem, stream>>>(keys, vals, n, begin_bit, passes, init_vals);
    else k_radix_small<false><<<1, kThreads, kSmallSmem, stream>>>(keys, nullptr, n, begin_bit, passes, 0);
    note_launch();
    RT_CHECK_LAUNCH();
    return RT_OK;
  }
  if (!scratch) return RT_ERR_SCRATCH_TOO_SMALL;
  const SortPlan S = sort_plan(n, 1);
  Carve c(scratch, scratch_bytes);
  const SortLayout L = carve_sort(c, n, 1, S);
  if (!c.ok()) return RT_ERR_SCRATCH_TOO_SMALL;
  return chunked_passes(keys, vals, n, begin_bit, passes, init_vals, S, L, nullptr, stream);
}

rt_status sort_codes_and_levels(uint32_t* codes, uint32_t* idx, uint32_t n, uint32_t* splits, uint32_t* level_counts, uint32_t count_stride,
                                void* scratch, size_t scratch_bytes, cudaStream_t stream, const uint32_t* seg_off, uint32_t M) {
  if (n == 0) return RT_OK;
  if (n > kMaxKeys) return RT_ERR_INVALID_ARGUMENT;
  if (M <= 1) seg_off = nullptr;
  if (n <= (uint32_t)kTile) return launch_segments(codes, idx, n, splits, level_counts, count_stride, seg_off, M, kTile, stream);
  if (!scratch) return RT_ERR_INVALID_ARGUMENT;
  const SortPlan S = sort_plan(n, M);
  Carve c(scratch, scratch_bytes);
  const SortLayout L = carve_sort(c, n, M, S);
  if (!c.ok()) return RT_ERR_SCRATCH_TOO_SMALL;
  if (L.chunk_seg) {
    k_chunk_segs<<<(S.chunks + 255) / 256, 256, 0, stream>>>(seg_off, M, S.per_chunk, S.short_segs, S.chunks, L.chunk_seg);
    note_launch();
    RT_CHECK_LAUNCH();
  }
  rt_status s = chunked_passes(codes, idx, n, 0, 32 / 8, 1, S, L, seg_off, stream);
  if (s != RT_OK) return s;
  // the split levels, from the sorted codes
  const bool self_count = !L.chunk_seg && S.chunks <= kSelfCountLevels;
  if (!self_count && cudaMemsetAsync(L.groups, 0, L.group_words * 4, stream) != cudaSuccess) return RT_ERR_CUDA;
  PassArgs P = {};
  P.keys_in = codes; P.vals_out = splits; P.val_base = 1;
  P.n = n; P.per_chunk = S.per_chunk; P.short_segs = S.short_segs;
  if (L.chunk_seg) { P.seg_off = seg_off; P.chunk_seg = L.chunk_seg; }
  P.rows = self_count ? nullptr : L.rows; P.groups = L.groups; P.totals = level_counts; P.totals_stride = count_stride;
  s = launch_pass<true, 6, 1>(P, S, stream);
  if (s != RT_OK || !S.short_segs) return s;
  return launch_segments(codes, idx, n, splits, level_counts, count_stride, seg_off, M, kSegWindow, stream);
}

}  // namespace rt

using namespace rt;

extern "C" rt_status rt_sort_scratch_bytes(uint32_t n, size_t* bytes) {
  if (!bytes) return RT_ERR_INVALID_ARGUMENT;
  *bytes = radix_scratch_bytes(n);
  return RT_OK;
}

static uint32_t bits_of(uint32_t bit_depth) {
  uint32_t bytes = bit_depth == 0 ? 1 : 1 + (bit_depth - 1) / 8;
  return 8 * (bytes > 4 ? 4 : bytes);
}

extern "C" rt_status rt_radix_sort_pairs(uint32_t* keys, uint32_t* values, uint32_t n, uint32_t bit_depth, int init_values,
                                         void* scratch, size_t scratch_bytes, rt_stream stream) {
  const rt::NvtxRange nvtx_range("rt_radix_sort_pairs");
  if (n && (!keys || !values)) return RT_ERR_INVALID_ARGUMENT;
  if (n > (uint32_t)kTile && (!scratch || scratch_bytes < radix_scratch_bytes(n))) return RT_ERR_SCRATCH_TOO_SMALL;
  if (rt_device_check() != RT_OK) return RT_ERR_NO_DEVICE;
  if (n == 1 && init_values) {
    k_iota<<<1, 32, 0, (cudaStream_t)stream>>>(values, 1);
    note_launch();
    RT_CHECK_LAUNCH();
    return RT_OK;
  }
  return radix_sort_pairs(keys, values, n, 0, bits_of(bit_depth), init_values, scratch, scratch_bytes, (cudaStream_t)stream);
}

extern "C" rt_status rt_radix_sort_keys(uint32_t* keys, uint32_t n, uint32_t bit_depth, void* scratch, size_t scratch_bytes, rt_stream stream) {
  if (n && !keys) return RT_ERR_INVALID_ARGUMENT;
  if (n > (uint32_t)kTile && (!scratch || scratch_bytes < radix_scratch_bytes(n))) return RT_ERR_SCRATCH_TOO_SMALL;
  if (rt_device_check() != RT_OK) return RT_ERR_NO_DEVICE;
  return radix_sort_pairs(keys, nullptr, n, 0, bits_of(bit_depth), 0, scratch, scratch_bytes, (cudaStream_t)stream);
}
