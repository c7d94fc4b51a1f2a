// rt_clusters.cu -- the cluster tree of the traversal blob (layout in rt_device.cuh).
//
// The node tree of an LBVH build stops at the build's tree depth (12 levels
// by default), so its leaves hold about N / 4096 triangles each: a quarter of
// a million triangles per mesh gives leaves of ~100 triangles, which a walk
// tests in 8-triangle groups. The cluster tree is a second, independent
// traversal tree over the same positions that goes down to leaf_max (4)
// triangles per leaf. Hits never depend on it: the closest hit is the minimum
// (t, position) over all triangles whatever tree prunes the search.
//
// Construction: the binary radix tree of the keys (Morton code << 32 |
// position), which are distinct and sorted, built bottom-up by the
// agglomerative scheme of Apetrei (Fast and Simple Agglomerative LBVH
// Construction, 2014): the boundary between positions b and b + 1 carries the
// value key(b) xor key(b + 1); a node covering positions l .. r merges with the
// neighbour across the flanking boundary of smaller value, and that boundary is
// the index of the parent (the internal node splitting between b and b + 1).
// One thread starts at each position and climbs; at each parent the first of
// the two children to arrive leaves (an atomic exchange on the parent's word
// hands over its far end of the range), the second completes the parent
// (box, 4-wide record) and climbs on, so no thread ever waits.
//
// Three launches keep almost all of that in shared memory:
//   k_cluster_chunk     one CTA per chunk of 512 positions of one mesh: the
//                       climb through the parents whose boundary lies inside
//                       the chunk, in rounds over a compacted list of the
//                       nodes moving up, with shared-memory arrival words,
//                       child references and boxes (every node completed here
//                       has both children inside the chunk), then the records
//                       of those nodes. A node whose parent boundary lies
//                       outside the chunk (at most one per side) is left in the
//                       chunk's frontier; the CTA writes all its arrival words
//                       and, for the next passes, the few nodes they read.
//   k_cluster_frontier  one thread per frontier node: the rest of the climb
//                       through global memory; an arriving child stores its
//                       reference and box in its side of the parent's slots,
//                       then exchanges the parent's word (acquire-release), so
//                       the second arrival reads the sibling's box at once.
//   k_cluster_records   the records of the nodes the frontier pass completed
//                       (each frontier thread lists the nodes it completed).
#include <cuda/atomic>

#include "rt_common.cuh"
#include "rt_device.cuh"

namespace rt {
namespace {

struct ClusterBuild {
  const float4* tris;    // {v0, e1, e2} per position, all meshes
  const uint32_t* codes; // sorted Morton codes per position (mesh-local order)
  const uint32_t* foff;  // batched: face offsets (M + 1 entries); single mesh: nullptr
  uint32_t M;            // meshes (1 for a single mesh)
  uint32_t N;            // positions, all meshes
  uint32_t leaf_max;     // largest cluster
  ClusterTemps T;
  uint32_t* hdr;         // header words, 64 per mesh
  float4* crec;          // records, all meshes
};

// Mesh m of chunk b (for which the warp's first chunk is `first`): its face offset, face count and b's index j among
// its chunks. The warp finds the mesh of `first` together, 32 meshes at a step; a lane whose chunk is later goes on
// from there (the lanes of a warp hold consecutive chunks).
__device__ __forceinline__ void mesh_of_chunk(const ClusterBuild& B, uint32_t first, uint32_t b, uint32_t& m, uint32_t& F, uint32_t& n,
                                              uint32_t& j) {
  if (!B.foff) {
    m = 0; F = 0; n = B.N; j = b;
    return;
  }
  uint32_t lo = 0, len = B.M;  // largest m with cluster_chunk_base(F_m, m) <= first
  while (len > 1) {
    const uint32_t step = (len + 31) / 32, at = lane_id() * step;
    const uint32_t c = (uint32_t)__popc(__ballot_sync(0xffffffffu, at < len && cluster_chunk_base(__ldg(B.foff + lo + at), lo + at) <= first)) - 1u;
    lo += c * step;
    len = min(step, len - c * step);
  }
  m = lo;
  while (m + 1 < B.M && cluster_chunk_base(__ldg(B.foff + m + 1), m + 1) <= b) ++m;
  F = __ldg(B.foff + m);
  n = __ldg(B.foff + m + 1) - F;
  j = b - cluster_chunk_base(F, m);
}

// The value of the boundary between positions pos - 1 and pos of a mesh's n codes, as its level: the number of leading
// bits that the two keys share, -1 at the mesh's ends. The two boundaries that flank a node differ in it, since sorted
// keys that agree up to a bit change there once, and the smaller value is the one with the higher level.
__device__ __forceinline__ int level_before(const uint32_t* __restrict__ codes, uint32_t n, uint32_t pos) {
  if (pos == 0 || pos >= n) return -1;
  const uint32_t x = __ldg(codes + pos - 1) ^ __ldg(codes + pos);
  return x ? __clz(x) : 32 + __clz((pos - 1) ^ pos);
}

__device__ __forceinline__ void tri_box(const float4* tr, float3& mn, float3& mx) {
  const float4 v0 = ldg4(tr), e1 = ldg4(tr + 1), e2 = ldg4(tr + 2);
  const float ax = __fadd_rn(v0.x, e1.x), ay = __fadd_rn(v0.y, e1.y), az = __fadd_rn(v0.z, e1.z);
  const float bx = __fadd_rn(v0.x, e2.x), by = __fadd_rn(v0.y, e2.y), bz = __fadd_rn(v0.z, e2.z);
  mn = make_float3(fminf(v0.x, fminf(ax, bx)), fminf(v0.y, fminf(ay, by)), fminf(v0.z, fminf(az, bz)));
  mx = make_float3(fmaxf(v0.x, fmaxf(ax, bx)), fmaxf(v0.y, fmaxf(ay, by)), fmaxf(v0.z, fmaxf(az, bz)));
  pad_box(mn, mx);
}

// One slot pair of a completed internal node's 4-wide record: the child of positions lo .. hi with reference c, whose own
// children (if any) are c0 and c1. A child that is a cluster (at most leaf_max positions) takes the first slot (the second
// keeps NaN bounds), any other child one slot for each of its two children (c, its index, is its split). The slots' boxes are
// the child's, or its children's.
struct SlotPair {
  uint32_t ref0, ref1;
};
__device__ __forceinline__ SlotPair slot_pair(uint32_t leaf_max, uint32_t lo, uint32_t hi, uint32_t c, uint32_t c0, uint32_t c1) {
  if (hi - lo + 1 <= leaf_max) return SlotPair{cluster_leaf_ref(lo, hi - lo + 1), kNoChild};
  return SlotPair{(c - lo + 1 <= leaf_max) ? cluster_leaf_ref(lo, c - lo + 1) : c0,
                  (hi - c <= leaf_max) ? cluster_leaf_ref(c + 1, hi - c) : c1};
}

// The record of node p (positions l .. r) from the global child references and boxes.
__device__ __forceinline__ void write_record(const ClusterBuild& B, uint32_t F, uint32_t p, uint32_t l, uint32_t r) {
  const float qnan = __int_as_float(0x7fffffff);
  float3 mn[4], mx[4];
  uint32_t ref[4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t lo = h ? p + 1 : l, hi = h ? r : p;
    const uint32_t c = __ldcg(B.T.child + 2 * ((size_t)F + p) + h);
    const bool leaf = hi - lo + 1 <= B.leaf_max;
    const uint2 kid = leaf ? make_uint2(0, 0) : __ldcg((const uint2*)(B.T.child + 2 * ((size_t)F + c)));
    const SlotPair S = slot_pair(B.leaf_max, lo, hi, c, kid.x, kid.y);
    ref[2 * h] = S.ref0;
    ref[2 * h + 1] = S.ref1;
    const float4* q = B.T.cbox + 4 * ((size_t)F + (leaf ? p : c)) + (leaf ? 2 * h : 0);
    const float4 a = __ldcg(q), b = __ldcg(q + 1);
    mn[2 * h] = make_float3(a.x, a.y, a.z);
    mx[2 * h] = make_float3(b.x, b.y, b.z);
    mn[2 * h + 1] = mx[2 * h + 1] = make_float3(qnan, qnan, qnan);
    if (!leaf) {
      const float4 u = __ldcg(q + 2), v = __ldcg(q + 3);
      mn[2 * h + 1] = make_float3(u.x, u.y, u.z);
      mx[2 * h + 1] = make_float3(v.x, v.y, v.z);
    }
  }
  float4* rec = B.crec + 8 * ((size_t)F + p);
  rec[0] = make_float4(mn[0].x, mn[1].x, mn[2].x, mn[3].x);
  rec[1] = make_float4(mn[0].y, mn[1].y, mn[2].y, mn[3].y);
  rec[2] = make_float4(mn[0].z, mn[1].z, mn[2].z, mn[3].z);
  rec[3] = make_float4(mx[0].x, mx[1].x, mx[2].x, mx[3].x);
  rec[4] = make_float4(mx[0].y, mx[1].y, mx[2].y, mx[3].y);
  rec[5] = make_float4(mx[0].z, mx[1].z, mx[2].z, mx[3].z);
  rec[6] = make_float4(__uint_as_float(ref[0]), __uint_as_float(ref[1]), __uint_as_float(ref[2]), __uint_as_float(ref[3]));
  rec[7] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// The root (positions 0 .. n - 1, box mn / mx, reference cur) is complete: header words, and a one-slot record
// at index n - 1 when the whole mesh is one cluster.
__device__ __forceinline__ void finish_root(const ClusterBuild& B, uint32_t m, uint32_t F, uint32_t n, uint32_t cur, const float3& mn,
                                            const float3& mx) {
  uint32_t root = cur;
  if (n <= B.leaf_max) {
    const float qnan = __int_as_float(0x7fffffff);
    float4* rec = B.crec + 8 * ((size_t)F + n - 1);
    rec[0] = make_float4(mn.x, qnan, qnan, qnan);
    rec[1] = make_float4(mn.y, qnan, qnan, qnan);
    rec[2] = make_float4(mn.z, qnan, qnan, qnan);
    rec[3] = make_float4(mx.x, qnan, qnan, qnan);
    rec[4] = make_float4(mx.y, qnan, qnan, qnan);
    rec[5] = make_float4(mx.z, qnan, qnan, qnan);
    rec[6] = make_float4(__uint_as_float(cluster_leaf_ref(0, n)), __uint_as_float(kNoChild), __uint_as_float(kNoChild),
                         __uint_as_float(kNoChild));
    rec[7] = make_float4(0.f, 0.f, 0.f, 0.f);
    root = n - 1;
  }
  uint32_t* hdr = B.hdr + 64 * (size_t)m;
  hdr[kHdrClusterN] = n;
  hdr[kHdrClusterRoot] = root;
  __threadfence();
  hdr[kHdrClusterValid] = 1u;
}

// A node moving up: reference, first and last position, box.
struct ChunkNode {
  uint32_t cur, l, r;
  float3 mn, mx;
};

// Shared memory of the chunk pass. A box is two float4 (a node read is two 16-byte loads; six arrays of floats cost three
// times the wavefronts), whose w words hold an inner node's first and last position (last 0: not complete).
struct ChunkShared {
  float4 box[2 * kClusterChunk][2];  // inner nodes (by boundary), then positions
  uint2 child[kClusterChunk];
  uint32_t other[kClusterChunk];     // arrival words
  int level[kClusterChunk + 1];      // of boundaries s - 1 .. s + 511
  alignas(16) uint32_t list[3][kClusterChunk];  // round r reads list r % 3 and fills list (r + 1) % 3
  uint32_t count[3];
  uint32_t records;

  // index in box of node ref of the chunk that starts at position s
  static __device__ __forceinline__ uint32_t at(uint32_t ref, uint32_t s) { return (ref & ~kClusterLeaf) - s + ((ref & kClusterLeaf) ? kClusterChunk : 0u); }
  __device__ __forceinline__ ChunkNode node(uint32_t ref, uint32_t s) const {
    const float4 a = box[at(ref, s)][0], b = box[at(ref, s)][1];
    const bool leaf = (ref & kClusterLeaf) != 0;
    const uint32_t pos = ref & ~kClusterLeaf;
    return ChunkNode{ref, leaf ? pos : __float_as_uint(a.w), leaf ? pos : __float_as_uint(b.w), make_float3(a.x, a.y, a.z), make_float3(b.x, b.y, b.z)};
  }
};

// One step of node c up: true if it arrived second at its parent, which is then complete and replaces it. False: the
// sibling completes the parent, or the climb leaves the chunk (positions s .. e), or c is the root.
__device__ __forceinline__ bool chunk_climb(const ClusterBuild& B, ChunkShared& S, uint32_t s, uint32_t e, uint32_t m, uint32_t F, uint32_t n,
                                            ChunkNode& c) {
  const int level_l = S.level[c.l - s], level_r = S.level[c.r + 1 - s];
  if (max(level_l, level_r) < 0) {
    finish_root(B, m, F, n, c.cur, c.mn, c.mx);
    return false;
  }
  const bool left_child = level_r > level_l;
  const uint32_t p = left_child ? c.r : c.l - 1;
  if (p < s || p >= e) {  // the parent's boundary is not inside the chunk: the frontier pass goes on from here
    B.T.frontier[2 * (size_t)blockIdx.x + (p < s ? 0 : 1)] = make_uint4(c.cur, c.l, c.r, 1u);
    return false;
  }
  const uint32_t k = p - s;
  (left_child ? S.child[k].x : S.child[k].y) = c.cur;
  __threadfence_block();
  const uint32_t old = atomicExch(S.other + k, (left_child ? c.l : c.r) + 1u);
  if (old == 0) return false;
  __threadfence_block();
  if (left_child) c.r = old - 1u; else c.l = old - 1u;
  const uint32_t sib = S.at(left_child ? S.child[k].y : S.child[k].x, s);
  const float4 a = S.box[sib][0], b = S.box[sib][1];
  c.mn = make_float3(fminf(c.mn.x, a.x), fminf(c.mn.y, a.y), fminf(c.mn.z, a.z));
  c.mx = make_float3(fmaxf(c.mx.x, b.x), fmaxf(c.mx.y, b.y), fmaxf(c.mx.z, b.z));
  c.cur = p;
  S.box[k][0] = make_float4(c.mn.x, c.mn.y, c.mn.z, __uint_as_float(c.l));
  S.box[k][1] = make_float4(c.mx.x, c.mx.y, c.mx.z, __uint_as_float(c.r));
  return true;
}

// The slot pair of a record's child (positions lo .. hi, reference c) and its boxes' indices.
constexpr uint32_t kNoBox = 0xffffu;
__device__ __forceinline__ SlotPair chunk_pair(uint32_t leaf_max, const ChunkShared& S, uint32_t s, uint32_t lo, uint32_t hi, uint32_t c,
                                               uint32_t& src) {
  uint2 kid = make_uint2(0, 0);
  if (hi - lo + 1 <= leaf_max) {
    src = S.at(c, s) | kNoBox << 16;
  } else {
    kid = S.child[c - s];
    src = S.at(kid.x, s) | S.at(kid.y, s) << 16;
  }
  return slot_pair(leaf_max, lo, hi, c, kid.x, kid.y);
}

// The chunk pass climbs in rounds: the nodes to move up (all positions first) sit in a compacted shared-memory
// list; in a round every listed node arrives at its parent, and the second arrival at a parent completes it
// (range and box, in shared memory) and lists it for the next round, so the threads of a warp work on listed
// nodes side by side. Once a warp can hold what is listed, the first warp climbs on alone, a node per lane and without
// barriers. Then the CTA writes every inner boundary's arrival word and the records of the nodes completed here: a thread
// per record works out its references and which boxes it holds, then the threads take its six 16-byte parts of box
// bounds one by one, so that neighbouring lanes store neighbouring bytes and read a box's neighbouring words. (A thread
// per whole record stored 16 bytes in each of 32 lines at a time and, with every round between barriers, took
// 87 us for 2^20 faces and 769 for 9.9M in 1024 meshes; now 63 and
// 544, by issue slots and the latency of the rounds.)
__global__ __launch_bounds__(kClusterChunk, 4) void k_cluster_chunk(ClusterBuild B) {
  __shared__ ChunkShared S;
  const uint32_t t = threadIdx.x, lane = t & 31u;
  uint32_t m, F, n, j;
  mesh_of_chunk(B, blockIdx.x, blockIdx.x, m, F, n, j);
  const uint32_t s = j * kClusterChunk;
  if (t < 2) B.T.frontier[2 * (size_t)blockIdx.x + t] = make_uint4(0, 0, 0, 0);
  if (s >= n) return;  // a gap in the batched grid (the whole CTA)
  const uint32_t e = min(n, s + kClusterChunk) - 1;  // the chunk's last position; inner boundaries s .. e - 1
  S.other[t] = 0;
  S.box[t][1].w = 0.f;
  const uint32_t i = s + t;
  S.level[t] = level_before(B.codes + F, n, i);
  if (t == 0) S.level[kClusterChunk] = level_before(B.codes + F, n, s + kClusterChunk);
  ChunkNode c;
  if (i <= e) {
    c.cur = kClusterLeaf | i;
    c.l = c.r = i;
    tri_box(B.tris + 3 * ((size_t)F + i), c.mn, c.mx);
    S.box[kClusterChunk + t][0] = make_float4(c.mn.x, c.mn.y, c.mn.z, 0.f);
    S.box[kClusterChunk + t][1] = make_float4(c.mx.x, c.mx.y, c.mx.z, 0.f);
  }
  if (t < 3) S.count[t] = 0;
  if (t == 3) S.records = 0;
  __syncthreads();
  uint32_t count = e - s + 1, round = 0;
  for (;; ++round) {
    // one barrier per round: the list after next (read two rounds ago) is emptied during this round
    const uint32_t cb = round % 3u, nb = (round + 1u) % 3u;
    if (round) {
      count = S.count[cb];
      if (count <= 32) break;
      if (t < count) c = S.node(S.list[cb][t], s);
    }
    const bool up = t < count && chunk_climb(B, S, s, e, m, F, n, c);
    // append to the next list, one shared-memory atomic per warp
    const uint32_t who = __ballot_sync(0xffffffffu, up);
    if (who) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(S.count + nb, (uint32_t)__popc(who));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (up) S.list[nb][base + __popc(who & ((1u << lane) - 1u))] = c.cur;
    }
    if (t == 0) S.count[(round + 2u) % 3u] = 0;
    __syncthreads();
  }
  if (t < 32) {
    bool up = t < count;
    if (up) c = S.node(S.list[round % 3u][t], s);
    while (__any_sync(0xffffffffu, up)) {
      if (up) up = chunk_climb(B, S, s, e, m, F, n, c);
      __syncwarp();
    }
  }
  __syncthreads();
  // Write-out. Every boundary's arrival word (coalesced; e's is zero: its children are never both inside one chunk),
  // the record of each node completed here with more than leaf_max positions, and
  // for the global pass and its records the nodes they read: the frontier nodes and the first child to arrive at
  // each parent still pending, each with its box and, when internal, its child references and their boxes.
  auto put_box = [&](float4* dst, uint32_t ref) {
    const float4 a = S.box[S.at(ref, s)][0], b = S.box[S.at(ref, s)][1];
    dst[0] = make_float4(a.x, a.y, a.z, 0.f);
    dst[1] = make_float4(b.x, b.y, b.z, 0.f);
  };
  auto export_kids = [&](uint32_t ref) {
    if (ref & kClusterLeaf) return;
    const uint2 k = S.child[ref - s];
    *(uint2*)(B.T.child + 2 * ((size_t)F + ref)) = k;
    put_box(B.T.cbox + 4 * ((size_t)F + ref), k.x);
    put_box(B.T.cbox + 4 * ((size_t)F + ref) + 2, k.y);
  };
  bool record = false;
  uint2 src;  // the record's four boxes (16-bit indices into box, kNoBox: none)
  if (i < e) {
    const uint32_t word = S.other[t];
    B.T.other[(size_t)F + i] = word;
    const uint32_t l = __float_as_uint(S.box[t][0].w), r = __float_as_uint(S.box[t][1].w);
    if (r != 0) {
      record = r - l + 1 > B.leaf_max;
    } else if (word != 0) {  // one child arrived: a left child stored its first position (<= i), a right one its last
      const uint32_t side = (word - 1u <= i) ? 0u : 1u;
      const uint32_t ch = side ? S.child[t].y : S.child[t].x;
      B.T.child[2 * ((size_t)F + i) + side] = ch;
      put_box(B.T.cbox + 4 * ((size_t)F + i) + 2 * side, ch);
      export_kids(ch);
    }
    if (record) {  // the references and the zeros (the record's last 32 bytes)
      float4* rec = B.crec + 8 * ((size_t)F + i);
      const uint2 ch = S.child[t];
      const SlotPair L = chunk_pair(B.leaf_max, S, s, l, i, ch.x, src.x), R = chunk_pair(B.leaf_max, S, s, i + 1, r, ch.y, src.y);
      rec[6] = make_float4(__uint_as_float(L.ref0), __uint_as_float(L.ref1), __uint_as_float(R.ref0), __uint_as_float(R.ref1));
      rec[7] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else if (i == e && i + 1 < n) {
    B.T.other[(size_t)F + i] = 0u;
  }
  if (t < 2) {
    const uint4 fr = B.T.frontier[2 * (size_t)blockIdx.x + t];
    if (fr.w) {
      put_box(B.T.fbox + 4 * (size_t)blockIdx.x + 2 * t, fr.x);
      export_kids(fr.x);
    }
  }
  const uint32_t who = __ballot_sync(0xffffffffu, record);
  uint32_t base = 0;
  if (lane == 0 && who) base = atomicAdd(&S.records, (uint32_t)__popc(who));
  base = __shfl_sync(0xffffffffu, base, 0);
  uint2* s_src = (uint2*)S.list[0];
  if (record) {
    const uint32_t q = base + __popc(who & ((1u << lane) - 1u));
    s_src[q] = src;
    S.list[2][q] = i;
  }
  __syncthreads();
  const float* box = (const float*)S.box;
  const float qnan = __int_as_float(0x7fffffff);
  const uint32_t parts = 6 * S.records;
  for (uint32_t q = t; q < parts; q += kClusterChunk) {
    const uint32_t k = q / 6u, part = q - 6u * k;
    const float* b = box + part + (part >= 3 ? 1u : 0u);
    const uint2 x = s_src[k];
    const uint32_t x1 = x.x >> 16, x3 = x.y >> 16;
    B.crec[8 * ((size_t)F + S.list[2][k]) + part] = make_float4(b[8 * (x.x & 0xffffu)], x1 == kNoBox ? qnan : b[8 * x1], b[8 * (x.y & 0xffffu)],
                                                                x3 == kNoBox ? qnan : b[8 * x3]);
  }
}

// The rest of the climb, from the frontier nodes, through global memory. Each arriving child stores its
// reference and box in its side of the parent's slots, then exchanges the parent's arrival word with
// acquire-release order at device scope; the second arrival reads the sibling's box, completes the parent and
// marks it (its range) for k_cluster_records.
__global__ __launch_bounds__(128) void k_cluster_frontier(ClusterBuild B) {
  const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x, nodes = 2 * cluster_chunks(B.N, B.M);
  if ((f & ~31u) >= nodes) return;
  uint4 fr = make_uint4(0, 0, 0, 0);
  if (f < nodes) fr = B.T.frontier[f];
  uint32_t m, F, n, j;
  mesh_of_chunk(B, (f & ~31u) >> 1, f >> 1, m, F, n, j);
  if (fr.w == 0) {
    if (f < nodes) B.T.chain[(size_t)f * (kClusterChain + 1) + kClusterChain] = 0;
    return;
  }
  const uint32_t* codes = B.codes + F;
  uint32_t cur = fr.x, l = fr.y, r = fr.z;
  const float4 b0 = B.T.fbox[2 * (size_t)f], b1 = B.T.fbox[2 * (size_t)f + 1];
  float3 mn = make_float3(b0.x, b0.y, b0.z), mx = make_float3(b1.x, b1.y, b1.z);
  uint32_t* chain = B.T.chain + (size_t)f * (kClusterChain + 1);
  uint32_t done = 0;  // nodes completed by this climb (listed in chain for k_cluster_records)
  int level_l = level_before(codes, n, l), level_r = level_before(codes, n, r + 1);
  for (;;) {
    if (max(level_l, level_r) < 0) {
      finish_root(B, m, F, n, cur, mn, mx);
      break;
    }
    const bool left_child = level_r > level_l;
    const uint32_t p = left_child ? r : l - 1;
    const uint32_t side = left_child ? 0u : 1u;
    float4* slot = B.T.cbox + 4 * ((size_t)F + p);
    B.T.child[2 * ((size_t)F + p) + side] = cur;
    slot[2 * side] = make_float4(mn.x, mn.y, mn.z, 0.f);
    slot[2 * side + 1] = make_float4(mx.x, mx.y, mx.z, 0.f);
    cuda::atomic_ref<uint32_t, cuda::thread_scope_device> word(B.T.other[(size_t)F + p]);
    const uint32_t old = word.exchange((left_child ? l : r) + 1u, cuda::memory_order_acq_rel);
    if (old == 0) break;  // the sibling completes the parent
    // the new flank's codes and the sibling's box come with one latency
    if (left_child) r = old - 1u; else l = old - 1u;
    const int level = level_before(codes, n, left_child ? r + 1 : l);
    const float4 s0 = __ldcg(slot + 2 * (1 - side)), s1 = __ldcg(slot + 2 * (1 - side) + 1);
    mn = make_float3(fminf(mn.x, s0.x), fminf(mn.y, s0.y), fminf(mn.z, s0.z));
    mx = make_float3(fmaxf(mx.x, s1.x), fmaxf(mx.y, s1.y), fmaxf(mx.z, s1.z));
    B.T.prange[(size_t)F + p] = make_uint2(l, r + 1u);
    if (done < kClusterChain) chain[done++] = p;
    cur = p;
    (left_child ? level_r : level_l) = level;
  }
  chain[kClusterChain] = done;
}

// Records of the nodes the frontier pass completed: one warp per frontier node, a lane per node of its climb.
__global__ __launch_bounds__(256) void k_cluster_records(ClusterBuild B) {
  const uint32_t f = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
  if (f >= 2 * cluster_chunks(B.N, B.M)) return;
  const uint32_t* chain = B.T.chain + (size_t)f * (kClusterChain + 1);
  const uint32_t done = chain[kClusterChain];
  if (done == 0) return;
  uint32_t m, F, n, j;
  mesh_of_chunk(B, f >> 1, f >> 1, m, F, n, j);
  for (uint32_t k = lane; k < done; k += 32) {
    const uint32_t p = chain[k];
    const uint2 pr = B.T.prange[(size_t)F + p];
    const uint32_t l = pr.x, r = pr.y - 1u;
    if (r - l + 1 > B.leaf_max) write_record(B, F, p, l, r);
  }
}

}  // namespace

rt_status build_cluster_tree(const float4* tris, const uint32_t* codes, uint32_t n, uint32_t leaf_max, const ClusterTemps& T,
                             uint32_t* hdr, float4* crec, cudaStream_t st) {
  return batch_build_cluster_tree(tris, codes, nullptr, 1, n, leaf_max, T, hdr, crec, st);
}

rt_status batch_build_cluster_tree(const float4* tris, const uint32_t* codes, const uint32_t* foff, uint32_t M, uint32_t N,
                                   uint32_t leaf_max, const ClusterTemps& T, uint32_t* hdr, float4* crec, cudaStream_t st) {
  if (N == 0) return RT_OK;
  if (N > kClusterFirstMask || leaf_max < 1 || leaf_max > kClusterLeafMax) return RT_ERR_UNSUPPORTED;
  ClusterBuild B;
  B.tris = tris; B.codes = codes; B.foff = foff; B.M = M; B.N = N; B.leaf_max = leaf_max; B.T = T; B.hdr = hdr; B.crec = crec;
  const uint32_t chunks = cluster_chunks(N, M);
  k_cluster_chunk<<<chunks, kClusterChunk, 0, st>>>(B);
  k_cluster_frontier<<<(2 * chunks + 127) / 128, 128, 0, st>>>(B);
  k_cluster_records<<<(2 * chunks * 32 + 255) / 256, 256, 0, st>>>(B);
  note_launch(3);
  RT_CHECK_LAUNCH();
  return RT_OK;
}

}  // namespace rt
