// rt_build.cu -- LBVH build for sm_100a.
//
// Replaces CUDA_buildMeshTreeLBVH (kernels/CUDA_buildMeshTreeLBVH.cu:457-681)
// and its helpers. The reference runs ~10 launches with a host sync after
// each, copies the split list to the host, builds the topology with a
// sequential host recursion (:309-455), copies the nodes back, then runs
// real_depth full passes for the boxes. Here everything stays on the device,
// with no host round trip:
//
//   k_boxes_morton   per face: box (4-wide min/max of the 3 vertices),
//                    Morton code (reference 11/11/10 layout or 10/10/10)
//   radix sort       (code, index) pairs, stable (rt_sort.cu)
//   level sort       split positions by split level (clz of the xor of adjacent
//                    codes, computed as the pass reads them): the per-level
//                    ascending split lists the recursion walks
//   k_topo_morton    one CTA: the Morton levels of the tree, level by level in
//                    shared memory, with the reference's split-pointer semantics (see below);
//                    leaf counts, pre-order ranks and node ids
//   k_leaves         32 final leaves at a time per warp: expands median subtrees, writes
//                    node records, reorders faces, pre-gathers triangles
//                    {v0, e1, e2}, reduces the leaf box and records the
//                    parents of median nodes
//   k_propagate      one thread per node: each leaf climbs to the root with
//                    per-node arrival counters (the second arrival merges the
//                    two child boxes; nobody waits)
//
// Node numbering follows the reference's recursion: the k-th internal node in
// pre-order gets children 2k+1 and 2k+2. A node's pre-order rank among
// internal nodes is computed from subtree leaf counts (rank(left) = rank + 1,
// rank(right) = rank + leaves(left)).
//
// Split-pointer semantics (host recursion :360-411): each level L keeps a
// pointer into the concatenated, level-ordered split list C. A Morton visit of
// a range [a, b) at level L (b - a >= min_leaf, L < tree_depth) is a leaf when
// the pointer sits exactly at the start of level L+1's list; otherwise the
// pointer advances past every entry <= a -- it may run into deeper levels'
// lists -- and the entry found cuts the range if it is < b. Because visits at a
// level come in increasing a, the pointer after a visit is "the first index at
// or after start(L) holding a value > a"; it sticks at start(L+1) exactly when
// the first visit with a >= last(P_L) finds C[start(L+1)] > a. Both facts make
// every visit of a level independent once that one visit is known.
#include "rt_device.cuh"

namespace rt {
namespace {

constexpr int kTopoThreads = 1024;      // of the one CTA of a single build
constexpr int kBatchTopoThreads = 512;  // of a mesh's CTA of a batched build

// ----------------------------------------------------------------------------
// hit box (when the caller gives none): min/max over all vertices
// ----------------------------------------------------------------------------
__global__ void k_set_hitbox(float4* hit, float4 mn, float4 mx) {
  hit[0] = mn;
  hit[1] = mx;
}

// Hit box over all vertices: each block reduces its grid-stride share to a partial box; the block that finishes
// last (a counter the host zeroes) combines the partials, strided over its threads and then as a shared-memory
// tree, and writes hit[0..1]. Nothing waits for it inside the launch.
__global__ __launch_bounds__(256) void k_hitbox(const float4* __restrict__ v, uint32_t count, float4* __restrict__ partial,
                                               uint32_t* __restrict__ done, float4* __restrict__ hit) {
  // four loads in flight per thread, one accumulator each
  float4 mn[4], mx[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    mn[k] = make_float4(kHuge, kHuge, kHuge, kHuge);
    mx[k] = make_float4(-kHuge, -kHuge, -kHuge, -kHuge);
  }
  const uint32_t stride = gridDim.x * blockDim.x;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  for (; (uint64_t)i + 3ull * stride < count; i += 4 * stride) {
    float4 p[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) p[k] = ldg4(v + i + k * stride);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mn[k] = f4min(mn[k], p[k]);
      mx[k] = f4max(mx[k], p[k]);
    }
  }
  for (; i < count; i += stride) {
    const float4 p = ldg4(v + i);
    mn[0] = f4min(mn[0], p);
    mx[0] = f4max(mx[0], p);
  }
  __shared__ float4 s_mn[256], s_mx[256];
  __shared__ uint32_t s_last;
  s_mn[threadIdx.x] = f4min(f4min(mn[0], mn[1]), f4min(mn[2], mn[3]));
  s_mx[threadIdx.x] = f4max(f4max(mx[0], mx[1]), f4max(mx[2], mx[3]));
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      s_mn[threadIdx.x] = f4min(s_mn[threadIdx.x], s_mn[threadIdx.x + o]);
      s_mx[threadIdx.x] = f4max(s_mx[threadIdx.x], s_mx[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = s_mn[0];
    partial[2 * blockIdx.x + 1] = s_mx[0];
    __threadfence();
    s_last = atomicAdd(done, 1u) == gridDim.x - 1 ? 1u : 0u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  float4 a = make_float4(kHuge, kHuge, kHuge, kHuge), b = make_float4(-kHuge, -kHuge, -kHuge, -kHuge);
  for (uint32_t j = threadIdx.x; j < gridDim.x; j += blockDim.x) {
    a = f4min(a, __ldcg(partial + 2 * j));
    b = f4max(b, __ldcg(partial + 2 * j + 1));
  }
  s_mn[threadIdx.x] = a;
  s_mx[threadIdx.x] = b;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      s_mn[threadIdx.x] = f4min(s_mn[threadIdx.x], s_mn[threadIdx.x + o]);
      s_mx[threadIdx.x] = f4max(s_mx[threadIdx.x], s_mx[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    hit[0] = s_mn[0];
    hit[1] = s_mx[0];
  }
}

// ----------------------------------------------------------------------------
// boxes + Morton + iota
// ----------------------------------------------------------------------------
// kernels/CUDA_calcMeshBoxes.cu:30-58 (boxes, iota) fused with
// kernels/CUDA_buildMeshTreeLBVH.cu:115-173 (Morton code of the box centre).
__global__ __launch_bounds__(256) void k_boxes_morton(const float4* __restrict__ verts, const uint4* __restrict__ faces, uint32_t n,
                                                     const float4* __restrict__ hit, int layout, float4* __restrict__ boxes,
                                                     uint32_t* __restrict__ codes, uint32_t* __restrict__ idx) {
  const float4 hmin = codes ? hit[0] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 hmax = codes ? hit[1] : make_float4(1.f, 1.f, 1.f, 1.f);
  const float lx = hmax.x - hmin.x, ly = hmax.y - hmin.y, lz = hmax.z - hmin.z;
  const float sx = (layout == 30 ? 1023.0f : 2047.0f) / lx;
  const float sy = (layout == 30 ? 1023.0f : 2047.0f) / ly;
  const float sz = 1023.0f / lz;
  auto face = [&](uint32_t k, const float4& v0, const float4& v1, const float4& v2) {
    const float4 mn = f4min(f4min(v0, v1), v2);
    const float4 mx = f4max(f4max(v0, v1), v2);
    boxes[2 * (size_t)k] = mn;
    boxes[2 * (size_t)k + 1] = mx;
    if (idx) idx[k] = k;
    if (codes) {
      const float cx = 0.5f * (mn.x + mx.x), cy = 0.5f * (mn.y + mx.y), cz = 0.5f * (mn.z + mx.z);
      const uint32_t qx = f2u_sat((cx - hmin.x) * sx);
      const uint32_t qy = f2u_sat((cy - hmin.y) * sy);
      const uint32_t qz = f2u_sat((cz - hmin.z) * sz);
      codes[k] = spread_code(qx, qy, qz, layout);
    }
  };
  // two faces per iteration: their face and vertex loads are in flight together
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += 2 * stride) {
    const uint32_t k2 = k + stride;
    const bool two = k2 < n;
    const uint4 f = ldg4(faces + k);
    const uint4 f2 = two ? ldg4(faces + k2) : f;
    const float4 v0 = ldg4(verts + f.x), v1 = ldg4(verts + f.y), v2 = ldg4(verts + f.z);
    const float4 w0 = ldg4(verts + f2.x), w1 = ldg4(verts + f2.y), w2 = ldg4(verts + f2.z);
    face(k, v0, v1, v2);
    if (two) face(k2, w0, w1, w2);
  }
}

// ----------------------------------------------------------------------------
// Morton top tree (one CTA)
// ----------------------------------------------------------------------------
struct TopoArgs {
  const uint32_t* C;         // split positions, level ordered
  const uint32_t* lev_count; // [33] per-level counts (level 32 = no split)
  uint32_t n, D, min_leaf, max_leaf, complete;
  uint32_t cap_m;
  // BFS arrays
  uint32_t *ra, *rb, *parent, *info, *child, *leaves, *mleaves, *rank, *lambda, *ord, *id;
  // Morton leaves in position order
  uint32_t* ml_lambda;
  uint4* ml_rec;     // (node id, first, count, depth | median << 31)
  uint32_t* ml_rank; // pre-order rank (median roots)
  uint32_t* parent_id; // [max_nodes] parent node id of Morton nodes
  uint32_t* nodes;     // bvnode words
  uint32_t max_nodes;
  uint32_t* hdr;       // [16] header: 0 leaf_count, 1 morton_leaves, 2 node_count, 3 real_depth, 4 split_count,
                       //             5 overrun, 6 nondet, 7 past_end, 8 error
  const uint32_t* level_hist;   // optional [33] pair counts of this mesh's levels (batched build); else lev_count
  uint32_t level_base;          // with level_hist: where this mesh's level lists start in C
  uint32_t pos_base;            // first position of this mesh (0 for a single mesh)
};

// Morton levels whose nodes fit in shared memory: kTopoNodeBytes each, `cap` of them. False, with nothing written, if
// there are more (topo_morton then does it in global memory). Level by level down, with the split lists' first cap / 2
// entries beside the nodes; leaf counts up; ranks and the records down, where a node's counts make room for its rank.
// One CTA, so all of it is latency: going down a level is one barrier and a binary search of a short list. (With every array
// in global memory the same levels took 81 us for 2^20 faces (4096 cells), 62 for a terrain of 32k and 314 for 1024
// meshes; now 38, 32 and 200.)
constexpr uint32_t kTopoNodeBytes = 26;
constexpr uint32_t kTopoNodes = 8192;        // of a single build: every tree of depth 12 or less fits
constexpr uint32_t kBatchTopoNodes = 2560;   // of a batched build: 65 KB, three CTAs an SM
template <int NT>
__device__ __forceinline__ bool topo_shared(const TopoArgs& A, const uint32_t cap, char* smem) {
  uint32_t* const ra = (uint32_t*)smem;
  uint32_t* const rb = ra + cap;
  uint32_t* const cnt = rb + cap;     // leaves of the subtree; going down, the pre-order rank
  uint32_t* const lambda = cnt + cap;
  uint32_t* const id = lambda + cap;
  uint32_t* const C = id + cap;       // [cap / 2]
  uint16_t* const child = (uint16_t*)(C + cap / 2);  // 0: none
  uint16_t* const mcnt = child + cap;                // Morton leaves of the subtree; going down, the ordinal
  __shared__ uint32_t s_start[34], s_last[32];   // per level: its list's start and last entry (0: empty, above no a)
  __shared__ uint32_t s_vstar[34], s_made[33];   // per level: the a of its first visit at or after s_last; nodes made below it
  __shared__ uint32_t s_level_lo[34];
  __shared__ uint32_t s_overrun, s_nondet, s_past, s_err, s_depth, s_leaves, s_mleaves;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, D = A.D;
  if (tid < 32) {
    const uint32_t v = A.level_hist ? A.level_hist[tid] : A.lev_count[tid];
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    const uint32_t start = (A.level_hist ? A.level_base : 0u) + x - v;
    s_start[tid] = start;
    s_last[tid] = v ? __ldg(A.C + start + v - 1) : 0u;
    s_vstar[tid] = kNone;
    s_made[tid] = 0;
    if (tid == 31) s_start[32] = s_start[33] = start + v;
    if (tid == 0) {
      s_vstar[32] = s_vstar[33] = kNone;
      s_made[32] = 0;
      s_overrun = s_nondet = s_past = s_err = s_depth = 0;
      ra[0] = A.pos_base;
      rb[0] = A.pos_base + A.n;
    }
  }
  __syncthreads();
  const uint32_t first = s_start[0], S = s_start[32], held = min(S - first, cap / 2);
  for (uint32_t i = tid; i < held; i += NT) C[i] = __ldg(A.C + first + i);
  // a node of level L that is visited, at or after the level's last entry
  auto note = [&](uint32_t L, uint32_t a, uint32_t b) {
    if (L < 32 && b - a >= A.min_leaf && a >= s_last[L]) atomicMin(&s_vstar[L], a);
  };
  if (tid == 0) note(0, A.pos_base, A.pos_base + A.n);
  __syncthreads();
  // first index at or after level L's list whose entry s is above a (the lists are walked in order), S and kNone if none
  auto scan = [&](uint32_t L, uint32_t a, uint32_t& s) {
    for (uint32_t l = L; l < 32; ++l) {
      if (s_last[l] <= a) continue;
      uint32_t lo = s_start[l], hi = s_start[l + 1] - 1;
      s = s_last[l];
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1, x = mid - first < held ? C[mid - first] : __ldg(A.C + mid);
        if (x > a) { hi = mid; s = x; } else lo = mid + 1;
      }
      return lo;
    }
    s = kNone;
    return S;
  };
  // A level's nodes stand in any order: a visit's place among the level's visits is its a. So children are handed their
  // slots by a counter, and a level takes one barrier. The same counter says whether they fit: nothing adds to it after
  // the level's barrier, so every thread leaves at the same level (a flag shared by the levels would not do: the next
  // level may set it before a slow warp has read it for this one).
  const uint32_t room = min(cap, A.cap_m);
  uint32_t lo = 0, hi = 1, L = 0;
  for (; lo < hi; ++L) {
    if (tid == 0) s_level_lo[L] = lo;
    const bool visits = L < D && L < 32 && s_start[L] < s_start[L + 1];
    const uint32_t vstar = visits ? s_vstar[L] : kNone;
    // the pointer sticks at the next list's start if that entry, or the end, is what the first visit at or after s_last finds
    bool stuck = false;
    if (vstar != kNone) {
      const uint32_t j = s_start[L + 1];
      stuck = j == S || (j - first < held ? C[j - first] : __ldg(A.C + j)) > vstar;
    }
    for (uint32_t base = lo; base < hi; base += NT) {
      const uint32_t i = base + tid;
      bool internal = false;
      uint32_t a = 0, b = 0, s = 0;
      if (i < hi) {
        a = ra[i]; b = rb[i];
        if (visits && b - a >= A.min_leaf && !(stuck && a > vstar)) {
          const uint32_t j = scan(L, a, s);
          internal = s < b;
          if (j >= s_start[L + 1]) atomicAdd(&s_overrun, 1u);
          if (j < S && j >= s_start[min(D + 1, 32u)]) atomicAdd(&s_nondet, 1u);
          if (j == S) atomicAdd(&s_past, 1u);
        }
      }
      const uint32_t who = __ballot_sync(0xffffffffu, internal);
      uint32_t c = 0;
      if (who) {
        if (lane == 0) c = atomicAdd(&s_made[L], 2u * (uint32_t)__popc(who));
        c = hi + __shfl_sync(0xffffffffu, c, 0) + 2u * (uint32_t)__popc(who & ((1u << lane) - 1u));
      }
      if (internal) {
        if (c + 2 <= room) {
          ra[c] = a; rb[c] = s; ra[c + 1] = s; rb[c + 1] = b;
          note(L + 1, a, s);
          note(L + 1, s, b);
        }
      }
      if (i < hi) child[i] = (uint16_t)(internal ? c : 0u);
    }
    __syncthreads();
    const uint32_t made = s_made[L];
    if (hi + made > room) return false;
    lo = hi;
    hi += made;
  }
  if (tid == 0) s_level_lo[L] = lo;
  __syncthreads();
  const uint32_t levels = L, maxl = A.max_leaf;
  auto median = [&](uint32_t size) { return A.complete && size > maxl; };
  for (int l = (int)levels - 1; l >= 0; --l) {
    for (uint32_t i = s_level_lo[l] + tid; i < s_level_lo[l + 1]; i += NT) {
      const uint32_t c = child[i], size = rb[i] - ra[i];
      cnt[i] = c ? cnt[c] + cnt[c + 1] : median(size) ? median_leaves(size, maxl) : 1u;
      mcnt[i] = c ? (uint16_t)(mcnt[c] + mcnt[c + 1]) : (uint16_t)1u;
    }
    __syncthreads();
  }
  if (tid == 0) {
    s_leaves = cnt[0]; s_mleaves = mcnt[0];
    cnt[0] = lambda[0] = id[0] = 0;
    mcnt[0] = 0;
    if (A.max_nodes) A.parent_id[0] = kNone;
  }
  __syncthreads();
  uint32_t depth = 0, err = 0;
  for (uint32_t l = 0; l < levels; ++l) {
    for (uint32_t i = s_level_lo[l] + tid; i < s_level_lo[l + 1]; i += NT) {
      const uint32_t c = child[i], nid = id[i], r = cnt[i], lam = lambda[i], o = mcnt[i];
      const bool fits = nid < A.max_nodes;
      if (!fits) err = RT_DEVERR_NODE_CAPACITY;
      if (c) {
        const uint32_t ll = cnt[c], ml = mcnt[c];
        cnt[c] = r + 1; lambda[c] = lam; id[c] = 2 * r + 1; mcnt[c] = (uint16_t)o;
        cnt[c + 1] = r + ll; lambda[c + 1] = lam + ll; id[c + 1] = 2 * r + 2; mcnt[c + 1] = (uint16_t)(o + ml);
        if (2 * r + 1 < A.max_nodes) A.parent_id[2 * r + 1] = nid;
        if (2 * r + 2 < A.max_nodes) A.parent_id[2 * r + 2] = nid;
        if (fits) *(uint2*)(A.nodes + 8 * (size_t)nid) = make_uint2((l % 3u) << 1, 2 * r + 1);
      } else if (fits) {
        const uint32_t size = rb[i] - ra[i];
        const bool med = median(size);
        A.ml_lambda[o] = lam;
        A.ml_rec[o] = make_uint4(nid, ra[i], size, l | (med ? 0x80000000u : 0u));
        A.ml_rank[o] = r;
        depth = max(depth, l + (med ? median_depth(size, maxl) : 0u) + 1u);
      }
    }
    __syncthreads();
  }
  if (depth) atomicMax(&s_depth, depth);
  if (err) atomicOr(&s_err, err);
  __syncthreads();
  if (tid == 0) {
    A.hdr[0] = s_leaves;
    A.hdr[1] = s_mleaves;
    A.hdr[2] = 2 * s_leaves - 1;
    A.hdr[3] = s_depth;
    A.hdr[4] = S - first;
    A.hdr[5] = s_overrun;
    A.hdr[6] = s_nondet;
    A.hdr[7] = s_past;
    A.hdr[8] = s_err | ((2 * s_leaves - 1 > A.max_nodes) ? (uint32_t)RT_DEVERR_NODE_CAPACITY : 0u);
  }
  return true;
}

template <int NT>
__device__ __forceinline__ void topo_morton(const TopoArgs& A) {
  __shared__ uint32_t s_start[34];
  __shared__ uint32_t s_level_lo[34];
  __shared__ uint32_t s_warp[NT / 32];
  __shared__ uint32_t s_vstar, s_stuck, s_levels;
  __shared__ uint32_t s_overrun, s_nondet, s_past, s_err, s_depth;
  const uint32_t tid = threadIdx.x;
  if (tid == 0) {
    if (A.level_hist) {
      uint32_t acc = A.level_base;
      for (int l = 0; l < 33; ++l) { s_start[l] = acc; acc += (l < 32) ? A.level_hist[l] : 0u; }
    } else {
      uint32_t acc = 0;
      for (int l = 0; l < 33; ++l) { s_start[l] = acc; acc += (l < 32) ? A.lev_count[l] : 0u; }
    }
    s_start[33] = s_start[32];
    s_overrun = s_nondet = s_past = s_err = s_depth = 0;
    A.ra[0] = A.pos_base; A.rb[0] = A.pos_base + A.n; A.parent[0] = kNone;
  }
  __syncthreads();
  const uint32_t S = s_start[32];
  const uint32_t D = A.D;
  uint32_t lo = 0, hi = 1, L = 0;
  for (; lo < hi; ++L) {
    if (tid == 0) { s_level_lo[L] = lo; s_vstar = kNone; s_stuck = 0; }
    __syncthreads();
    const bool nonempty = L < 32 && s_start[L] < s_start[L + 1];
    const uint32_t lastL = nonempty ? __ldg(A.C + s_start[L + 1] - 1) : 0u;
    if (nonempty && L < D) {
      for (uint32_t i = lo + tid; i < hi; i += NT) {
        uint32_t a = A.ra[i], b = A.rb[i];
        if (b - a >= A.min_leaf && a >= lastL) atomicMin(&s_vstar, i);
      }
    }
    __syncthreads();
    if (tid == 0 && s_vstar != kNone) {
      uint32_t j = split_scan(A.C, s_start, L, A.ra[s_vstar]);
      s_stuck = (j == s_start[L + 1]) ? 1u : 0u;
    }
    __syncthreads();
    uint32_t running = hi;
    for (uint32_t base = lo; base < hi; base += NT) {
      const uint32_t i = base + tid;
      bool internal = false;
      uint32_t a = 0, b = 0, s = 0, inf = 0;
      if (i < hi) {
        a = A.ra[i]; b = A.rb[i];
        const bool visit = (b - a >= A.min_leaf) && L < D && nonempty;
        if (visit && !(s_vstar != kNone && i > s_vstar && s_stuck)) {
          uint32_t j = split_scan(A.C, s_start, L, a);
          s = (j < S) ? __ldg(A.C + j) : kNone;
          internal = s < b;
          if (j >= s_start[L + 1]) atomicAdd(&s_overrun, 1u);
          if (j < S && j >= s_start[min(D + 1, 32u)]) atomicAdd(&s_nondet, 1u);
          if (j == S) atomicAdd(&s_past, 1u);
        }
        const bool median = !internal && A.complete && (b - a > A.max_leaf);
        inf = L | (internal ? 0x100u : 0u) | (median ? 0x200u : 0u);
      }
      uint32_t total;
      uint32_t ex = block_excl_scan_nt<NT>(internal ? 2u : 0u, s_warp, total);
      if (i < hi) {
        uint32_t c = kNone;
        if (internal) {
          c = running + ex;
          if (c + 1 < A.cap_m) {
            A.ra[c] = a; A.rb[c] = s; A.ra[c + 1] = s; A.rb[c + 1] = b;
            A.parent[c] = i; A.parent[c + 1] = i;
          } else {
            // cannot happen (the Morton levels hold at most min(2^(D+1), 2n) - 1
            // nodes); kept as a guarded leaf so that no index leaves its array
            atomicOr(&s_err, (uint32_t)RT_DEVERR_MORTON_CAPACITY);
            c = kNone;
            inf &= ~0x100u;
          }
        }
        A.child[i] = c;
        A.info[i] = inf;
      }
      running += total;
    }
    __syncthreads();
    lo = hi;
    hi = min(running, A.cap_m);
  }
  if (tid == 0) { s_level_lo[L] = lo; s_levels = L; }
  __syncthreads();
  const uint32_t levels = s_levels;
  const uint32_t maxl = A.max_leaf;

  // bottom-up: leaves (final tree) and Morton leaves per subtree
  for (int l = (int)levels - 1; l >= 0; --l) {
    for (uint32_t i = s_level_lo[l] + tid; i < s_level_lo[l + 1]; i += NT) {
      uint32_t inf = A.info[i];
      if (inf & 0x100u) {
        uint32_t c = A.child[i];
        A.leaves[i] = A.leaves[c] + A.leaves[c + 1];
        A.mleaves[i] = A.mleaves[c] + A.mleaves[c + 1];
      } else {
        uint32_t size = A.rb[i] - A.ra[i];
        A.leaves[i] = (inf & 0x200u) ? median_leaves(size, maxl) : 1u;
        A.mleaves[i] = 1u;
      }
    }
    __syncthreads();
  }
  // top-down: rank, lambda (leaves to the left), Morton-leaf ordinal, node id
  if (tid == 0) { A.rank[0] = 0; A.lambda[0] = 0; A.ord[0] = 0; A.id[0] = 0; }
  __syncthreads();
  for (uint32_t l = 0; l < levels; ++l) {
    for (uint32_t i = s_level_lo[l] + tid; i < s_level_lo[l + 1]; i += NT) {
      if (A.info[i] & 0x100u) {
        uint32_t c = A.child[i];
        uint32_t r = A.rank[i], lam = A.lambda[i], o = A.ord[i];
        uint32_t ll = A.leaves[c];
        A.rank[c] = r + 1; A.lambda[c] = lam; A.ord[c] = o; A.id[c] = 2 * r + 1;
        A.rank[c + 1] = r + ll; A.lambda[c + 1] = lam + ll; A.ord[c + 1] = o + A.mleaves[c]; A.id[c + 1] = 2 * r + 2;
      }
    }
    __syncthreads();
  }
  // emit Morton node records and the Morton-leaf table
  const uint32_t total_m = s_level_lo[levels];
  for (uint32_t i = tid; i < total_m; i += NT) {
    const uint32_t inf = A.info[i];
    const uint32_t lvl = inf & 0xFFu;
    const uint32_t nid = A.id[i];
    if (nid >= A.max_nodes) { atomicOr(&s_err, (uint32_t)RT_DEVERR_NODE_CAPACITY); continue; }
    A.parent_id[nid] = (i == 0) ? kNone : A.id[A.parent[i]];
    if (inf & 0x100u) {
      uint2 w = make_uint2((lvl % 3u) << 1, 2 * A.rank[i] + 1);
      *(uint2*)(A.nodes + 8 * (size_t)nid) = w;
    } else {
      const uint32_t k = A.ord[i];
      const uint32_t first = A.ra[i], cnt = A.rb[i] - A.ra[i];
      const bool median = (inf & 0x200u) != 0;
      A.ml_lambda[k] = A.lambda[i];
      A.ml_rec[k] = make_uint4(nid, first, cnt, lvl | (median ? 0x80000000u : 0u));
      A.ml_rank[k] = A.rank[i];
      uint32_t depth = lvl + (median ? median_depth(cnt, maxl) : 0u) + 1u;
      atomicMax(&s_depth, depth);
    }
  }
  __syncthreads();
  if (tid == 0) {
    const uint32_t leaves = A.leaves[0];
    A.hdr[0] = leaves;
    A.hdr[1] = A.mleaves[0];
    A.hdr[2] = 2 * leaves - 1;
    A.hdr[3] = s_depth;
    A.hdr[4] = S - s_start[0];
    A.hdr[5] = s_overrun;
    A.hdr[6] = s_nondet;
    A.hdr[7] = s_past;
    A.hdr[8] = s_err | ((2 * leaves - 1 > A.max_nodes) ? (uint32_t)RT_DEVERR_NODE_CAPACITY : 0u);
  }
}

__global__ __launch_bounds__(kTopoThreads) void k_topo_morton(TopoArgs A) {
  extern __shared__ __align__(16) char topo_smem[];
  if (!topo_shared<kTopoThreads>(A, kTopoNodes, topo_smem)) {
    __syncthreads();
    topo_morton<kTopoThreads>(A);
  }
}

// ----------------------------------------------------------------------------
// leaves: a warp takes 32 consecutive leaves at a time
// ----------------------------------------------------------------------------
struct LeafArgs {
  const float4* verts;
  const uint4* faces_in;
  uint4* faces_out;      // may be null (tree_complete == 0)
  float4* tris;          // may be null
  const uint32_t* indices;
  const uint32_t* ml_lambda;
  const uint4* ml_rec;
  const uint32_t* ml_rank;
  uint32_t* parent_id;
  uint32_t* arrive;
  uint32_t* nodes;
  uint32_t max_nodes;
  uint32_t max_leaf;
  const uint32_t* hdr;
  uint32_t* err;
  // traversal blob (optional): leaf table in leaf order, 8-triangle group boxes
  uint4* acc_leaves;
  float4* acc_groups;
  uint32_t* leaf_lambda;  // node id -> leaf order index
  uint32_t pos_base;      // first position of this mesh (node records store positions relative to it)
  uint32_t vert_base;     // first vertex of this mesh (faces index vertices relative to it)
  uint32_t* local_indices; // optional: indices[i] - pos_base written here (batched build)
  uint32_t parent_cap;     // entries of parent_id (median nodes' parents are written here)
};

constexpr int kMaxMedianDepth = 40;

// What a lane knows of one final leaf: where its faces are, its node and its place in the blob.
struct LeafMeta {
  uint32_t first;   // absolute position of its first face
  uint32_t cnt;
  uint32_t node;    // its node, counted from the first mesh's root (~0: beyond the node array)
  uint32_t group;   // its first group box, counted from the first mesh's
  uint32_t vert_base, pos_base;  // its mesh's first vertex and first position
};

// Last k < n with v[k] <= x (v ascending, v[0] <= x), the same x for the whole warp: 32 places at a time.
__device__ __forceinline__ uint32_t warp_last_le(const uint32_t* __restrict__ v, uint32_t n, uint32_t x) {
  const uint32_t lane = lane_id();
  uint32_t lo = 0, len = n;
  while (len > 1) {
    const uint32_t step = (len + 31) / 32, at = lane * step;
    const uint32_t c = (uint32_t)__popc(__ballot_sync(0xffffffffu, at < len && v[lo + at] <= x)) - 1u;
    lo += c * step;
    len = min(step, len - c * step);
  }
  return lo;
}
// The Morton leaves of leaves g .. g + 31 of one mesh (lane l: leaf g + l), the first one's found by the whole warp.
__device__ __forceinline__ uint32_t warp_morton_leaf(const LeafArgs& A, uint32_t g) {
  const uint32_t lane = lane_id(), count = A.hdr[1];
  const uint32_t first = warp_last_le(A.ml_lambda, count, g);
  const uint32_t v = first + lane < count ? A.ml_lambda[first + lane] : ~0u;
  uint32_t lo = 0;
#pragma unroll
  for (uint32_t step = 16; step; step >>= 1)
    if (__shfl_sync(0xffffffffu, v, lo + step) <= g + lane) lo += step;
  return first + lo;
}

// Leaf g (in its mesh's leaf order, in Morton leaf lo) of the mesh that A describes. Writes what does not need the faces: the nodes of a
// median subtree whose first leaf this is, the blob's leaf entry.
__device__ __forceinline__ LeafMeta leaf_meta(const LeafArgs& A, const uint32_t g, const uint32_t lo, uint32_t node_first,
                                              uint32_t group_first) {
  const uint4 rec = A.ml_rec[lo];
  uint32_t nid = rec.x, first = rec.y, size = rec.z;  // first: absolute position
  if (rec.w & 0x80000000u) {
    uint32_t q = g - A.ml_lambda[lo], rank = A.ml_rank[lo], depth = rec.w & 0xFFFFu;
    int plen = 0;  // median levels walked
    while (size >= A.max_leaf && plen < kMaxMedianDepth) {
      const uint32_t left = size >> 1, right = size - left;
      const uint32_t ll = median_leaves(left, A.max_leaf);
      // the subtree's first leaf writes the internal record and its children's parent ids
      if (q == 0 && nid < A.max_nodes) {
        *(uint2*)(A.nodes + 8 * (size_t)nid) = make_uint2((depth % 3u) << 1, 2 * rank + 1);
        if (2 * rank + 2 < A.parent_cap) {
          A.parent_id[2 * rank + 1] = nid;
          A.parent_id[2 * rank + 2] = nid;
        }
      }
      ++plen;
      if (q < ll) { nid = 2 * rank + 1; rank = rank + 1; size = left; }
      else { q -= ll; nid = 2 * rank + 2; rank = rank + ll; first += left; size = right; }
      ++depth;
    }
  }
  LeafMeta L;
  L.first = first; L.cnt = size;
  L.vert_base = A.vert_base; L.pos_base = A.pos_base;
  const uint32_t lfirst = first - A.pos_base;   // position inside the mesh
  const uint32_t gbase = (lfirst >> 3) + g;     // leaf g's groups: disjoint across leaves, no scan needed
  L.group = group_first + gbase;
  const bool fits = nid < A.max_nodes;
  L.node = fits ? node_first + nid : kNone;
  if (A.acc_leaves && fits) {
    A.acc_leaves[g] = make_uint4(lfirst, size, gbase, nid);
    A.leaf_lambda[nid] = g;
  }
  if (!fits) atomicOr(A.err, (uint32_t)RT_DEVERR_NODE_CAPACITY);
  return L;
}

// The faces of up to 32 consecutive leaves, one leaf's metadata per lane (cnt 0: none), by one warp: per face the
// reordered face, the triangle {v0, e1, e2} and (batched) the mesh-local index, per 8 faces of a leaf a padded group
// box, per leaf its box and node words. The leaves' faces are taken 32 at a time as one sequence, cut back to whole
// groups, so that short leaves share a step; the boxes are reduced inside the lanes of each group and then over a
// leaf's groups, which are eight lanes apart, and a leaf that goes on past a step carries its box along. Boxes are
// combined in position order with the selects of a sequential scan. The next step's indices and faces are loaded
// while this one's vertices are on their way. (A warp per leaf with lane 0 finding it, one leaf and one dependent load
// after another, took 1.29 ms for 2^24 faces of a soup and 1.31 ms for 9.9M in 1024 meshes; this takes 0.98 ms, bound by
// DRAM (5.8 TB/s of scattered reads, 276 bytes per face), and 0.63.)
// `out`: arrays of the whole build (nodes and group boxes of the first mesh).
__device__ __forceinline__ void leaf_faces(const LeafArgs& out, const LeafMeta& L) {
  const uint32_t lane = lane_id();
  uint32_t incl = L.cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  const uint32_t off = incl - L.cnt, total = __shfl_sync(0xffffffffu, incl, 31);
  struct Step {
    uint32_t owner, rel, cnt, n;  // the lane's leaf, its place in it, the leaf's faces; faces of the step (lanes 0 .. n - 1)
    uint32_t pos, idx;
    uint4 f;
  };
  auto begin_step = [&](uint32_t w) {
    Step s;
    const uint32_t item = w + lane;
    uint32_t lo = 0;
#pragma unroll
    for (uint32_t step = 16; step; step >>= 1) {  // last leaf that starts at or before the item
      const uint32_t o = __shfl_sync(0xffffffffu, off, lo + step);
      if (o <= item) lo += step;
    }
    // (empty leaves at the end start at `total`: items before it never reach them)
    s.owner = lo;
    s.rel = item - __shfl_sync(0xffffffffu, off, lo);
    s.cnt = __shfl_sync(0xffffffffu, L.cnt, lo);
    const bool whole = item < total && item - (s.rel & 7u) + min(8u, s.cnt - (s.rel & ~7u)) <= w + 32;
    s.n = (uint32_t)__popc(__ballot_sync(0xffffffffu, whole));
    s.pos = __shfl_sync(0xffffffffu, L.first, lo) + s.rel;
    s.idx = 0;
    s.f = make_uint4(0, 0, 0, 0);
    if (lane < s.n) {
      s.idx = __ldg(out.indices + s.pos);
      s.f = ldg4(out.faces_in + s.idx);
    }
    return s;
  };
  float3 cmn = make_float3(kHuge, kHuge, kHuge), cmx = make_float3(-kHuge, -kHuge, -kHuge);  // box of a leaf that goes on
  uint32_t w = 0;
  if (total == 0) return;
  Step s = begin_step(0);
  while (w < total) {
    const bool act = lane < s.n;
    const uint32_t vb = __shfl_sync(0xffffffffu, L.vert_base, s.owner);
    float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0, v2 = v0;
    if (act) {
      v0 = ldg4(out.verts + vb + s.f.x);
      v1 = ldg4(out.verts + vb + s.f.y);
      v2 = ldg4(out.verts + vb + s.f.z);
    }
    const Step c = s;
    const uint32_t wn = w + c.n;
    if (wn < total) s = begin_step(wn);
    const uint32_t pb = __shfl_sync(0xffffffffu, L.pos_base, c.owner), group = __shfl_sync(0xffffffffu, L.group, c.owner);
    const uint32_t node = __shfl_sync(0xffffffffu, L.node, c.owner), first = __shfl_sync(0xffffffffu, L.first, c.owner);
    float3 mn = make_float3(kHuge, kHuge, kHuge), mx = make_float3(-kHuge, -kHuge, -kHuge);
    if (act) {
      if (out.local_indices) out.local_indices[c.pos] = c.idx - pb;
      if (out.faces_out) out.faces_out[c.pos] = c.f;
      if (out.tris) {
        out.tris[3 * (size_t)c.pos + 0] = make_float4(v0.x, v0.y, v0.z, 0.0f);
        out.tris[3 * (size_t)c.pos + 1] = make_float4(v1.x - v0.x, v1.y - v0.y, v1.z - v0.z, 0.0f);
        out.tris[3 * (size_t)c.pos + 2] = make_float4(v2.x - v0.x, v2.y - v0.y, v2.z - v0.z, 0.0f);
      }
      mn = make_float3(fmin_sel(fmin_sel(v0.x, v1.x), v2.x), fmin_sel(fmin_sel(v0.y, v1.y), v2.y), fmin_sel(fmin_sel(v0.z, v1.z), v2.z));
      mx = make_float3(fmax_sel(fmax_sel(v0.x, v1.x), v2.x), fmax_sel(fmax_sel(v0.y, v1.y), v2.y), fmax_sel(fmax_sel(v0.z, v1.z), v2.z));
    }
    // lanes past which the lane's group and leaf end (inside the step)
    const uint32_t gend = lane - (c.rel & 7u) + min(8u, c.cnt - (c.rel & ~7u));
    const uint32_t lend = min(c.n, lane + c.cnt - c.rel);
    auto combine = [&](uint32_t o, uint32_t end) {
      const float3 bn = make_float3(__shfl_down_sync(0xffffffffu, mn.x, o), __shfl_down_sync(0xffffffffu, mn.y, o),
                                    __shfl_down_sync(0xffffffffu, mn.z, o));
      const float3 bx = make_float3(__shfl_down_sync(0xffffffffu, mx.x, o), __shfl_down_sync(0xffffffffu, mx.y, o),
                                    __shfl_down_sync(0xffffffffu, mx.z, o));
      if (lane + o < end) {
        mn = make_float3(fmin_sel(mn.x, bn.x), fmin_sel(mn.y, bn.y), fmin_sel(mn.z, bn.z));
        mx = make_float3(fmax_sel(mx.x, bx.x), fmax_sel(mx.y, bx.y), fmax_sel(mx.z, bx.z));
      }
    };
    combine(1, gend);
    combine(2, gend);
    combine(4, gend);
    if (act && (c.rel & 7u) == 0 && out.acc_groups) {
      float3 pmn = mn, pmx = mx;
      pad_box(pmn, pmx);
      const size_t gi = (size_t)group + (c.rel >> 3);
      out.acc_groups[2 * gi] = make_float4(pmn.x, pmn.y, pmn.z, 0.0f);
      out.acc_groups[2 * gi + 1] = make_float4(pmx.x, pmx.y, pmx.z, 0.0f);
    }
    combine(8, lend);
    combine(16, lend);
    // a leaf's first lane of the step now holds the leaf's box over the step; lane 0 may hold the rest of a leaf
    const bool head = act && (c.rel == 0 || lane == 0);
    if (lane == 0 && c.rel != 0) {
      mn = make_float3(fmin_sel(cmn.x, mn.x), fmin_sel(cmn.y, mn.y), fmin_sel(cmn.z, mn.z));
      mx = make_float3(fmax_sel(cmx.x, mx.x), fmax_sel(cmx.y, mx.y), fmax_sel(cmx.z, mx.z));
    }
    const bool done = lane + c.cnt - c.rel <= c.n;  // the leaf ends inside the step
    if (head && done && node != kNone) {
      uint32_t* nd = out.nodes + 8 * (size_t)node;
      *(uint2*)nd = make_uint2(1u | (c.cnt << 1), first - pb);
      write_box(nd, mn, mx);
    }
    const uint32_t open = __ballot_sync(0xffffffffu, head && !done);  // at most the step's last leaf
    if (open) {
      const int o = __ffs(open) - 1;
      cmn = make_float3(__shfl_sync(0xffffffffu, mn.x, o), __shfl_sync(0xffffffffu, mn.y, o), __shfl_sync(0xffffffffu, mn.z, o));
      cmx = make_float3(__shfl_sync(0xffffffffu, mx.x, o), __shfl_sync(0xffffffffu, mx.y, o), __shfl_sync(0xffffffffu, mx.z, o));
    }
    w = wn;
  }
}

// Node boxes bottom-up, one thread per leaf: the leaf (its box written by the
// leaf kernel) climbs through parent_id; at each internal node the first of
// its two children to arrive stops, the second merges both children's boxes
// and climbs on. cap bounds every node id (the node array's capacity).
__device__ __forceinline__ void climb(uint32_t* __restrict__ nodes, const uint32_t* __restrict__ parent_id, uint32_t* __restrict__ arrive,
                                      uint32_t cap, uint32_t leaf) {
  uint32_t cur = leaf;
  for (;;) {
    const uint32_t p = parent_id[cur];
    if (p == kNone || p >= cap) break;
    __threadfence();
    if (atomicAdd(arrive + p, 1u) == 0u) break;
    __threadfence();
    const uint32_t c0 = __ldcg(nodes + 8 * (size_t)p + 1);
    if (c0 + 1 >= cap) break;
    const float* l = (const float*)(nodes + 8 * (size_t)c0);
    const float* r = (const float*)(nodes + 8 * (size_t)(c0 + 1));
    float lb[6], rb[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) { lb[q] = __ldcg(l + 2 + q); rb[q] = __ldcg(r + 2 + q); }
    float3 bmn, bmx;
    // kernels/CUDA_buildMeshTreeLBVH.cu:269-300: merged only when both children have a positive z extent
    if (lb[5] - lb[2] > 0.0f && rb[5] - rb[2] > 0.0f) {
      bmn = make_float3(fmin_sel(lb[0], rb[0]), fmin_sel(lb[1], rb[1]), fmin_sel(lb[2], rb[2]));
      bmx = make_float3(fmax_sel(lb[3], rb[3]), fmax_sel(lb[4], rb[4]), fmax_sel(lb[5], rb[5]));
    } else {
      bmn = make_float3(kHuge, kHuge, kHuge);
      bmx = make_float3(-kHuge, -kHuge, -kHuge);
    }
    write_box(nodes + 8 * (size_t)p, bmn, bmx);
    cur = p;
  }
}

// Bottom-up boxes of a single mesh: one thread per node, the leaves climb.
__global__ __launch_bounds__(256) void k_propagate(uint32_t* __restrict__ nodes, const uint32_t* __restrict__ parent_id,
                                                   uint32_t* __restrict__ arrive, const uint32_t* __restrict__ hdr, uint32_t cap) {
  if (hdr[8] & (RT_DEVERR_NODE_CAPACITY | RT_DEVERR_MORTON_CAPACITY)) return;
  const uint32_t node_count = min(hdr[2], cap);
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < node_count; p += gridDim.x * blockDim.x)
    if (nodes[8 * (size_t)p] & 1u) climb(nodes, parent_id, arrive, cap, p);
}

// The next run of leaves of a warp, from a counter (zero at the start): runs of about 512 faces (fewer where that leaves
// warps without one), at most 32 leaves, so that a warp with large leaves does not keep the launch waiting: runs dealt
// out beforehand, by leaves alone, left half of the SM time idle on meshes of mixed sizes.
__device__ __forceinline__ uint32_t leaf_run(uint32_t leaf_count, uint32_t faces) {
  const unsigned long long want = max(64u, min(512u, faces / 8192u));
  return (uint32_t)max(1ull, min(32ull, want * leaf_count / faces));
}
__device__ __forceinline__ uint32_t next_run(uint32_t* counter, uint32_t run) {
  uint32_t g = 0;
  if (lane_id() == 0) g = atomicAdd(counter, run);
  return __shfl_sync(0xffffffffu, g, 0);
}

__global__ __launch_bounds__(256) void k_leaves(LeafArgs A, uint32_t faces, uint32_t* counter) {
  const uint32_t leaf_count = A.hdr[0], lane = lane_id();
  if (A.hdr[8] & (RT_DEVERR_NODE_CAPACITY | RT_DEVERR_MORTON_CAPACITY)) return;
  const uint32_t run = leaf_run(leaf_count, faces);
  for (;;) {
    const uint32_t g = next_run(counter, run);
    if (g >= leaf_count) break;
    const uint32_t lo = warp_morton_leaf(A, g);
    LeafMeta L = {};
    if (lane < run && g + lane < leaf_count) L = leaf_meta(A, g + lane, lo, 0u, 0u);
    leaf_faces(A, L);
  }
}

// Two-child traversal records, indexed by pre-order rank (internal node p
// with left child c has rank (c - 1) / 2): both children's padded boxes and
// references (rank for an internal child, ~leaf index for a leaf child).
__global__ __launch_bounds__(256) void k_accel_nodes(const uint32_t* __restrict__ nodes, const uint32_t* __restrict__ hdr,
                                                    const uint32_t* __restrict__ leaf_lambda, float4* __restrict__ tnodes,
                                                    float4* __restrict__ wide, uint32_t* __restrict__ acc_hdr) {
  const uint32_t node_count = hdr[2];
  if (hdr[8] & (RT_DEVERR_NODE_CAPACITY | RT_DEVERR_MORTON_CAPACITY)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const bool root_leaf = (nodes[0] & 1u) != 0;
    acc_hdr[0] = root_leaf ? ~0u : 0u;  // root reference
    acc_hdr[1] = hdr[0];                // leaf count
    acc_hdr[2] = node_count;
  }
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < node_count; p += gridDim.x * blockDim.x)
    accel_wide_node(nodes, leaf_lambda, tnodes, wide, p);
}

__global__ void k_write_info(const uint32_t* __restrict__ hdr, const uint32_t* __restrict__ err, rt_build_info* info) {
  if (threadIdx.x != 0) return;
  info->leaf_count = hdr[0];
  info->node_count = hdr[2];
  info->real_depth = hdr[3];
  info->split_count = hdr[4];
  info->overrun_visits = hdr[5];
  info->nondet_reads = hdr[6];
  info->past_end_reads = hdr[7];
  info->error = hdr[8] | *err;
}

struct BuildLayout {
  uint32_t n, cap_m, max_nodes, tiles;
  float4* hit;
  float4* partial;
  uint32_t* codes;
  uint32_t* C;
  uint32_t* lev_count;
  void* sort_scratch;
  size_t sort_bytes;
  uint32_t *ra, *rb, *parent, *info, *child, *leaves, *mleaves, *rank, *lambda, *ord, *id;
  uint32_t* ml_lambda;
  uint4* ml_rec;
  uint32_t* ml_rank;
  uint32_t* parent_id;
  uint32_t* arrive;
  uint32_t* hdr;
  uint32_t* err;
  uint32_t* leaf_lambda;
  uint4* faces_tmp;
  uint32_t* hit_done;  // the hit box's block counter, then the next leaf to hand out
  ClusterTemps ct;   // cluster tree build (RT_ACCEL_CLUSTERS only)
};

constexpr uint32_t kHitParts = 1184;  // 8 blocks per SM on 148 SMs
constexpr uint32_t kHitSplit = 8;     // CTAs per mesh of the batched hit box, at most

__host__ __device__ uint32_t morton_cap_dev(uint32_t n, uint32_t D) {
  uint64_t a = (D >= 31) ? (1ull << 32) : ((1ull << (D + 1)) - 1);
  uint64_t b = 2ull * n + 1;
  uint64_t c = a < b ? a : b;
  return (uint32_t)(c + 2);
}

uint32_t morton_cap(uint32_t n, uint32_t D) {
  uint64_t a = (D >= 31) ? (1ull << 32) : ((1ull << (D + 1)) - 1);
  uint64_t b = 2ull * n + 1;
  uint64_t c = a < b ? a : b;
  return (uint32_t)(c + 2);
}

size_t carve_build(Carve& c, BuildLayout& L, uint32_t n, uint32_t D, bool need_codes, bool need_faces_tmp, bool clusters) {
  L.n = n;
  L.cap_m = morton_cap(n, D);
  L.max_nodes = 2 * n - 1;
  L.hit = c.take<float4>(2);
  L.partial = c.take<float4>(2 * kHitParts);
  L.codes = need_codes ? c.take<uint32_t>(n) : nullptr;
  L.C = c.take<uint32_t>(n);
  L.lev_count = c.take<uint32_t>(256);
  L.sort_bytes = hmax<size_t>(radix_scratch_bytes(n), segment_sort_scratch_bytes(n, 1));
  L.sort_scratch = c.take<char>(L.sort_bytes);
  uint32_t** bfs[] = {&L.ra, &L.rb, &L.parent, &L.info, &L.child, &L.leaves, &L.mleaves, &L.rank, &L.lambda, &L.ord, &L.id};
  for (auto p : bfs) *p = c.take<uint32_t>(L.cap_m);
  L.ml_lambda = c.take<uint32_t>(L.cap_m);
  L.ml_rec = c.take<uint4>(L.cap_m);
  L.ml_rank = c.take<uint32_t>(L.cap_m);
  L.parent_id = c.take<uint32_t>(L.max_nodes);
  L.arrive = c.take<uint32_t>(L.max_nodes);
  L.hdr = c.take<uint32_t>(16);
  L.err = c.take<uint32_t>(4);
  L.leaf_lambda = c.take<uint32_t>(L.max_nodes);
  L.faces_tmp = need_faces_tmp ? c.take<uint4>(n) : nullptr;
  L.hit_done = c.take<uint32_t>(2);
  L.ct = ClusterTemps{};
  if (clusters) carve_cluster_temps(c, L.ct, n, 1);
  return c.off + 256;
}

// SM count of the current device (cached per device).
int sm_count() {
  static std::atomic<int> cache[PerDeviceOnce::kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= PerDeviceOnce::kMaxDevices) return 148;
  int s = cache[dev].load(std::memory_order_relaxed);
  if (s <= 0) {
    if (cudaDeviceGetAttribute(&s, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || s <= 0) s = 148;
    cache[dev].store(s, std::memory_order_relaxed);
  }
  return s;
}

// Blocks of `kernel` (with `threads` per block and no dynamic shared memory)
// that one SM holds at once: a grid of sm_count() times this is one resident
// wave. Queried once per kernel (the first call).
template <typename K>
int resident_blocks_of(K kernel, int threads) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, 0) != cudaSuccess || nb <= 0) {
    cudaGetLastError();
    nb = 1;
  }
  return nb;
}

// Lets a topology kernel (one instance each) have the shared memory of `nodes` nodes; once per device.
template <typename K>
bool topo_smem_once(K kernel, uint32_t nodes) {
  static PerDeviceOnce once;
  return once.run([&] {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(nodes * kTopoNodeBytes)) == cudaSuccess;
  });
}

}  // namespace

SideStream* side_stream(cudaStream_t st) {
  // one per host thread and device (a stream takes part in one capture at a time, and a thread's calls are
  // ordered, so the fork and join events of two calls never interleave); kept until the process exits
  constexpr int kMaxDevices = 64;
  thread_local SideStream per_device[kMaxDevices];
  thread_local int state[kMaxDevices] = {};  // 0 not yet, 1 ready, -1 refused
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return nullptr;
  }
  if (state[dev] == 0) {
    SideStream& x = per_device[dev];
    const bool ok = cudaStreamCreateWithFlags(&x.s, cudaStreamNonBlocking) == cudaSuccess &&
                    cudaEventCreateWithFlags(&x.fork, cudaEventDisableTiming) == cudaSuccess &&
                    cudaEventCreateWithFlags(&x.join, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) cudaGetLastError();
    state[dev] = ok ? 1 : -1;
  }
  if (state[dev] != 1) return nullptr;
  // an earlier call of this thread may have taken the side stream into a capture that has not ended: only that capture's
  // calls can use it until then
  cudaStreamCaptureStatus side = cudaStreamCaptureStatusNone, own = cudaStreamCaptureStatusNone;
  unsigned long long side_id = 0, own_id = 0;
  if (cudaStreamGetCaptureInfo(per_device[dev].s, &side, &side_id) != cudaSuccess ||
      (side != cudaStreamCaptureStatusNone && cudaStreamGetCaptureInfo(st, &own, &own_id) != cudaSuccess)) {
    cudaGetLastError();
    return nullptr;
  }
  if (side != cudaStreamCaptureStatusNone && (own == cudaStreamCaptureStatusNone || own_id != side_id)) return nullptr;
  return &per_device[dev];
}

}  // namespace rt

using namespace rt;

static rt_build_params normalized(const rt_build_params* p) {
  rt_build_params q = p ? *p : rt_build_params{12, 1, 0, 0, 32};
  if (q.tree_depth == 0) q.tree_depth = 12;
  if (q.tree_depth > 32) q.tree_depth = 32;
  if (q.min_leaf == 0) q.min_leaf = kMinLeafDefault;
  if (q.max_leaf == 0) q.max_leaf = kMaxLeafDefault;
  if (q.morton_bits == 0) q.morton_bits = 32;
  if (q.cluster_leaf == 0) q.cluster_leaf = kClusterLeafDefault;
  return q;
}

extern "C" rt_status rt_lbvh_scratch_bytes(uint32_t face_count, const rt_build_params* params, size_t* scratch_bytes, uint32_t* max_nodes) {
  if (!scratch_bytes || face_count == 0) return RT_ERR_INVALID_ARGUMENT;
  rt_build_params q = normalized(params);
  Carve c(nullptr, 0);
  BuildLayout L;
  *scratch_bytes = carve_build(c, L, face_count, q.tree_depth, true, true, (q.accel_trees & RT_ACCEL_CLUSTERS) != 0);
  if (max_nodes) *max_nodes = 2 * face_count - 1;
  return RT_OK;
}

extern "C" rt_status rt_lbvh_accel_bytes(uint32_t face_count, size_t* bytes) {
  if (!bytes || face_count == 0) return RT_ERR_INVALID_ARGUMENT;
  Carve c(nullptr, 0);
  AccelLayout A;
  *bytes = carve_accel(c, A, face_count);
  return RT_OK;
}

extern "C" rt_status rt_lbvh_build(const rt_build_desc* d, rt_stream stream_) {
  const rt::NvtxRange nvtx_range("rt_lbvh_build");
  if (!d || d->face_count == 0 || !d->vertices || !d->faces_in || !d->boxes || !d->indices || !d->nodes || d->max_nodes == 0)
    return RT_ERR_INVALID_ARGUMENT;
  if (d->face_count > 0x7FFFFFFFu) return RT_ERR_INVALID_ARGUMENT;
  const rt_build_params q = normalized(&d->params);
  if (q.morton_bits != 32 && q.morton_bits != 30) return RT_ERR_INVALID_ARGUMENT;
  const uint32_t n = d->face_count;
  // every size check comes before the first launch, so that a refused call leaves the caller's buffers untouched
  if (d->max_nodes < 2 * n - 1) return RT_ERR_CAPACITY;
  const bool complete = q.tree_complete != 0;
  const bool in_place = complete && d->faces_out && (d->faces_out == d->faces_in);
  Carve c(d->scratch, d->scratch_bytes);
  BuildLayout L;
  const bool clusters = (q.accel_trees & RT_ACCEL_CLUSTERS) != 0;
  if (clusters && (n > kClusterFirstMask || q.cluster_leaf > kClusterLeafMax)) return RT_ERR_UNSUPPORTED;
  carve_build(c, L, n, q.tree_depth, d->codes == nullptr, in_place, clusters);
  if (!d->scratch || !c.ok()) return RT_ERR_SCRATCH_TOO_SMALL;
  AccelLayout AL{};
  const bool accel = complete && d->accel && d->tris;
  if (accel) {
    Carve ca(d->accel, d->accel_bytes);
    carve_accel(ca, AL, n);
    if (!ca.ok()) return RT_ERR_SCRATCH_TOO_SMALL;
  }
  if (rt_device_check() != RT_OK) return RT_ERR_NO_DEVICE;
  cudaStream_t st = (cudaStream_t)stream_;
  uint32_t* codes = d->codes ? d->codes : L.codes;
  const int sms = sm_count();

  // 1. hit box
  if (cudaMemsetAsync(L.hit_done, 0, 8, st) != cudaSuccess) return RT_ERR_CUDA;
  if (d->hitbox) {
    float4 mn = make_float4(d->hitbox[0], d->hitbox[1], d->hitbox[2], d->hitbox[3]);
    float4 mx = make_float4(d->hitbox[4], d->hitbox[5], d->hitbox[6], d->hitbox[7]);
    k_set_hitbox<<<1, 1, 0, st>>>(L.hit, mn, mx);
    note_launch();
  } else {
    k_hitbox<<<kHitParts, 256, 0, st>>>((const float4*)d->vertices, d->vertex_count, L.partial, L.hit_done, L.hit);
    note_launch();
  }
  RT_CHECK_LAUNCH();
  // 2. boxes, codes
  {
    uint32_t blocks = (uint32_t)hmin<uint64_t>((n + 255) / 256, (uint64_t)sms * 16);
    k_boxes_morton<<<blocks, 256, 0, st>>>((const float4*)d->vertices, (const uint4*)d->faces_in, n, L.hit, (int)q.morton_bits,
                                           (float4*)d->boxes, codes, nullptr);
    note_launch();
    RT_CHECK_LAUNCH();
  }
  // 3. sort (code, index)
  // 4. per-level split lists
  if (cudaMemsetAsync(L.err, 0, 16, st) != cudaSuccess) return RT_ERR_CUDA;
  rt_status s = sort_codes_and_levels(codes, d->indices, n, L.C, L.lev_count, 256, L.sort_scratch, L.sort_bytes, st);
  if (s != RT_OK) return s;
  // 5. Morton top tree
  {
    TopoArgs A;
    A.C = L.C; A.lev_count = L.lev_count; A.n = n; A.D = q.tree_depth; A.min_leaf = q.min_leaf; A.max_leaf = q.max_leaf;
    A.complete = complete ? 1u : 0u; A.cap_m = L.cap_m;
    A.ra = L.ra; A.rb = L.rb; A.parent = L.parent; A.info = L.info; A.child = L.child; A.leaves = L.leaves; A.mleaves = L.mleaves;
    A.rank = L.rank; A.lambda = L.lambda; A.ord = L.ord; A.id = L.id;
    A.ml_lambda = L.ml_lambda; A.ml_rec = L.ml_rec; A.ml_rank = L.ml_rank; A.parent_id = L.parent_id;
    A.nodes = d->nodes; A.max_nodes = d->max_nodes; A.hdr = L.hdr;
    A.level_hist = nullptr; A.level_base = 0; A.pos_base = 0;
    if (!topo_smem_once(k_topo_morton, kTopoNodes)) return RT_ERR_CUDA;
    k_topo_morton<<<1, kTopoThreads, kTopoNodes * kTopoNodeBytes, st>>>(A);
    note_launch();
    RT_CHECK_LAUNCH();
  }
  // 6. leaves: median subtrees, reorder, triangles, boxes bottom-up
  {
    uint32_t count = d->max_nodes < L.max_nodes ? d->max_nodes : L.max_nodes;
    if (cudaMemsetAsync(L.arrive, 0, (size_t)count * 4, st) != cudaSuccess) return RT_ERR_CUDA;
    LeafArgs A;
    A.verts = (const float4*)d->vertices;
    A.faces_in = (const uint4*)d->faces_in;
    A.faces_out = complete && d->faces_out ? (in_place ? L.faces_tmp : (uint4*)d->faces_out) : nullptr;
    A.tris = complete ? (float4*)d->tris : nullptr;
    A.indices = d->indices; A.ml_lambda = L.ml_lambda; A.ml_rec = L.ml_rec; A.ml_rank = L.ml_rank; A.parent_id = L.parent_id;
    A.arrive = L.arrive; A.nodes = d->nodes; A.max_nodes = d->max_nodes; A.max_leaf = q.max_leaf; A.hdr = L.hdr; A.err = L.err;
    A.acc_leaves = accel ? AL.leaves : nullptr;
    A.acc_groups = accel ? AL.groups : nullptr;
    A.leaf_lambda = L.leaf_lambda;
    A.pos_base = 0;
    A.vert_base = 0;
    A.local_indices = nullptr;
    A.parent_cap = count;
    static const int leaf_blocks = resident_blocks_of(k_leaves, 256);
    k_leaves<<<(uint32_t)hmin<uint64_t>((uint64_t)sms * leaf_blocks, (n + 255) / 256), 256, 0, st>>>(A, n, L.hit_done + 1);
    note_launch();
    RT_CHECK_LAUNCH();
    // the node boxes and records (from the nodes) and the cluster tree (from the codes and triangles) are independent:
    // the node half runs on a side stream beside it (2^20 faces: 35 of 455 us). The header's valid word, which the
    // cluster tree sets, is cleared before they part.
    const bool cluster_tree = accel && clusters;
    if (accel && cudaMemsetAsync(AL.hdr + kHdrClusterValid, 0, 4, st) != cudaSuccess) return RT_ERR_CUDA;
    SideStream* side = cluster_tree ? side_stream(st) : nullptr;
    cudaStream_t ns = st;
    if (side) {
      if (cudaEventRecord(side->fork, st) != cudaSuccess || cudaStreamWaitEvent(side->s, side->fork, 0) != cudaSuccess)
        return RT_ERR_CUDA;
      ns = side->s;
    }
    k_propagate<<<sms * 8, 256, 0, ns>>>(d->nodes, L.parent_id, L.arrive, L.hdr, count);
    note_launch();
    RT_CHECK_LAUNCH();
    if (accel) {
      k_accel_nodes<<<sms * 4, 256, 0, ns>>>(d->nodes, L.hdr, L.leaf_lambda, AL.tnodes, AL.wide, AL.hdr);
      note_launch();
      RT_CHECK_LAUNCH();
    }
    if (cluster_tree) {
      s = build_cluster_tree((const float4*)d->tris, codes, n, q.cluster_leaf, L.ct, AL.hdr, AL.crec, st);
      if (side && (cudaEventRecord(side->join, side->s) != cudaSuccess || cudaStreamWaitEvent(st, side->join, 0) != cudaSuccess))
        return RT_ERR_CUDA;
      if (s != RT_OK) return s;
    }
  }
  if (in_place && cudaMemcpyAsync(d->faces_out, L.faces_tmp, (size_t)n * 16, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
    return RT_ERR_CUDA;
  if (d->info) {
    k_write_info<<<1, 32, 0, st>>>(L.hdr, L.err, d->info);
    note_launch();
    RT_CHECK_LAUNCH();
  }
  return RT_OK;
}

extern "C" rt_status rt_mesh_boxes(const float* vertices, const uint32_t* faces, uint32_t n, float* boxes, uint32_t* indices, rt_stream st) {
  if (n == 0) return RT_OK;
  if (!vertices || !faces || !boxes) return RT_ERR_INVALID_ARGUMENT;
  if (rt_device_check() != RT_OK) return RT_ERR_NO_DEVICE;
  uint32_t blocks = (uint32_t)hmin<uint64_t>((n + 255) / 256, (uint64_t)sm_count() * 16);
  k_boxes_morton<<<blocks, 256, 0, (cudaStream_t)st>>>((const float4*)vertices, (const uint4*)faces, n, nullptr, 32, (float4*)boxes,
                                                      nullptr, indices);
    note_launch();
  RT_CHECK_LAUNCH();
  return RT_OK;
}

namespace rt { namespace {
__global__ __launch_bounds__(256) void k_reorder(const uint4* __restrict__ in, const uint32_t* __restrict__ idx, uint32_t n, uint4* __restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = ldg4(in + __ldg(idx + i));
}
}}  // namespace rt

extern "C" rt_status rt_reorder_faces(const uint32_t* faces_in, const uint32_t* indices, uint32_t n, uint32_t* faces_out, rt_stream st) {
  if (n == 0) return RT_OK;
  if (!faces_in || !indices || !faces_out) return RT_ERR_INVALID_ARGUMENT;
  const char* a = (const char*)faces_in;
  const char* b = (const char*)faces_out;
  if (a < b + (size_t)n * 16 && b < a + (size_t)n * 16) return RT_ERR_INVALID_ARGUMENT;
  if (rt_device_check() != RT_OK) return RT_ERR_NO_DEVICE;
  uint32_t blocks = (uint32_t)hmin<uint64_t>((n + 255) / 256, (uint64_t)sm_count() * 16);
  k_reorder<<<blocks, 256, 0, (cudaStream_t)st>>>((const uint4*)faces_in, indices, n, (uint4*)faces_out);
    note_launch();
  RT_CHECK_LAUNCH();
  return RT_OK;
}

// ============================================================================
// Batched build: M meshes, every stage in one set of launches.
// ============================================================================
namespace rt {
namespace {


struct BatchArgs {
  uint32_t M, N;
  const uint32_t* foff;
  const uint32_t* voff;
  const float4* verts;
  const uint4* faces_in;
  uint4* faces_out;
  float4* boxes;
  uint32_t* indices_out;
  uint32_t* codes;
  uint32_t* nodes;
  float4* tris;
  rt_build_params q;
  // scratch
  float4* hits;           // [2M]
  float4* hitpart;        // [2 M kHitSplit]: the hit box shares of k_batch_hitbox
  uint32_t hit_split;     // shares per mesh, at most kHitSplit
  uint32_t* hitdone;      // [M]: finished shares per mesh
  uint32_t* idx;          // [N] global face index in sorted order
  uint32_t* C;            // [N] split positions
  uint32_t* hist;         // [M * 64]: split positions per mesh and level
  uint32_t *ra, *rb, *parent, *info, *child, *leaves, *mleaves, *rank, *lambda, *ord, *id;  // [2N + 3M]
  uint32_t* ml_lambda;
  uint4* ml_rec;
  uint32_t* ml_rank;
  uint32_t* parent_id;    // [2N - M]
  uint32_t* arrive;       // [2N - M]
  uint32_t* leaf_lambda;  // [2N - M]
  uint32_t* hdr;          // [16 M]
  uint32_t* leaf_base;    // [M + 1]
  uint32_t* err;          // [4]
  uint32_t* topo_done;    // finished topology CTAs, then the next leaf to hand out
  uint32_t* leaf_next;
  // traversal blob
  uint32_t* acc_hdr;      // [64 M]
  float4* tnodes;         // [4 N]
  uint4* acc_leaves;      // [N]
  float4* groups;         // [2 (N + N/8 + M + 1)]
  float4* wide;           // [8 N]
  float4* crec;           // cluster records (from F_m per mesh)
  ClusterTemps ct;        // cluster tree build temporaries (RT_ACCEL_CLUSTERS only)
  rt_build_info* info_out;
};

// Per-mesh hitbox: one 512-thread block per mesh, four loads in flight per
// thread (the largest meshes bound the launch).
__global__ __launch_bounds__(512) void k_batch_hitbox(BatchArgs B) {
  // `split` CTAs per mesh, each over its share of the mesh's vertices; the last of them combines the shares
  const uint32_t split = B.hit_split;
  const uint32_t m = blockIdx.x / split, part = blockIdx.x % split;
  const uint32_t w0 = B.voff[m], w1 = B.voff[m + 1], share = (w1 - w0 + split - 1) / split;
  const uint32_t v0 = min(w1, w0 + part * share), v1 = min(w1, v0 + share);
  if (part == 0 && threadIdx.x == 0) {
    B.acc_hdr[64 * (size_t)m + kHdrClusterValid] = 0;  // set again by the cluster build, if any
  }
  float4 mn[4], mx[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    mn[k] = make_float4(kHuge, kHuge, kHuge, kHuge);
    mx[k] = make_float4(-kHuge, -kHuge, -kHuge, -kHuge);
  }
  uint32_t i = v0 + threadIdx.x;
  for (; i + 3 * 512 < v1; i += 4 * 512) {
    float4 p[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) p[k] = ldg4(B.verts + i + k * 512);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mn[k] = f4min(mn[k], p[k]);
      mx[k] = f4max(mx[k], p[k]);
    }
  }
  for (; i < v1; i += 512) {
    const float4 p = ldg4(B.verts + i);
    mn[0] = f4min(mn[0], p);
    mx[0] = f4max(mx[0], p);
  }
  __shared__ float4 s_mn[512], s_mx[512];
  s_mn[threadIdx.x] = f4min(f4min(mn[0], mn[1]), f4min(mn[2], mn[3]));
  s_mx[threadIdx.x] = f4max(f4max(mx[0], mx[1]), f4max(mx[2], mx[3]));
  __syncthreads();
  if (threadIdx.x >= 32) return;  // (a barrier per step of the tree and eight CTAs a mesh: 118 us for 1024 meshes, now 73)
  // the first warp pairs the threads 256, 128, .. 1 apart: 16 values per lane, then the lanes
  float4 a[16], c[16];
#pragma unroll
  for (int w = 0; w < 16; ++w) { a[w] = s_mn[32 * w + threadIdx.x]; c[w] = s_mx[32 * w + threadIdx.x]; }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1)
#pragma unroll
    for (int w = 0; w < o; ++w) { a[w] = f4min(a[w], a[w + o]); c[w] = f4max(c[w], c[w + o]); }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    auto down = [&](const float4& v) {
      return make_float4(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o), __shfl_down_sync(0xffffffffu, v.z, o),
                         __shfl_down_sync(0xffffffffu, v.w, o));
    };
    a[0] = f4min(a[0], down(a[0]));
    c[0] = f4max(c[0], down(c[0]));
  }
  if (threadIdx.x == 0) {
    B.hitpart[2 * (size_t)blockIdx.x] = a[0];
    B.hitpart[2 * (size_t)blockIdx.x + 1] = c[0];
    __threadfence();
    // the mesh's last share to finish combines its shares in share order (an empty share holds +-huge
    // and changes nothing); nothing waits for it inside the launch
    if (atomicAdd(B.hitdone + m, 1u) == split - 1) {
      __threadfence();
      float4 lo = __ldcg(B.hitpart + 2 * (size_t)m * split), hi = __ldcg(B.hitpart + 2 * (size_t)m * split + 1);
      for (uint32_t p = 1; p < split; ++p) {
        lo = f4min(lo, __ldcg(B.hitpart + 2 * ((size_t)m * split + p)));
        hi = f4max(hi, __ldcg(B.hitpart + 2 * ((size_t)m * split + p) + 1));
      }
      B.hits[2 * m] = lo;
      B.hits[2 * m + 1] = hi;
    }
  }
}

// A warp takes 32 consecutive faces at a time and finds the first one's mesh together; the lanes of later meshes go on from
// there. (Runs of 256 faces with one search each left seven warps in eight of a small batch without work: 64 meshes of
// 1000 faces 7.5 us, now 3.2; and 10.8M faces in 512 meshes 165, now 158.)
__global__ __launch_bounds__(256) void k_batch_boxes_morton(BatchArgs B) {
  const int layout = (int)B.q.morton_bits;
  const uint32_t lane = lane_id();
  for (uint64_t first = (uint64_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; first < B.N; first += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t m = warp_last_le(B.foff, B.M, (uint32_t)first);
    const uint32_t k = (uint32_t)first + lane;
    if (k >= B.N) continue;
    const uint4 f = ldg4(B.faces_in + k);
    while (__ldg(B.foff + m + 1) <= k) ++m;
    const uint32_t vb = __ldg(B.voff + m);
    const float4 hmin = B.hits[2 * m], hmax = B.hits[2 * m + 1];
    const float sx = (layout == 30 ? 1023.0f : 2047.0f) / (hmax.x - hmin.x);
    const float sy = (layout == 30 ? 1023.0f : 2047.0f) / (hmax.y - hmin.y);
    const float sz = 1023.0f / (hmax.z - hmin.z);
    const float4 v0 = ldg4(B.verts + vb + f.x), v1 = ldg4(B.verts + vb + f.y), v2 = ldg4(B.verts + vb + f.z);
    const float4 mn = f4min(f4min(v0, v1), v2);
    const float4 mx = f4max(f4max(v0, v1), v2);
    B.boxes[2 * (size_t)k] = mn;
    B.boxes[2 * (size_t)k + 1] = mx;
    const float cx = 0.5f * (mn.x + mx.x), cy = 0.5f * (mn.y + mx.y), cz = 0.5f * (mn.z + mx.z);
    B.codes[k] = spread_code(f2u_sat((cx - hmin.x) * sx), f2u_sat((cy - hmin.y) * sy), f2u_sat((cz - hmin.z) * sz), layout);
  }
}

__global__ __launch_bounds__(kBatchTopoThreads, 3) void k_batch_topo(BatchArgs B) {
  extern __shared__ __align__(16) char topo_smem[];
  const uint32_t m = blockIdx.x;
  const uint32_t F = B.foff[m], n = B.foff[m + 1] - F;
  const uint32_t bb = bfs_base(F, m), nb = node_base(F, m);
  TopoArgs A;
  A.C = B.C; A.lev_count = nullptr; A.n = n; A.D = B.q.tree_depth; A.min_leaf = B.q.min_leaf; A.max_leaf = B.q.max_leaf;
  A.complete = 1u; A.cap_m = morton_cap_dev(n, B.q.tree_depth);
  A.ra = B.ra + bb; A.rb = B.rb + bb; A.parent = B.parent + bb; A.info = B.info + bb; A.child = B.child + bb;
  A.leaves = B.leaves + bb; A.mleaves = B.mleaves + bb; A.rank = B.rank + bb; A.lambda = B.lambda + bb; A.ord = B.ord + bb;
  A.id = B.id + bb; A.ml_lambda = B.ml_lambda + bb; A.ml_rec = B.ml_rec + bb; A.ml_rank = B.ml_rank + bb;
  A.parent_id = B.parent_id + nb; A.nodes = B.nodes + 8 * (size_t)nb; A.max_nodes = 2 * n - 1; A.hdr = B.hdr + 16 * m;
  // the meshes before m hold F positions, so this mesh's level lists start at F
  A.level_hist = B.hist + 64 * m; A.level_base = F; A.pos_base = F;
  if (!topo_shared<kBatchTopoThreads>(A, kBatchTopoNodes, topo_smem)) {
    __syncthreads();
    topo_morton<kBatchTopoThreads>(A);
  }
  // the CTA that finishes last (every other mesh's header is written) makes the leaf-order bases per mesh (an
  // exclusive scan of the leaf counts) and their total; nothing waits for it inside this kernel
  __shared__ uint32_t s_last;
  __shared__ uint32_t s_warp2[kBatchTopoThreads / 32];
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(B.topo_done, 1u) == B.M - 1 ? 1u : 0u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  uint32_t running = 0;
  for (uint32_t c = 0; c < B.M; c += kBatchTopoThreads) {
    const uint32_t i = c + threadIdx.x;
    const uint32_t bad = i < B.M ? (__ldcg(B.hdr + 16 * i + 8) & (RT_DEVERR_NODE_CAPACITY | RT_DEVERR_MORTON_CAPACITY)) : 0u;
    const uint32_t v = (i < B.M && !bad) ? __ldcg(B.hdr + 16 * i) : 0u;
    uint32_t tot;
    const uint32_t ex = block_excl_scan_nt<kBatchTopoThreads>(v, s_warp2, tot);
    if (i < B.M) B.leaf_base[i] = running + ex;
    running += tot;
  }
  if (threadIdx.x == 0) B.leaf_base[B.M] = running;
}

__global__ __launch_bounds__(256) void k_batch_leaves(BatchArgs B) {
  const uint32_t total = B.leaf_base[B.M];
  const uint32_t lane = lane_id();
  LeafArgs out = {};  // the whole build's arrays
  out.verts = B.verts; out.faces_in = B.faces_in; out.faces_out = B.faces_out; out.tris = B.tris; out.indices = B.idx;
  out.nodes = B.nodes; out.acc_groups = B.groups; out.local_indices = B.indices_out; out.err = B.err;
  const uint32_t run = leaf_run(total, B.N);
  for (;;) {
    const uint32_t g = next_run(B.leaf_next, run);
    if (g >= total) break;
    const bool have = lane < run && g + lane < total;
    const uint32_t m0 = warp_last_le(B.leaf_base, B.M, g);
    uint32_t m = m0;
    while (have && __ldg(B.leaf_base + m + 1) <= g + lane) ++m;
    const uint32_t F = B.foff[m], n = B.foff[m + 1] - F, bb = bfs_base(F, m), nb = node_base(F, m);
    LeafArgs A = {};
    A.ml_lambda = B.ml_lambda + bb; A.ml_rec = B.ml_rec + bb; A.ml_rank = B.ml_rank + bb;
    A.parent_id = B.parent_id + nb; A.nodes = B.nodes + 8 * (size_t)nb; A.max_nodes = 2 * n - 1;
    A.max_leaf = B.q.max_leaf; A.hdr = B.hdr + 16 * m; A.err = B.err;
    A.acc_leaves = B.acc_leaves + F; A.leaf_lambda = B.leaf_lambda + nb;
    A.pos_base = F; A.vert_base = B.voff[m]; A.parent_cap = 2 * n - 1;
    const uint32_t lg = g + lane - B.leaf_base[m];  // the leaf in its mesh
    uint32_t lo = 0;
    if (__all_sync(0xffffffffu, m == m0)) {
      lo = warp_morton_leaf(A, g - B.leaf_base[m]);
    } else if (have) {  // leaves of several meshes: each lane by itself
      uint32_t hi = A.hdr[1] - 1;
      while (lo < hi) {  // last k with ml_lambda[k] <= lg (non-decreasing)
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (A.ml_lambda[mid] <= lg) lo = mid; else hi = mid - 1;
      }
    }
    LeafMeta L = {};
    if (have) L = leaf_meta(A, lg, lo, nb, group_base(F, m));
    leaf_faces(out, L);
  }
}

// Mesh of item i of a list with base[m] items before mesh m's, for the 32 consecutive items of a warp (item = the first
// one's plus the lane; lanes without an item pass have = false): the first one's is found by the whole warp.
__device__ __forceinline__ uint32_t warp_mesh(const uint32_t* __restrict__ base, uint32_t M, uint32_t first, uint32_t item, bool have) {
  uint32_t m = warp_last_le(base, M, first);
  while (have && __ldg(base + m + 1) <= item) ++m;
  return m;
}

// Bottom-up boxes of every mesh: one thread per leaf, which climbs. (A thread per node slot, each with a search for its
// mesh, took 388 us for 1024 meshes of 9.9M faces, nine slots in ten unused; now 91, and the records 220 -> 104.)
__global__ __launch_bounds__(256) void k_batch_propagate(BatchArgs B) {
  const uint32_t total = B.leaf_base[B.M];
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total; base += gridDim.x * blockDim.x) {
    const uint32_t g = base + lane_id();
    const uint32_t m = warp_mesh(B.leaf_base, B.M, base, g, g < total);
    if (g >= total) continue;
    const uint32_t F = B.foff[m], n = B.foff[m + 1] - F, nb = node_base(F, m), cap = 2 * n - 1;
    const uint32_t leaf = __ldg(&B.acc_leaves[(size_t)F + g - B.leaf_base[m]].w);
    climb(B.nodes + 8 * (size_t)nb, B.parent_id + nb, B.arrive + nb, cap, leaf);
  }
}

// Traversal records of every mesh (two-child and 4-wide, per internal node) and each mesh's build info. A thread per
// leaf takes two nodes: leaf k the nodes 2k - 1 and 2k of its mesh's 2 leaves - 1.
__global__ __launch_bounds__(256) void k_batch_records(BatchArgs B) {
  const uint32_t total = B.leaf_base[B.M];
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total; base += gridDim.x * blockDim.x) {
    const uint32_t g = base + lane_id();
    const uint32_t m = warp_mesh(B.leaf_base, B.M, base, g, g < total);
    if (g >= total) continue;
    const uint32_t F = B.foff[m], nb = node_base(F, m), k = g - B.leaf_base[m];
    const uint32_t* h = B.hdr + 16 * m;
    if (k == 0) {
      uint32_t* ah = B.acc_hdr + 64 * m;
      ah[0] = (B.nodes[8 * (size_t)nb] & 1u) ? ~0u : 0u;
      ah[1] = h[0];
      ah[2] = h[2];
    }
    for (uint32_t p = k ? 2 * k - 1 : 0; p <= 2 * k; ++p)
      accel_wide_node(B.nodes + 8 * (size_t)nb, B.leaf_lambda + nb, B.tnodes + 4 * (size_t)F, B.wide + 8 * (size_t)F, p);
  }
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < B.M; m += gridDim.x * blockDim.x) {
    const uint32_t* h = B.hdr + 16 * m;
    rt_build_info* o = B.info_out + m;
    o->leaf_count = h[0]; o->node_count = h[2]; o->real_depth = h[3]; o->split_count = h[4];
    o->overrun_visits = h[5]; o->nondet_reads = h[6]; o->past_end_reads = h[7]; o->error = h[8] | *B.err;
  }
}

size_t batch_sort_bytes(uint32_t N, uint32_t M) { return hmax<size_t>(radix_scratch_bytes(N), segment_sort_scratch_bytes(N, M)); }

size_t carve_batch(Carve& c, BatchArgs& B, uint32_t M, uint32_t N, bool clusters) {
  B.hits = c.take<float4>(2 * (size_t)M);
  B.hitpart = c.take<float4>(2 * (size_t)M * kHitSplit);
  B.hitdone = c.take<uint32_t>(M);
  B.idx = c.take<uint32_t>(N);
  B.C = c.take<uint32_t>(N);
  B.hist = c.take<uint32_t>((size_t)M * 64);
  const size_t bfs = 2 * (size_t)N + 3 * (size_t)M + 4;
  uint32_t** arrs[] = {&B.ra, &B.rb, &B.parent, &B.info, &B.child, &B.leaves, &B.mleaves, &B.rank, &B.lambda, &B.ord, &B.id};
  for (auto a : arrs) *a = c.take<uint32_t>(bfs);
  B.ml_lambda = c.take<uint32_t>(bfs);
  B.ml_rec = c.take<uint4>(bfs);
  B.ml_rank = c.take<uint32_t>(bfs);
  const size_t nodes = 2 * (size_t)N;
  B.parent_id = c.take<uint32_t>(nodes);
  B.arrive = c.take<uint32_t>(nodes);
  B.leaf_lambda = c.take<uint32_t>(nodes);
  B.hdr = c.take<uint32_t>(16 * (size_t)M);
  B.leaf_base = c.take<uint32_t>((size_t)M + 1);
  B.err = c.take<uint32_t>(4);
  B.topo_done = c.take<uint32_t>(2);
  B.leaf_next = B.topo_done ? B.topo_done + 1 : nullptr;
  B.ct = ClusterTemps{};
  if (clusters) carve_cluster_temps(c, B.ct, N, M);
  const size_t sort_bytes = batch_sort_bytes(N, M);
  c.take<char>(sort_bytes);
  return c.off + 256;
}

size_t carve_batch_accel(Carve& c, BatchArgs& B, uint32_t M, uint32_t N) {
  BatchAccel L;
  const size_t bytes = carve_batch_accel_layout(c, L, M, N);
  B.acc_hdr = L.hdr; B.tnodes = L.tnodes; B.acc_leaves = L.leaves; B.groups = L.groups; B.wide = L.wide; B.crec = L.crec;
  return bytes;
}

}  // namespace
}  // namespace rt

extern "C" rt_status rt_batch_sizes(uint32_t M, uint32_t N, const rt_build_params* params, size_t* scratch_bytes, size_t* accel_bytes) {
  if (M == 0 || N < M || !scratch_bytes) return RT_ERR_INVALID_ARGUMENT;
  const rt_build_params q = normalized(params);
  Carve c(nullptr, 0);
  BatchArgs B;
  *scratch_bytes = carve_batch(c, B, M, N, (q.accel_trees & RT_ACCEL_CLUSTERS) != 0);
  if (accel_bytes) {
    Carve a(nullptr, 0);
    *accel_bytes = carve_batch_accel(a, B, M, N);
  }
  return RT_OK;
}

extern "C" rt_status rt_batch_build(const rt_batch_build_desc* d, rt_stream stream_) {
  const rt::NvtxRange nvtx_range("rt_batch_build");
  if (!d || d->mesh_count == 0 || d->face_count < d->mesh_count || !d->face_offsets || !d->vertex_offsets || !d->vertices ||
      !d->faces_in || !d->faces_out || !d->boxes || !d->indices || !d->codes || !d->nodes || !d->tris || !d->accel || !d->info)
    return RT_ERR_INVALID_ARGUMENT;
  if (d->faces_out == d->faces_in) return RT_ERR_INVALID_ARGUMENT;
  if (d->mesh_count > 65536u || d->face_count > 0x3FFFFFFFu) return RT_ERR_INVALID_ARGUMENT;
  rt_build_params q = normalized(&d->params);
  if (!q.tree_complete || (q.morton_bits != 32 && q.morton_bits != 30)) return RT_ERR_INVALID_ARGUMENT;
  const uint32_t M = d->mesh_count, N = d->face_count;
  const bool clusters = (q.accel_trees & RT_ACCEL_CLUSTERS) != 0;
  if (clusters && (N > kClusterFirstMask || q.cluster_leaf > kClusterLeafMax)) return RT_ERR_UNSUPPORTED;
  Carve c(d->scratch, d->scratch_bytes);
  BatchArgs B;
  carve_batch(c, B, M, N, clusters);
  if (!d->scratch || !c.ok()) return RT_ERR_SCRATCH_TOO_SMALL;
  // the sort scratch is the last region
  const size_t sort_bytes = batch_sort_bytes(N, M);
  void* sort_scratch = (char*)d->scratch + (c.off - sort_bytes - 0);
  {
    Carve a(d->accel, d->accel_bytes);
    carve_batch_accel(a, B, M, N);
    if (!a.ok()) return RT_ERR_SCRATCH_TOO_SMALL;
  }
  if (rt_device_check() != RT_OK) return RT_ERR_NO_DEVICE;
  B.M = M; B.N = N; B.foff = d->face_offsets; B.voff = d->vertex_offsets; B.verts = (const float4*)d->vertices;
  B.faces_in = (const uint4*)d->faces_in; B.faces_out = (uint4*)d->faces_out; B.boxes = (float4*)d->boxes;
  B.indices_out = d->indices; B.codes = d->codes; B.nodes = d->nodes; B.tris = (float4*)d->tris; B.q = q; B.info_out = d->info;
  cudaStream_t st = (cudaStream_t)stream_;
  const int sms = sm_count();
  const uint32_t fblocks = (uint32_t)hmin<uint64_t>((N + 255) / 256, (uint64_t)sms * 16);
  if (cudaMemsetAsync(B.err, 0, 16, st) != cudaSuccess) return RT_ERR_CUDA;
  if (cudaMemsetAsync(B.topo_done, 0, 8, st) != cudaSuccess) return RT_ERR_CUDA;
  if (cudaMemsetAsync(B.hist, 0, (size_t)M * 64 * 4, st) != cudaSuccess) return RT_ERR_CUDA;
  if (cudaMemsetAsync(B.hitdone, 0, (size_t)M * 4, st) != cudaSuccess) return RT_ERR_CUDA;
  // shares of the hit box: while the CTAs fit the chip at once (four an SM) a share of 1024 vertices is worth a CTA, beyond
  // that one of 8192 (on average: the largest meshes want more). By shares 1 / 2 / 4 / 8: 64 meshes of 1000 faces 5.6 / 5.1 /
  // 5.7 / 8.2 us, of 10,000 32 / 19 / 13 / 13, of 62,000 183 / 103 / 66 / 52; 256 of 1000 7 / 9 / 13 / 21, of 8000 41 / 34 /
  // 34 / 40, of 30,000 118 / 93 / 84 / 82; 1024 of 200 14 / 20 / 36 / 64, of 9000 98 / 92 / 102 / 135; 65,536 of 10
  // 0.67 / 1.16 / 2.19 / 4.16 ms.
  const uint64_t share = M * kHitSplit <= 4u * (uint32_t)sms ? 1024 : 8192;
  B.hit_split = 1;
  while (B.hit_split < kHitSplit && (uint64_t)d->vertex_count >= 2 * B.hit_split * share * M) B.hit_split *= 2;
  k_batch_hitbox<<<M * B.hit_split, 512, 0, st>>>(B);
  k_batch_boxes_morton<<<fblocks, 256, 0, st>>>(B);
  note_launch(2);
  RT_CHECK_LAUNCH();
  // every mesh's faces in Morton order (a mesh is a segment of the sort), then its split positions in level order
  rt_status s = sort_codes_and_levels(B.codes, B.idx, N, B.C, B.hist, 64, sort_scratch, sort_bytes, st, B.foff, M);
  if (s != RT_OK) return s;
  if (!topo_smem_once(k_batch_topo, kBatchTopoNodes)) return RT_ERR_CUDA;
  k_batch_topo<<<M, kBatchTopoThreads, kBatchTopoNodes * kTopoNodeBytes, st>>>(B);
  note_launch();
  RT_CHECK_LAUNCH();
  if (cudaMemsetAsync(B.arrive, 0, (2 * (size_t)N) * 4, st) != cudaSuccess) return RT_ERR_CUDA;
  static const int leaf_blocks = resident_blocks_of(k_batch_leaves, 256);
  k_batch_leaves<<<(uint32_t)hmin<uint64_t>((uint64_t)sms * leaf_blocks, (N + 255) / 256), 256, 0, st>>>(B);
  note_launch();
  RT_CHECK_LAUNCH();
  // the node boxes and records (from the nodes) and the cluster trees (from the codes and triangles) are
  // independent: with cluster trees, the node half runs on a side stream beside them
  SideStream* side = clusters ? side_stream(st) : nullptr;
  cudaStream_t ns = st;
  if (side) {
    if (cudaEventRecord(side->fork, st) != cudaSuccess || cudaStreamWaitEvent(side->s, side->fork, 0) != cudaSuccess)
      return RT_ERR_CUDA;
    ns = side->s;
  }
  k_batch_propagate<<<sms * 8, 256, 0, ns>>>(B);
  k_batch_records<<<sms * 4, 256, 0, ns>>>(B);
  note_launch(2);
  RT_CHECK_LAUNCH();
  if (clusters) {
    s = batch_build_cluster_tree(B.tris, B.codes, B.foff, M, N, q.cluster_leaf, B.ct, B.acc_hdr, B.crec, st);
    if (side && (cudaEventRecord(side->join, side->s) != cudaSuccess || cudaStreamWaitEvent(st, side->join, 0) != cudaSuccess))
      return RT_ERR_CUDA;
    if (s != RT_OK) return s;
  }
  return RT_OK;
}
