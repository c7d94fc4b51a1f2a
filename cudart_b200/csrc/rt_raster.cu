// rt_raster.cu -- the rasteriser (CUDA_rasterizeMeshTree,
// kernels/CUDA_rasterizeMeshTree.cu:77-297) on sm_100a.
//
// The reference runs 2 x 2 blocks of 8 x 4 threads over the whole screen,
// each block walking every face through a 192-face shared-memory cache. Here
// the work is binned instead: one thread per face transforms its vertices,
// drops faces off screen (and faces the barycentric test always rejects),
// computes the reference's zone rectangle and counts the zones of it that the
// face can touch (zone_touched); every face is appended to the lists of those
// zones (a counting sort: count, scan, fill); then one
// warp per 8 x 4 zone (lane = pixel, the reference's thread layout) walks its
// zone's faces, keeping depth / id / (u, v) in registers and taking the
// minimum (depth, face index). The per-pixel result is the reference's: the
// same tests on the same faces, and the face the reference's index-order walk
// with a strict depth test keeps. Faces are processed in chunks, in index
// order, whose pair count fits the scratch (a face can cover many zones); the
// surfaces carry the state across chunks.
#include <cstring>
#include <vector>

#include "../../include/rt_raster.h"
#include "rt_device.cuh"

namespace rt {
namespace {

constexpr float kRasterEps = 0.000001f;  // EPSILON, :31
constexpr uint32_t kFacesPerBlock = 128;  // granularity of the chunking
constexpr uint32_t kMinPairCap = 16u << 20;

struct Mat4 {
  float4 r0, r1, r2, r3;
};

__device__ __forceinline__ float dot4(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }

// matrixTransform, then /= |w| (a multiply by the reciprocal), w = 0 (:112-117)
__device__ __forceinline__ float4 project(const Mat4& m, float4 v) {
  v.w = 1.0f;
  float4 o = make_float4(dot4(m.r0, v), dot4(m.r1, v), dot4(m.r2, v), dot4(m.r3, v));
  const float inv = 1.0f / fabsf(o.w);
  o = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
  o.w = 0.0f;
  return o;
}

struct Zones {
  int zcx, zcy;
  float zsx, zsy;  // zone_scale = 0.5 * zone_count (:94-95)
};

// The pixel rectangle of a screen in device coordinates, as the zone pass computes them.
struct Screen {
  int zcx;
  float w, h;
};
__device__ __forceinline__ float pixel_x(int x, const Screen& S) { return (float)x * 2.0f / S.w - 1.0f; }
__device__ __forceinline__ float pixel_y(int y, const Screen& S) { return 1.0f - (float)y * 2.0f / S.h; }

// Whether some pixel of a zone may pass the zone pass's test of a face: false only where u, v or u + v stay outside
// [0, 1] at every pixel of the zone. The three are affine in the pixel (taken from the face's first vertex here), so
// over a zone they stay within r of their value at its centre. `m` bounds what rounding changes, in the pixel's test and
// in this one: a handful of roundings of 2^-24 on products below d^2, and pixel positions known to 2e-7, d being the
// largest distance from the first vertex; with a factor of five to spare. NaN and infinities compare false: the pair is
// kept. A rectangle starts on an even zone and a triangle fills half of it at the most: of the 2^20-face soup's 24M
// (zone, face) pairs at 1080p under half are left, and the zone pass takes 0.75 ms instead of 1.50.
struct ZoneTest {
  float kx, ky, dx, dy;  // the zone's centre less the first vertex: kx + i dx, ky + j dy
  float ux, uy, vx, vy;  // gradients
  float ulo, uhi, vlo, shi;
};
__device__ __forceinline__ ZoneTest zone_test(const float4& a, const float4& b, const float4& c, const int4& r, const Screen& S) {
  ZoneTest t;
  const float sx = 2.0f / S.w, sy = 2.0f / S.h, hx = 3.5f * sx, hy = 1.5f * sy;
  t.dx = 8.0f * sx;
  t.dy = -4.0f * sy;
  t.kx = (hx - 1.0f) - a.x;
  t.ky = (1.0f - hy) - a.y;
  const float bx = b.x - a.x, by = b.y - a.y, cx = c.x - a.x, cy = c.y - a.y, inv = a.w;
  t.ux = cy * inv; t.uy = -cx * inv; t.vx = -by * inv; t.vy = bx * inv;
  const float x0 = fabsf(t.kx + (float)r.x * t.dx) + hx, x1 = fabsf(t.kx + (float)r.z * t.dx) + hx;
  const float y0 = fabsf(t.ky + (float)r.y * t.dy) + hy, y1 = fabsf(t.ky + (float)r.w * t.dy) + hy;
  const float d = fmaxf(fmaxf(fmaxf(x0, x1), fmaxf(y0, y1)), fmaxf(fmaxf(fabsf(bx), fabsf(by)), fmaxf(fabsf(cx), fabsf(cy))));
  const float m = (4e-6f * d + 2e-6f) * d * fabsf(inv) + 1e-5f;
  const float ru = fabsf(t.ux) * hx + fabsf(t.uy) * hy, rv = fabsf(t.vx) * hx + fabsf(t.vy) * hy;
  const float rs = fabsf(t.ux + t.vx) * hx + fabsf(t.uy + t.vy) * hy;
  t.ulo = -m - ru; t.uhi = 1.0f + m + ru; t.vlo = -m - rv; t.shi = 1.0f + m + rs;
  return t;
}
__device__ __forceinline__ bool zone_touched(const ZoneTest& t, int i, int j) {
  const float x = __fmaf_rn((float)i, t.dx, t.kx), y = __fmaf_rn((float)j, t.dy, t.ky);
  const float u = __fmaf_rn(x, t.ux, y * t.uy), v = __fmaf_rn(x, t.vx, y * t.vy);
  return !(u < t.ulo || u > t.uhi || v < t.vlo || u + v > t.shi);
}

// Calls use(owner lane, zone) for every zone of the faces' rectangles that they may touch: a lane its own face's, or the
// whole warp one lane's face after another where the rectangle has more than kOwnZones zones. Returns the number of
// zones of the lane's own face.
constexpr uint32_t kOwnZones = 64;
template <class Use>
__device__ __forceinline__ uint32_t for_touched_zones(bool have, const float4& a, const float4& b, const float4& c, const int4& r,
                                                      const Screen& S, const Use& use) {
  const uint32_t lane = lane_id();
  const uint32_t n = have ? (uint32_t)(r.z - r.x + 1) * (uint32_t)(r.w - r.y + 1) : 0u;
  uint32_t count = 0;
  ZoneTest t = {};
  if (n) t = zone_test(a, b, c, r, S);
  if (n && n <= kOwnZones) {
    for (int j = r.y; j <= r.w; ++j)
      for (int i = r.x; i <= r.z; ++i)
        if (zone_touched(t, i, j)) {
          use(lane, (uint32_t)(j * S.zcx + i));
          ++count;
        }
  }
  for (uint32_t big = __ballot_sync(0xffffffffu, n > kOwnZones); big; big &= big - 1u) {
    const int o = __ffs(big) - 1;
    const uint32_t on = __shfl_sync(0xffffffffu, n, o);
    const int x0 = __shfl_sync(0xffffffffu, r.x, o), y0 = __shfl_sync(0xffffffffu, r.y, o), x1 = __shfl_sync(0xffffffffu, r.z, o);
    ZoneTest q;
    const float* from = (const float*)&t;
    float* to = (float*)&q;
#pragma unroll
    for (int k = 0; k < (int)(sizeof(ZoneTest) / 4); ++k) to[k] = __shfl_sync(0xffffffffu, from[k], o);
    const uint32_t w = (uint32_t)(x1 - x0 + 1);
    uint32_t mine = 0;
    for (uint32_t k = lane; k < on; k += 32) {
      const int i = x0 + (int)(k % w), j = y0 + (int)(k / w);
      if (zone_touched(q, i, j)) {
        use((uint32_t)o, (uint32_t)(j * S.zcx + i));
        ++mine;
      }
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if ((int)lane == o) count = mine;
  }
  return count;
}

// Per face: projected vertices, the zone rectangle (x0, y0, x1, y1) and the
// number of zones it may touch (0 when dropped); also every zone's count over
// all faces (zcount), which serves if the pairs fit one chunk. Faces naming a
// vertex past the mesh are skipped with an error bit.
__global__ __launch_bounds__(kFacesPerBlock) void k_raster_setup(const float4* __restrict__ verts, uint32_t vcount,
                                                                 const uint4* __restrict__ faces, uint32_t n, Mat4 M, Zones Z, Screen S,
                                                                 float4* __restrict__ tri, int4* __restrict__ rect,
                                                                 uint32_t* __restrict__ cnt, uint32_t* __restrict__ block_sum,
                                                                 uint32_t* __restrict__ zcount, unsigned long long* __restrict__ total,
                                                                 uint32_t* err) {
  __shared__ uint32_t s_sum;
  if (threadIdx.x == 0) s_sum = 0;
  __syncthreads();
  const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
  bool have = false;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, cc = a;
  int4 r = make_int4(0, 0, -1, -1);
  if (f < n) {
    const uint4 fc = __ldg(faces + f);
    if (fc.x >= vcount || fc.y >= vcount || fc.z >= vcount) {
      atomicOr(err, (uint32_t)RT_DEVERR_NODE_CAPACITY);
    } else {
      a = project(M, __ldg(verts + fc.x));
      b = project(M, __ldg(verts + fc.y));
      cc = project(M, __ldg(verts + fc.z));
      // the face's determinant (intersectTriPoint, :52-71, the same arithmetic as the
      // zone pass would do per pixel): a face the test always rejects gets no zone
      // pairs; otherwise its reciprocal rides in a.w
      const float det = (b.x - a.x) * (cc.y - a.y) - (cc.x - a.x) * (b.y - a.y);
      const bool degenerate = det > -kRasterEps && det < kRasterEps;
      a.w = degenerate ? 0.0f : 1.0f / det;
      // a depth that no point of the face lies below, as the zone pass computes them: its weights are within 2^-22 of
      // convex and its sum rounds five times, together less than half of 2^-20 of the largest depth
      cc.w = fminf(fminf(a.z, b.z), cc.z) - 9.5367431640625e-7f * fmaxf(fmaxf(fabsf(a.z), fabsf(b.z)), fabsf(cc.z));
      tri[3 * (size_t)f] = a;
      tri[3 * (size_t)f + 1] = b;
      tri[3 * (size_t)f + 2] = cc;
      const float mnx = fminf(fminf(fminf(kHuge, a.x), b.x), cc.x), mny = fminf(fminf(fminf(kHuge, a.y), b.y), cc.y);
      const float mxx = fmaxf(fmaxf(fmaxf(-kHuge, a.x), b.x), cc.x), mxy = fmaxf(fmaxf(fmaxf(-kHuge, a.y), b.y), cc.y);
      // intersectRectRect with [-1, 1]^2 (:47-50, :150)
      if (!degenerate && mnx < 1.0f && mxx > -1.0f && mny < 1.0f && mxy > -1.0f) {
        const int x0 = max(__float2int_rz(Z.zsx * (mnx + 1.0f)), 0) / 2 * 2;
        const int y0 = max(__float2int_rz(Z.zsy * (1.0f - mxy)), 0) / 2 * 2;
        const int x1 = min(__float2int_rz(Z.zsx * (mxx + 1.0f)), Z.zcx - 1);
        const int y1 = min(__float2int_rz(Z.zsy * (1.0f - mny)), Z.zcy - 1);
        r = make_int4(x0, y0, x1, y1);
        have = x1 >= x0 && y1 >= y0;
        if (have) rect[f] = r;
      }
    }
  }
  const uint32_t c = for_touched_zones(have, a, b, cc, r, S, [&](uint32_t, uint32_t z) { atomicAdd(zcount + z, 1u); });
  if (f < n) cnt[f] = c;
  // per block of kFacesPerBlock faces (= blockDim) the pair count, for the host's chunking
  atomicAdd(&s_sum, c);
  __syncthreads();
  if (threadIdx.x == 0) {
    block_sum[blockIdx.x] = s_sum;
    if (s_sum) atomicAdd(total, (unsigned long long)s_sum);
  }
}

// Launches that were made before the host knew the frame's pair count do nothing when it is above what the pair buffer
// holds, or nought (total null: the host knows that there are some and that they fit). A mesh without pairs is one off
// the screen or finer than the determinant's threshold: 4.5M such faces at 7680 x 4320 281 us with the zones walked, 202
// without, 229 when the host waited for the count first.
struct PairLimit {
  const unsigned long long* total;
  unsigned long long cap;
  __device__ __forceinline__ bool passed() const { return total && (*total > cap || *total == 0); }
};

// The (zone, face) pairs of faces [f0, f1) binned by zone without a sort: the zones' counts (from k_raster_setup when
// the chunk is the whole mesh, else from k_raster_bin<false>) are turned into list starts by an exclusive scan, and
// k_raster_bin<true> appends every face to its zones' lists. The order inside a list is whatever the atomics give; the
// zone pass takes the minimum (depth, face index), which is what visiting the faces in index order with a strict depth
// test keeps.
template <bool kFill>
__global__ __launch_bounds__(256) void k_raster_bin(const float4* __restrict__ tri, const int4* __restrict__ rect,
                                                    const uint32_t* __restrict__ cnt, uint32_t f0, uint32_t f1, Screen S,
                                                    const uint32_t* __restrict__ zoff, uint32_t* __restrict__ zcount,
                                                    uint32_t* __restrict__ vals, PairLimit limit) {
  if (limit.passed()) return;
  // whole warps step together: a face with many zones is shared by its warp
  for (uint32_t base = f0 + blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < f1; base += gridDim.x * blockDim.x) {
    const uint32_t f = base + lane_id();
    const bool have = f < f1 && cnt[f] != 0u;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, c = a;
    int4 r = make_int4(0, 0, -1, -1);
    if (have) {
      a = __ldg(tri + 3 * (size_t)f); b = __ldg(tri + 3 * (size_t)f + 1); c = __ldg(tri + 3 * (size_t)f + 2);
      r = rect[f];
    }
    // four zones at a time: their atomics are in flight together before the stores
    uint32_t held = 0, hz[4], ho[4];
    auto flush = [&]() {
      uint32_t k[4];
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q)
        if (q < held) k[q] = zoff[hz[q]] + atomicAdd(zcount + hz[q], 1u);
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q)
        if (q < held) vals[k[q]] = base + ho[q];
      held = 0;
    };
    for_touched_zones(have, a, b, c, r, S, [&](uint32_t owner, uint32_t z) {
      if (!kFill) {
        atomicAdd(zcount + z, 1u);
      } else {
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
          if (q == held) { hz[q] = z; ho[q] = owner; }
        if (++held == 4) flush();
      }
    });
    if (kFill && held) flush();
  }
}

// One warp per zone; lane = pixel (x = lane % 8, y = lane / 8 inside the zone). The zone's faces are taken 32 at a time,
// one per lane, and those whose nearest depth lies behind the zone's farthest pixel so far go at once; the others are
// tested by the whole warp. 2^20 faces of a soup at 1920 x 1080: 754 us with a test of every face, now 556, by issue
// slots (74%) and the loads' wavefronts. (Taking the nearest of the 32 first: 620.)
__global__ __launch_bounds__(256) void k_raster_zones(const float4* __restrict__ tri, const uint32_t* __restrict__ vals,
                                                      const uint32_t* __restrict__ zs, const uint32_t* __restrict__ ze, uint32_t nz, PairLimit limit,
                                                      Screen S, int width, int height, uint32_t id_mode, int32_t* __restrict__ fid,
                                                      float2* __restrict__ uv, float* __restrict__ depth) {
  if (limit.passed()) return;
  const uint32_t lane = threadIdx.x & 31u;
  const int zcx = S.zcx;
  for (uint32_t z = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; z < nz; z += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t s = zs[z], e = ze[z];
    if (s >= e) continue;
    const int x = (int)(z % (uint32_t)zcx) * 8 + (int)(lane & 7u);
    const int y = (int)(z / (uint32_t)zcx) * 4 + (int)(lane >> 3);
    const bool inside = x >= 0 && x < width && y >= 0 && y < height;
    const size_t l = (size_t)y * (size_t)width + (size_t)x;
    const float px = pixel_x(x, S), py = pixel_y(y, S);
    float best = inside ? depth[l] : 0.0f;
    int32_t bf = -1;
    float bu = 0.0f, bv = 0.0f;
    // the zone's farthest depth so far; as integers, since a pixel whose depth is not positive takes no face at all
    float far = 0.0f;
    auto farthest = [&] { far = __int_as_float(__reduce_max_sync(0xffffffffu, inside ? __float_as_int(best) : (int)0x80000000)); };
    farthest();
    uint32_t f32 = 0;
    float lo32 = 0.0f;
    auto load32 = [&](uint32_t p) {  // a face per lane, and its nearest depth (c.w)
      if (p >= e) return;
      f32 = __ldg(vals + p);
      lo32 = __ldg(&tri[3 * (size_t)f32 + 2].w);
    };
    load32(s + lane);
    for (uint32_t p = s; p < e; p += 32) {
      const uint32_t mine = f32;
      const float lo = lo32;
      uint32_t todo = __ballot_sync(0xffffffffu, p + lane < e && !(lo > far));
      load32(p + 32 + lane);
      while (todo) {
        const uint32_t f = __shfl_sync(0xffffffffu, mine, __ffs((int)todo) - 1);
        todo &= todo - 1u;
        const float4 a = __ldg(tri + 3 * (size_t)f), b = __ldg(tri + 3 * (size_t)f + 1), c = __ldg(tri + 3 * (size_t)f + 2);
        // intersectTriPoint (:52-71); the face setup pass computed 1 / det (a.w) and
        // emitted no pairs for faces with |det| below the threshold
        const float inv_det = a.w;
        const float u = ((c.x - px) * (a.y - py) - (a.x - px) * (c.y - py)) * inv_det;
        const float v = ((a.x - px) * (b.y - py) - (b.x - px) * (a.y - py)) * inv_det;
        bool won = false;
        if (!(u < 0.0f || u > 1.0f) && !(v < 0.0f || u + v > 1.0f)) {
          const float t = (1.0f - u - v) * a.z + u * b.z + v * c.z;
          // the earliest face wins a depth tie: faces arrive in any order, and the
          // depth of an earlier chunk (bf < 0) is only beaten by a strictly nearer face
          if (inside && t > 0 && (t < best || (t == best && bf >= 0 && (int32_t)f < bf))) {
            best = t;
            bf = (int32_t)f;
            bu = u;
            bv = v;
            won = true;
          }
        }
        if (__any_sync(0xffffffffu, won)) {
          farthest();
          todo &= __ballot_sync(0xffffffffu, !(lo > far));
        }
      }
    }
    if (bf >= 0) {
      fid[l] = id_mode == 1 ? bf - bf % 192 : bf;
      uv[l] = make_float2(bu, bv);
      depth[l] = best;
    }
  }
}

int sm_count_r() {
  int dev = 0, n = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

Zones zones_of(uint32_t width, uint32_t height) {
  Zones Z;
  Z.zcx = 1 + ((int)width - 1) / 8;
  Z.zcy = 1 + ((int)height - 1) / 4;
  Z.zsx = 0.5f * (float)Z.zcx;
  Z.zsy = 0.5f * (float)Z.zcy;
  return Z;
}

struct RasterLayout {
  float4* tri;
  int4* rect;
  uint32_t *cnt, *block_sum, *vals, *zoff, *zfill, *zsums, *err;
  unsigned long long* total;  // pairs of the frame
  uint32_t cap;
};

size_t carve_raster(Carve& c, RasterLayout& L, uint32_t n, uint32_t width, uint32_t height, uint32_t pair_capacity) {
  const Zones Z = zones_of(width, height);
  const uint64_t nz = (uint64_t)Z.zcx * (uint64_t)Z.zcy;
  uint64_t cap = pair_capacity ? pair_capacity : kMinPairCap;
  if (cap < (uint64_t)kFacesPerBlock * nz) cap = (uint64_t)kFacesPerBlock * nz;  // one block of faces always fits
  L.cap = (uint32_t)(cap > 0x7FFFFFFFull ? 0x7FFFFFFFull : cap);
  L.tri = c.take<float4>(3 * (size_t)n);
  L.rect = c.take<int4>(n);
  L.cnt = c.take<uint32_t>(n);
  L.block_sum = c.take<uint32_t>(n / kFacesPerBlock + 1);
  L.vals = c.take<uint32_t>(L.cap);
  L.zoff = c.take<uint32_t>(nz + 1);
  L.total = c.take<unsigned long long>(1);
  L.zfill = c.take<uint32_t>(nz);
  L.zsums = c.take<uint32_t>(nz / 1024 + 2);
  L.err = c.take<uint32_t>(1);
  return c.off + 256;
}

}  // namespace
}  // namespace rt

using namespace rt;

extern "C" rt_status rt_raster_scratch_bytes(uint32_t face_count, uint32_t width, uint32_t height, uint32_t pair_capacity, size_t* bytes) {
  if (!bytes || face_count == 0 || width == 0 || height == 0 || face_count > 0x7FFFFFFFu) return RT_ERR_INVALID_ARGUMENT;
  Carve c(nullptr, 0);
  RasterLayout L;
  *bytes = carve_raster(c, L, face_count, width, height, pair_capacity);
  return RT_OK;
}

extern "C" rt_status rt_rasterize(const rt_raster_desc* d, rt_stream stream) {
  if (!d || !d->vertices || !d->faces || !d->face_id || !d->uv || !d->depth || d->width == 0 || d->height == 0 || d->id_mode > 1)
    return RT_ERR_INVALID_ARGUMENT;
  if (rt_device_check() != RT_OK) return RT_ERR_NO_DEVICE;
  if (d->face_count == 0) return RT_OK;
  size_t need = 0;
  rt_raster_scratch_bytes(d->face_count, d->width, d->height, d->pair_capacity, &need);
  if (!d->scratch || d->scratch_bytes < need) return RT_ERR_SCRATCH_TOO_SMALL;
  cudaStream_t st = (cudaStream_t)stream;
  const uint32_t n = d->face_count;
  Carve c(d->scratch, d->scratch_bytes);
  RasterLayout L;
  carve_raster(c, L, n, d->width, d->height, d->pair_capacity);
  const Zones Z = zones_of(d->width, d->height);
  const uint32_t nz = (uint32_t)Z.zcx * (uint32_t)Z.zcy;
  Mat4 M;
  memcpy(&M, d->matrix, 64);
  uint32_t* err = d->error_word ? d->error_word : L.err;
  if (!d->error_word && cudaMemsetAsync(L.err, 0, 4, st) != cudaSuccess) return RT_ERR_CUDA;
  const Screen S{Z.zcx, (float)(int)d->width, (float)(int)d->height};
  const uint32_t nblocks = (n + kFacesPerBlock - 1) / kFacesPerBlock;
  if (cudaMemsetAsync(L.zoff, 0, ((size_t)nz + 1) * 4, st) != cudaSuccess || cudaMemsetAsync(L.total, 0, 8, st) != cudaSuccess)
    return RT_ERR_CUDA;
  k_raster_setup<<<nblocks, kFacesPerBlock, 0, st>>>((const float4*)d->vertices, d->vertex_count, (const uint4*)d->faces, n, M, Z, S,
                                                      L.tri, L.rect, L.cnt, L.block_sum, L.zoff, L.total, err);
  note_launch();
  RT_CHECK_LAUNCH();
  const int sms = sm_count_r();
  // zone lists and zone pass of faces [f0, f1), whose zone counts stand in zoff
  auto chunk = [&](uint32_t f0, uint32_t f1, PairLimit limit) {
    if (cudaMemsetAsync(L.zfill, 0, (size_t)nz * 4, st) != cudaSuccess) return RT_ERR_CUDA;
    const uint32_t fblocks = (uint32_t)hmin<uint64_t>((f1 - f0 + 255) / 256, (uint64_t)sms * 8);
    excl_scan(L.zoff, nz + 1, L.zsums, nullptr, st);
    k_raster_bin<true><<<fblocks, 256, 0, st>>>(L.tri, L.rect, L.cnt, f0, f1, S, L.zoff, L.zfill, L.vals, limit);
    note_launch();
    RT_CHECK_LAUNCH();
    k_raster_zones<<<(uint32_t)hmin<uint64_t>(((uint64_t)nz * 32 + 255) / 256, (uint64_t)sms * 16), 256, 0, st>>>(
        L.tri, L.vals, L.zoff, L.zoff + 1, nz, limit, S, (int)d->width, (int)d->height, d->id_mode, d->face_id, (float2*)d->uv, d->depth);
    note_launch();
    RT_CHECK_LAUNCH();
    return RT_OK;
  };
  // Most frames fit the pair buffer: the whole frame is launched as one chunk that does nothing if it does not fit, and
  // the pair count is read beside it on a side stream, so that the host's wait for it is no gap on the device (2^20
  // faces 1020 -> 965 us, of 2394 before this file's other changes).
  SideStream* side = side_stream(st);
  cudaStream_t rs = side ? side->s : st;
  if (side && (cudaEventRecord(side->fork, st) != cudaSuccess || cudaStreamWaitEvent(side->s, side->fork, 0) != cudaSuccess)) return RT_ERR_CUDA;
  rt_status s = chunk(0, n, PairLimit{L.total, L.cap});
  if (s != RT_OK) return s;
  unsigned long long total = 0;
  if (cudaMemcpyAsync(&total, L.total, 8, cudaMemcpyDeviceToHost, rs) != cudaSuccess || cudaStreamSynchronize(rs) != cudaSuccess)
    return RT_ERR_CUDA;
  if (total <= L.cap) return RT_OK;
  std::vector<uint32_t> bsum(nblocks);
  if (cudaMemcpyAsync(bsum.data(), L.block_sum, (size_t)nblocks * 4, cudaMemcpyDeviceToHost, rs) != cudaSuccess ||
      cudaStreamSynchronize(rs) != cudaSuccess)
    return RT_ERR_CUDA;
  uint32_t b = 0;
  while (b < nblocks) {
    // the longest run of face blocks whose pairs fit the pair buffer
    uint64_t P = 0;
    uint32_t e = b;
    while (e < nblocks && P + bsum[e] <= L.cap) P += bsum[e++];
    if (e == b) return RT_ERR_CAPACITY;  // cannot happen: one block's pairs always fit
    const uint32_t f0 = b * kFacesPerBlock, f1 = e * kFacesPerBlock < n ? e * kFacesPerBlock : n;
    b = e;
    if (P == 0) continue;
    if (cudaMemsetAsync(L.zoff, 0, ((size_t)nz + 1) * 4, st) != cudaSuccess) return RT_ERR_CUDA;
    k_raster_bin<false><<<(uint32_t)hmin<uint64_t>((f1 - f0 + 255) / 256, (uint64_t)sms * 8), 256, 0, st>>>(L.tri, L.rect, L.cnt, f0, f1, S,
                                                                                                        nullptr, L.zoff, nullptr, PairLimit{});
    note_launch();
    RT_CHECK_LAUNCH();
    s = chunk(f0, f1, PairLimit{});
    if (s != RT_OK) return s;
  }
  return RT_OK;
}
