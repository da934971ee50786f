// Trace kernels: the k-closest-hit forward pass and its adjoint.
//
// Replaces the reference's OptiX programs tritracer/forward.cu (raygen
// :161-215, chunk loop :76-155), tritracer/closestk.h (k-closest query) and
// tritracer/backward.cu (adjoint :191-391).
//
// Shape of the kernels:
//  * persistent: every warp pulls 8x4-pixel tiles from an atomic counter until
//    the image is done, so rays of very different depth complexity balance;
//  * one ray per thread. Warp packets walk the BVH together for the frustum
//    around their rays; independent lanes each keep a traversal stack (node
//    reference + entry distance) in shared memory, strided by the block size
//    (no bank conflicts);
//  * k-buffer: the k nearest (t, primitive) pairs packed as 64-bit keys in
//    shared memory (one column per lane): sorted by insertion as hits arrive
//    (lanes), or filled in any order and sorted at the end (packets);
//  * the chunked march of the reference is reproduced exactly on top of the
//    key stream: after every 16th visited hit the next query starts AT the
//    last hit's t (closed interval, optixTrace) or strictly after it;
//  * per hit, the window function runs in FP64 from the plane intersection
//    (the FP32 hit point loses ~4 digits on small triangles far from the
//    camera); SH, compositing and the side outputs are FP32 like the
//    reference; the adjoint re-traverses instead of storing hit lists.
#include <algorithm>
#include <cfloat>

#include "trace.cuh"

namespace tt {
namespace {

constexpr int kMaxChunks = 1 << 20;   // bound on re-traces per ray
constexpr int kMaxSteps = 1 << 24;    // bound on stack pops per query
// Resident blocks per SM the register budget must allow: 4 x 128 threads
// leave 128 registers a thread. Measured on 1M triangles, 4 x 800^2 rays,
// packets of 32: forward 19.0 / adjoint 21.6 ms at 4 blocks, 20.5 / 23.2 at
// 5 (96 registers, ~300 bytes of spills a thread), 21.8 / 24.9 at 6; later,
// with the forward at 18.2 ms at 4 blocks, 19.9 at 3 (168 registers, no
// spills, 12 warps per SM).
#ifndef TT_MIN_BLOCKS
#define TT_MIN_BLOCKS 4
#endif
constexpr int kMinBlocks = TT_MIN_BLOCKS;

// Per-lane traversal stack: the top SD entries in shared memory (strided by
// the block size, conflict-free), continued in thread-local memory for deep
// trees (only touched when the shared part is full).
constexpr int kLaneStack = 96;
struct Stack {
  uint32_t* ref;
  float* tn;
  int stride;
  __device__ __forceinline__ void put(int i, uint32_t r, float t) {
    ref[i * stride] = r;
    tn[i * stride] = t;
  }
};

// Sorted insert into the lane's k-buffer in shared memory (hits are rare
// next to box tests, so the buffer need not occupy 32 registers). `n` counts
// the valid keys (the slots from n on hold kEmptyKey): the insert shifts only
// the valid keys above the new one, not the empty tail, and once the buffer
// is full the largest key drops out. Returns true when the buffer is full
// after the insert (its last key then bounds the query).
template <int K>
__device__ __forceinline__ bool kb_insert_smem(unsigned long long* kb, int stride, unsigned long long key, int& n) {
  int i = n < K ? n : K - 1;
  while (i > 0) {
    const unsigned long long prev = kb[(i - 1) * stride];
    if (prev <= key) break;
    kb[i * stride] = prev;
    --i;
  }
  kb[i * stride] = key;
  if (n < K) ++n;
  return n == K;
}

// A candidate key enters a k-buffer holding n valid keys iff the buffer has
// room or the key is below its largest key.
template <int K>
__device__ __forceinline__ bool kb_accepts(const unsigned long long* kb, int stride, unsigned long long key, int n) {
  return n < K || key < kb[(K - 1) * stride];
}


struct Counters {
  unsigned nodes = 0, tris = 0, queries = 0, warp_nodes = 0;
  unsigned cont = 0, restart = 0;  // proposed intervals left by continuation / re-trace
  unsigned replays = 0;            // queries taken from the hit cache (adjoint)
  __device__ __forceinline__ void add_cont() { ++cont; }
  __device__ __forceinline__ void add_restart() { ++restart; }
};

// The packet drivers keep their counters in per-warp shared-memory words
// instead (warp-uniform updates by lane 0, shared atomics for the rare
// per-lane events), so the traversal carries no counter registers; they are
// folded into the thread's Counters when the warp is done.
constexpr int kWNodes = 0, kWTris = 1, kWWarpNodes = 2, kWQueries = 3, kWReplays = 4, kWCont = 5, kWRestart = 6,
              kWCounters = 8;
struct WarpCounters {
  unsigned* w;
  __device__ __forceinline__ void add_cont() { atomicAdd(w + kWCont, 1u); }
  __device__ __forceinline__ void add_restart() { atomicAdd(w + kWRestart, 1u); }
};

// Three-input FP32 min / max (one instruction on sm_100); min and max are
// exact, so the fold order does not change the result.
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Slab test of one ray against the 8 child boxes of a wide node:
// tn[c] = max(t_lo, near planes), tf[c] = min(tmax, far planes), the child is
// entered iff tn[c] <= tf[c]. The near and far plane of each axis are picked
// per ray by the sign of the direction (`nx`, `ny`, `nz`: word offset of the
// near planes; the far ones are at ^2). Two children's planes of one axis go
// through one packed FP32 FMA (each lane rounds like fmaf), and the three
// axes fold with 3-input min / max: 5 instructions per child where the
// scalar form takes 13, with bit-identical tn / tf.
__device__ __forceinline__ void slab8(const float4* __restrict__ nd, int nx, int ny, int nz, const RayW& r,
                                      float t_lo, float tmax, float (&tn)[8], float (&tf)[8]) {
  const float2 ix = make_float2(r.ix, r.ix), iy = make_float2(r.iy, r.iy), iz = make_float2(r.iz, r.iz);
  const float2 ox = make_float2(-r.oix, -r.oix), oy = make_float2(-r.oiy, -r.oiy), oz = make_float2(-r.oiz, -r.oiz);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float4 xn = __ldg(nd + nx + h), xf = __ldg(nd + (nx ^ 2) + h);
    const float4 yn = __ldg(nd + ny + h), yf = __ldg(nd + (ny ^ 2) + h);
    const float4 zn = __ldg(nd + nz + h), zf = __ldg(nd + (nz ^ 2) + h);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = 4 * h + 2 * q;
      const float2 axn = __ffma2_rn(q ? make_float2(xn.z, xn.w) : make_float2(xn.x, xn.y), ix, ox);
      const float2 ayn = __ffma2_rn(q ? make_float2(yn.z, yn.w) : make_float2(yn.x, yn.y), iy, oy);
      const float2 azn = __ffma2_rn(q ? make_float2(zn.z, zn.w) : make_float2(zn.x, zn.y), iz, oz);
      const float2 axf = __ffma2_rn(q ? make_float2(xf.z, xf.w) : make_float2(xf.x, xf.y), ix, ox);
      const float2 ayf = __ffma2_rn(q ? make_float2(yf.z, yf.w) : make_float2(yf.x, yf.y), iy, oy);
      const float2 azf = __ffma2_rn(q ? make_float2(zf.z, zf.w) : make_float2(zf.x, zf.y), iz, oz);
      tn[c] = fmaxf(max3f(axn.x, ayn.x, azn.x), t_lo);
      tn[c + 1] = fmaxf(max3f(axn.y, ayn.y, azn.y), t_lo);
      tf[c] = fminf(min3f(axf.x, ayf.x, azf.x), tmax);
      tf[c + 1] = fminf(min3f(axf.y, ayf.y, azf.y), tmax);
    }
  }
}

// The kChunk smallest hit keys >= key_min (t <= t_hi) along the ray, in
// ascending order, EMPTY-padded. If the stack overflowed, subtrees were
// dropped and t_drop is the smallest entry distance among them: only keys with
// t < t_drop are then guaranteed.
//
// Node visit: the near and far slab planes of each axis are picked per ray by
// the sign of the direction, so each child costs 6 FMAs and 6 min/max; child
// boxes are padded outward when written (k_wide_boxes) so the rounded test
// never culls a reported hit, and empty slots hold inverted boxes that never
// pass. Hit children are pushed in slot order with the nearest one on top.
template <int SD>
__device__ __forceinline__ void query(const BvhView& bvh, const RayW& r, unsigned long long key_min, float t_hi,
                                      unsigned long long* kb, int kstride, Stack st, float& t_drop, int* status,
                                      Counters& cnt, int count_work) {
  ++cnt.queries;
#pragma unroll
  for (int i = 0; i < kChunk; ++i) kb[i * kstride] = kEmptyKey;
  int kb_n = 0;
  t_drop = INFINITY;
  if (!bvh.has_root) return;
  const float t_lo = key_t(key_min);
  float tmax = t_hi;
  // word offsets of the near / far planes (lo at +0, hi at +2 within each axis)
  const int nx = r.ix >= 0.f ? 0 : 2, ny = r.iy >= 0.f ? 4 : 6, nz = r.iz >= 0.f ? 8 : 10;
  // entries at index >= SD live in thread-local memory
  constexpr int kSpill = kLaneStack - SD;
  uint32_t xref[kSpill];
  float xtn[kSpill];
  auto put = [&](int i, uint32_t r, float t) {
    if (i < SD) {
      st.put(i, r, t);
    } else {
      xref[i - SD] = r;
      xtn[i - SD] = t;
    }
  };
  int sp = 0;
  put(sp++, 0u, t_lo);
  int steps = 0;
  while (sp > 0) {
    if (++steps > kMaxSteps) {
      atomicOr(status, kStatusTimeout);
      break;
    }
    --sp;
    const uint32_t ref = sp < SD ? st.ref[sp * st.stride] : xref[sp - SD];
    if ((sp < SD ? st.tn[sp * st.stride] : xtn[sp - SD]) > tmax) continue;
    if (ref_is_leaf(ref)) {
      const uint32_t first = leaf_first(ref), ntri = leaf_count(ref);
      if (!TT_IN_BOUNDS(status, first + ntri <= (uint32_t)bvh.P)) continue;
      if (count_work) cnt.tris += ntri;
      for (uint32_t j = 0; j < ntri; ++j) {
        const float4* tr = bvh.tris + 3 * (size_t)(first + j);
        const float4 a = __ldg(tr), b = __ldg(tr + 1), c = __ldg(tr + 2);
        float t;
        if (!isect_tri(r, a, b, c, t)) continue;
        if (!(t >= t_lo) || !(t <= tmax)) continue;
        const unsigned long long key = hit_key(t, (uint32_t)__float_as_int(a.w));
        if (key >= key_min && kb_accepts<kChunk>(kb, kstride, key, kb_n)) {
          if (kb_insert_smem<kChunk>(kb, kstride, key, kb_n)) tmax = key_t(kb[(kChunk - 1) * kstride]);
        }
      }
      continue;
    }
    if (!TT_IN_BOUNDS(status, ref < (uint32_t)bvh.wide_cap)) continue;
    if (count_work) ++cnt.nodes;
    const float4* nd = bvh.nodes + (size_t)ref * kNodeF4;
    float tn[8], tf[8];
    bool hit[8];
    slab8(nd, nx, ny, nz, r, t_lo, tmax, tn, tf);
#pragma unroll
    for (int c = 0; c < 8; ++c) hit[c] = tn[c] <= tf[c];
    int nhit = 0, best = -1;
    float best_t = INFINITY;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (hit[c]) {
        ++nhit;
        if (tn[c] < best_t) {
          best_t = tn[c];
          best = c;
        }
      }
    }
    if (nhit == 0) continue;
    const float4 r0 = __ldg(nd + 12), r1 = __ldg(nd + 13);
    const uint32_t cref[8] = {__float_as_uint(r0.x), __float_as_uint(r0.y), __float_as_uint(r0.z),
                              __float_as_uint(r0.w), __float_as_uint(r1.x), __float_as_uint(r1.y),
                              __float_as_uint(r1.z), __float_as_uint(r1.w)};
    // nearest child last (top of the stack); on overflow drop the others and
    // remember the smallest distance dropped
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (!hit[c] || c == best) continue;
      if (sp < SD + kSpill - 1) {
        put(sp++, cref[c], tn[c]);
      } else {
        t_drop = fminf(t_drop, tn[c]);
      }
    }
    put(sp++, cref[best], best_t);
  }
}

// ---------------------------------------------------------------- packets
// Warp packet traversal. The rays of a warp (an 8x4-pixel tile) are bounded by
// one frustum, and the warp walks the BVH for the frustum instead of for each
// ray: a lane tests one child box of one of four nodes, so 32 boxes cost what
// one ray's test of a single child would. The triangles of entered leaves are
// culled one a lane against the frustum, and the survivors, 32 at a time, one
// a lane again, against every ray's line through the common origin (2 FMAs an
// edge). Only the (triangle, ray) pairs left over run the watertight test, so
// the hits do not depend on the culling: it only has to be conservative. A
// triangle meets ~2 of a tile's 32 rays on the benchmark's clouds; testing
// each against all rays, as the rays' own traversal did, wasted the rest.
// Hits are appended to their ray's buffer in any order and the buffers sorted
// at the end, all lanes at once; when one is full, all are sorted and cut back
// to their K nearest, which then bound the rest.
//
// Traversal pass of 1M triangles, 4 views of 800^2, K = 32 (2.56M rays): 10.9
// ms with a slab test per ray and child and an insert per hit, 6.4 with the
// frustum alone (104k -> 41k instructions a tile), 5.3 with the hits deferred
// and the pairs compacted (26k), 3.9 with the seven loads of a node wave in
// flight at once (the test's short cuts had serialised them), 3.3 with 20
// instead of 16 warps per SM (ray data shuffled instead of in shared memory); 3.4
// with a stack that holds every scene's nodes and a count of what the frustum
// holds (below).
// What bounds it: issue (62 % of cycles at 20 warps) and the latencies between,
// fixed ones and the node and triangle loads' from L2.
//
// The frustum lives in the axes of the rays' dominant direction z: for z' (z
// times the sign of the directions) in [z0, z1], every ray's u lies between
// two lines u = off + slope z', and so does its v. Rays of one origin have the
// lines of their extreme slopes; for others the chords between the extreme
// positions at z0 and z1 bound them (the maximum of linear functions is
// convex). Everything is padded by 2^-17 of the largest coordinate inside the
// frustum, an order above the rounding of these lines (slopes are at most 2) and of
// boxes clipped to it. A triangle's vertices may lie far outside: the cull and the
// watertight test shear each of them, with some ten roundings of 2^-24 of its own
// coordinates, so a triangle is culled only beyond 2^-20 of its largest.
//
// A wide frustum (coarse images, unrelated rays) holds many more triangles
// than its rays hit. Such a warp takes its rays one by one: the frustum is
// then the ray.
//
// The stack holds 136 nodes. A wave that opens several nodes may fill it only up to
// kWarpRoom; from there one node at a time is opened, nearest first, which adds at
// most 7 entries a level. Where even that does not fit, the packet is given up for
// its rays one by one, which enter fewer nodes. (With 96 entries, waves of four up to 64
// and what did not fit dropped, rays lost nodes wherever most boxes overlap:
// 100k triangles over one another, 4252 of 65536 pixels ended early.)
// Distances are kept as the upper half of their float, which rounds them down: a node
// behind the rays' bounds may at worst be opened. Costs 1-2 % (1M triangles, 4
// views of 800^2 9.09 -> 9.21 ms a step; a wave limited by the children it finds 9.27).
constexpr int kWarpStack = 136;  // interior nodes: ref, nearest z' - z0
constexpr int kWarpRoom = 80;    // entries after a wave of several nodes: 56 are left to a walk in depth
constexpr int kWarpQueue = 128;  // triangles of entered leaves (ring)
constexpr int kWarpKept = 64;    // triangles the frustum kept (ring)
constexpr int kWarpPairs = 64;   // (triangle, ray) pairs tested between two compactions
constexpr float kVertexMargin = 9.5367431640625e-7f;
constexpr int kSpare = 4;        // slots of a ray's buffer beyond its K keys

struct WarpStack {
  float4* slope;    // [16]: (a, a, b, b) of two rays: du/dz', dv/dz'
  uint32_t* ref;
  uint32_t* queue;
  uint32_t* kept;
  int* hits;        // [32] hits found so far, those past a full buffer included
  unsigned* cnt;    // kWCounters words: the warp's traversal counters
  float* scene;     // root box lo[3], hi[3], mean triangle extent
  unsigned short* pair;
  unsigned short* z;  // upper halves of z' - z0
};
constexpr size_t kWarpBytes = 16 * 16 + kWarpStack * 6 + kWarpQueue * 4 + kWarpKept * 4 + kWarpPairs * 2 + 32 * 4 +
                              kWCounters * 4 + 8 * 4;
static_assert(kWarpBytes % 16 == 0, "the next warp's slopes are float4");

// Warp-wide minimum / maximum (NaN operands are ignored).
__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// The scene's box and the mean extent of 32 sampled triangles, taken by a warp
// for the rules that decide how rays are traversed.
struct SceneStats {
  float lo[3], hi[3], extent;
};
__device__ __forceinline__ SceneStats scene_stats(const BvhView& bvh) {
  const int lane = threadIdx.x & 31;
  SceneStats st;
  const float* nd = reinterpret_cast<const float*>(bvh.nodes) + (lane & 7);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    st.lo[a] = warp_min(__ldg(nd + 16 * a));
    st.hi[a] = warp_max(__ldg(nd + 16 * a + 8));
  }
  const float4* tr = bvh.tris + 3 * (size_t)(((long long)lane * bvh.P) >> 5);
  const float4 a = __ldg(tr), b = __ldg(tr + 1), c = __ldg(tr + 2);
  float e = max3f(a.x, b.x, c.x) - min3f(a.x, b.x, c.x) + max3f(a.y, b.y, c.y) - min3f(a.y, b.y, c.y) +
            max3f(a.z, b.z, c.z) - min3f(a.z, b.z, c.z);
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) e += __shfl_xor_sync(0xFFFFFFFFu, e, s);
  st.extent = e * (1.0f / 96.0f);
  return st;
}

__device__ __forceinline__ void warp_scene(const BvhView& bvh, const WarpStack& ws) {
  if (!bvh.has_root) return;
  const SceneStats st = scene_stats(bvh);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      ws.scene[a] = st.lo[a];
      ws.scene[3 + a] = st.hi[a];
    }
    ws.scene[6] = st.extent;
  }
  __syncwarp();
}

// A packet is taken when the triangles its frustum holds are expected to number
// at most kPacketMin + kPacketRatio times those its rays meet, for triangles of the
// mean extent spread evenly over the scene's box. Forwards of pinhole images, every
// warp with whole tiles (ms; as packets / ray by ray): 1M triangles 128^2 3.5 / 5.8,
// 256^2 1.7 / 5.7; 3M triangles 64^2 22.0 / 9.2, 128^2 8.5 / 9.3, 256^2 3.9 / 9.8;
// 616k triangles 31 x 38 21.2 / 3.5; 100k triangles 64^2 0.6 / 1.0. (Images as coarse
// as the 64^2 and 31 x 38 are now taken in parts, a ray or two a warp.)
//
// One far triangle makes the box, and with it the expected spread, as large as
// one likes. So the walk counts what its frustum does hold, and a packet past the
// same line is given up for its rays: at once where the rays have no common origin,
// as each triangle held then costs a test with every ray, and kPacketTrial times later where
// a cull by the rays' lines makes it cheap. 65k rays in a cone from scattered origins over 200k
// triangles, one of them 50 away: 278 ms without the count, 6.7 with it (8.5, 11.6 and
// 17.3 at 2, 4 and 8 times the line; a walk with a box test per ray and child took 7.0).
// A camera inside those triangles and a shell around them, 256^2 at 90 degrees: 5.2 ms
// given up at the line, 4.4 at twice, 4.0 at 4 times. The count costs
// 0.2 to 0.5 % (3M triangles at 1080p 7.76 / 7.80 ms).
constexpr int kPacketTrial = 4, kPacketUnits = 2, kPacketMost = 1 << 30;
constexpr float kPacketMin = 1024.0f, kPacketRatio = 2.5f;

// Sorts the first n keys of a lane's column, of which the first `done` are in
// order (insertion: traversal finds hits nearly in order).
__device__ __forceinline__ void kb_sort(unsigned long long* kb, int stride, int done, int n) {
  for (int i = max(done, 1); i < n; ++i) {
    const unsigned long long key = kb[i * stride];
    int j = i;
    for (; j > 0; --j) {
      const unsigned long long prev = kb[(j - 1) * stride];
      if (prev <= key) break;
      kb[j * stride] = prev;
    }
    if (j != i) kb[j * stride] = key;
  }
}

// A lane's (triangle, ray) pair, `ray` a lane of the warp: the watertight test
// with that lane's ray, a hit appended to that lane's buffer. When a buffer has
// no room, all are sorted and cut back to their K nearest, which bound their
// rays' tmax, and what did not fit tries again if still near enough: returns
// true then. `room` gains `gain` for each pair that meets, near or far. `hits`: keys in each lane's buffer; kb_n: how many of this lane's
// are in order.
template <int K>
__device__ __forceinline__ bool test_pairs(const RayW& r, unsigned long long key_min, float& tmax, int& kb_n,
                                           unsigned long long* kb, int kstride, int* hits, bool have, int ray, float4 a,
                                           float4 b, float4 c, int gain, int& room) {
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  RayW q;
  q.ox = __shfl_sync(full, r.ox, ray), q.oy = __shfl_sync(full, r.oy, ray), q.oz = __shfl_sync(full, r.oz, ray);
  q.Sx = __shfl_sync(full, r.Sx, ray), q.Sy = __shfl_sync(full, r.Sy, ray), q.Sz = __shfl_sync(full, r.Sz, ray);
  q.perm = __shfl_sync(full, r.perm, ray);
  const unsigned long long lo = __shfl_sync(full, key_min, ray);
  const float far = __shfl_sync(full, tmax, ray);
  unsigned long long key = kEmptyKey;
  float t = 0.f;
  const bool meets = have && isect_tri(q, a, b, c, t);
  if (meets && t >= 0.f && t <= far) {
    key = hit_key(t, (uint32_t)__float_as_int(a.w));
    if (key < lo) key = kEmptyKey;
  }
  if (gain != 0) room = min(room + gain * __popc(__ballot_sync(full, meets)), kPacketMost);
  bool cut = false;
  while (__any_sync(full, key != kEmptyKey)) {
    if (key != kEmptyKey) {
      const int slot = atomicAdd(hits + ray, 1);
      if (slot < K + kSpare) {
        kb[slot * kstride + (ray - lane)] = key;
        key = kEmptyKey;
      }
    }
    if (!__any_sync(full, key != kEmptyKey)) break;
    cut = true;
    __syncwarp();
    const int n = min(hits[lane], K + kSpare);
    kb_sort(kb, kstride, kb_n, n);
    kb_n = min(n, K);
    hits[lane] = kb_n;
    if (kb_n == K) tmax = fminf(tmax, key_t(kb[(K - 1) * kstride]));
    __syncwarp();
    const float nearer = __shfl_sync(full, tmax, ray);
    if (key != kEmptyKey && key_t(key) > nearer) key = kEmptyKey;
  }
  return cut;
}

// The rays (bits, ray i of the packet in bit i) that may hit a triangle, given
// as its vertices relative to the common origin in (u, v, z'): all three edge
// planes through the origin have the ray on the inner side, up to 2^-18 of
// |vertex| |edge| (L1 norms), an order above the rounding of both this test
// and the watertight one for slopes of at most 2. An edge-on triangle, whose
// side is in doubt, meets every ray.
__device__ __forceinline__ unsigned rays_meeting(const float4* slope, float Au, float Av, float Az, float Bu, float Bv,
                                                 float Bz, float Cu, float Cv, float Cz) {
  const float kMargin = 3.814697265625e-6f;
  const float abu = Bu - Au, abv = Bv - Av, abz = Bz - Az;
  const float bcu = Cu - Bu, bcv = Cv - Bv, bcz = Cz - Bz;
  const float cau = Au - Cu, cav = Av - Cv, caz = Az - Cz;
  const float la = fabsf(Au) + fabsf(Av) + fabsf(Az), lb = fabsf(Bu) + fabsf(Bv) + fabsf(Bz),
              lc = fabsf(Cu) + fabsf(Cv) + fabsf(Cz);
  const float eab = fabsf(abu) + fabsf(abv) + fabsf(abz), ebc = fabsf(bcu) + fabsf(bcv) + fabsf(bcz),
              eca = fabsf(cau) + fabsf(cav) + fabsf(caz);
  // edge planes: n = vertex x edge
  float n0u = fmaf(Bv, bcz, -(Bz * bcv)), n0v = fmaf(Bz, bcu, -(Bu * bcz)), n0z = fmaf(Bu, bcv, -(Bv * bcu));
  float n1u = fmaf(Cv, caz, -(Cz * cav)), n1v = fmaf(Cz, cau, -(Cu * caz)), n1z = fmaf(Cu, cav, -(Cv * cau));
  float n2u = fmaf(Av, abz, -(Az * abv)), n2v = fmaf(Az, abu, -(Au * abz)), n2z = fmaf(Au, abv, -(Av * abu));
  const float det = fmaf(Au, n0u, fmaf(Av, n0v, Az * n0z));
  if (!(fabsf(det) > kMargin * la * lb * ebc)) return 0xFFFFFFFFu;
  const float s = det < 0.f ? -1.f : 1.f;
  n0u *= s, n0v *= s, n1u *= s, n1v *= s, n2u *= s, n2v *= s;
  n0z = fmaf(s, n0z, kMargin * lb * ebc);
  n1z = fmaf(s, n1z, kMargin * lc * eca);
  n2z = fmaf(s, n2z, kMargin * la * eab);
  unsigned out = 0u;  // sign bits, ray 0 ends in bit 31
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float4 ab = slope[i];
    const float2 a = make_float2(ab.x, ab.y), b = make_float2(ab.z, ab.w);
    const float2 e0 = __ffma2_rn(make_float2(n0u, n0u), a, __ffma2_rn(make_float2(n0v, n0v), b, make_float2(n0z, n0z)));
    const float2 e1 = __ffma2_rn(make_float2(n1u, n1u), a, __ffma2_rn(make_float2(n1v, n1v), b, make_float2(n1z, n1z)));
    const float2 e2 = __ffma2_rn(make_float2(n2u, n2u), a, __ffma2_rn(make_float2(n2v, n2v), b, make_float2(n2z, n2z)));
    out = __funnelshift_l(__float_as_uint(min3f(e0.x, e1.x, e2.x)), out, 1);
    out = __funnelshift_l(__float_as_uint(min3f(e0.y, e1.y, e2.y)), out, 1);
  }
  return __brev(~out);
}

template <int K>
__device__ __forceinline__ void packet_query(const BvhView& bvh, const RayW& r, bool want,
                                             unsigned long long key_min, float t_hi, unsigned long long* kb, int kstride,
                                             WarpStack ws, float& t_drop, int* status, int count_work) {
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  t_drop = INFINITY;
  float tmax = t_hi;
  int kb_n = 0;  // leading keys of this lane's buffer that are in order
  const float dm = max3f(fabsf(r.dx), fabsf(r.dy), fabsf(r.dz));
  // a ray with a NaN, an infinity or no direction hits nothing
  const bool usable = want && bvh.has_root && dm > 0.f &&
                      fabsf(r.ox) + fabsf(r.oy) + fabsf(r.oz) + fabsf(r.dx) + fabsf(r.dy) + fabsf(r.dz) < INFINITY;
  {
    const unsigned asked = __ballot_sync(full, want);
    if (lane == 0) ws.cnt[kWQueries] += __popc(asked);
  }
  ws.hits[lane] = 0;
  bool single = false;
  for (unsigned rest = __ballot_sync(full, usable); rest != 0u;) {
    const unsigned G = single ? (rest & (0u - rest)) : rest;
    const int lead = __ffs(G) - 1;
    const bool in = (G >> lane) & 1u;
    const int kz = (__shfl_sync(full, r.perm, lead) >> 4) & 3;
    const float sg = __shfl_sync(full, sel3(r.dx, r.dy, r.dz, kz), lead) < 0.f ? -1.f : 1.f;
    const float dk = sg * sel3(r.dx, r.dy, r.dz, kz);
    const float oz = sg * sel3(r.ox, r.oy, r.oz, kz);
    float z0, z1, pad, oU1, oU0, oV1, oV0, sU1, sU0, sV1, sV0;
    bool common;
    {
      const float ou = sel3(r.oy, r.oz, r.ox, kz), ov = sel3(r.oz, r.ox, r.oy, kz);
      bool packet = __all_sync(full, !in || dk >= 0.5f * dm);
      const float a = sel3(r.dy, r.dz, r.dx, kz) / dk, b = sel3(r.dz, r.dx, r.dy, kz) / dk;
      const float rl = ws.scene[kz], rh = ws.scene[3 + kz];
      z0 = fmaxf(warp_min(in ? fmaf(key_t(key_min), dk, oz) : INFINITY), sg > 0.f ? rl : -rh);
      z1 = fminf(warp_max(in ? fmaf(tmax, dk, oz) : -INFINITY), sg > 0.f ? rh : -rl);
      float m = fmaxf(warp_max(in ? max3f(fabsf(ou), fabsf(ov), fabsf(oz)) : 0.f), fmaxf(fabsf(z0), fabsf(z1)));
      const float ou_l = __shfl_sync(full, ou, lead), ov_l = __shfl_sync(full, ov, lead),
                  oz_l = __shfl_sync(full, oz, lead);
      common = __all_sync(full, !in || (ou == ou_l && ov == ov_l && oz == oz_l));
      if (common) {
        sU1 = warp_max(in ? a : -INFINITY);
        sU0 = warp_min(in ? a : INFINITY);
        sV1 = warp_max(in ? b : -INFINITY);
        sV0 = warp_min(in ? b : INFINITY);
        oU1 = fmaf(-sU1, oz_l, ou_l);
        oU0 = fmaf(-sU0, oz_l, ou_l);
        oV1 = fmaf(-sV1, oz_l, ov_l);
        oV0 = fmaf(-sV0, oz_l, ov_l);
        float* sl = reinterpret_cast<float*>(ws.slope + (lane >> 1)) + (lane & 1);
        sl[0] = in ? a : 0.f;
        sl[2] = in ? b : 0.f;
      } else {
        const float zc = fmaxf(z1, z0 + fmaxf(m * 0.015625f, 1e-30f));  // chords over no shorter a range
        const float ua = fmaf(a, z0 - oz, ou), ub = fmaf(a, zc - oz, ou);
        const float va = fmaf(b, z0 - oz, ov), vb = fmaf(b, zc - oz, ov);
        const float U1a = warp_max(in ? ua : -INFINITY), U0a = warp_min(in ? ua : INFINITY);
        const float V1a = warp_max(in ? va : -INFINITY), V0a = warp_min(in ? va : INFINITY);
        const float U1b = warp_max(in ? ub : -INFINITY), U0b = warp_min(in ? ub : INFINITY);
        const float V1b = warp_max(in ? vb : -INFINITY), V0b = warp_min(in ? vb : INFINITY);
        const float inv = 1.0f / (zc - z0);
        sU1 = (U1b - U1a) * inv;
        sU0 = (U0b - U0a) * inv;
        sV1 = (V1b - V1a) * inv;
        sV0 = (V0b - V0a) * inv;
        oU1 = fmaf(-sU1, z0, U1a);
        oU0 = fmaf(-sU0, z0, U0a);
        oV1 = fmaf(-sV1, z0, V1a);
        oV0 = fmaf(-sV0, z0, V0a);
      }
      m = fmaxf(m, fmaxf(max3f(fabsf(fmaf(sU1, z1, oU1)), fabsf(fmaf(sU0, z1, oU0)), fabsf(fmaf(sU1, z0, oU1))),
                         max3f(fabsf(fmaf(sV1, z1, oV1)), fabsf(fmaf(sV0, z1, oV0)), fabsf(fmaf(sV1, z0, oV1)))));
      pad = m * 7.62939453125e-6f;
      if (!single) {
        // the expected triangles the frustum holds against those its rays meet, for
        // triangles of the mean extent spread over the scene's box
        const float zm = 0.5f * (z0 + z1);
        const float w = fmaf(sU1 - sU0, zm, oU1 - oU0), h = fmaf(sV1 - sV0, zm, oV1 - oV0);
        const float e = ws.scene[6];
        const int ku = kz == 2 ? 0 : kz + 1, kv = kz == 0 ? 2 : kz - 1;
        const float dens = (float)bvh.P / ((ws.scene[3 + ku] - ws.scene[ku]) * (ws.scene[3 + kv] - ws.scene[kv]));
        packet = packet && (w + e) * (h + e) * dens <= fmaf(kPacketRatio * (float)__popc(G) * e * e, dens, kPacketMin);
        if (!packet && __popc(G) > 1) {
          single = true;
          continue;
        }
      }
    }
    rest &= ~G;
    z0 -= pad;
    z1 += pad;
    oU1 += pad;
    oU0 -= pad;
    oV1 += pad;
    oV0 -= pad;
    float zcur = z1;
    if (lane == 0) {
      ws.ref[0] = 0u;
      ws.z[0] = 0;
    }
    __syncwarp();
    int sp = z0 <= z1 ? 1 : 0, qh = 0, qn = 0, kh = 0, kn = 0;
    // triangles the frustum may still hold, in units of 1 / kPacketUnits of one
    int room = (int)(kPacketMin * kPacketUnits) * (common ? kPacketTrial : 1);
    for (int steps = 0;; ++steps) {
      if (steps > kMaxSteps) {
        if (lane == 0) atomicOr(status, kStatusTimeout);
        break;
      }
      if (kn >= 32 || (sp == 0 && qn == 0 && kn > 0)) {
        // ---- a batch of kept triangles, one a lane
        const int n = min(kn, 32);
        const uint32_t ti = ws.kept[(kh + lane) & (kWarpKept - 1)];
        kh = (kh + n) & (kWarpKept - 1);
        kn -= n;
        float4 A = make_float4(0.f, 0.f, 0.f, 0.f), B = A, C = A;
        unsigned m = 0u;  // rays the triangle may meet
        const float cox = __shfl_sync(full, r.ox, lead), coy = __shfl_sync(full, r.oy, lead),
                    coz = __shfl_sync(full, r.oz, lead);
        if (lane < n) {
          const float4* tr = bvh.tris + 3 * (size_t)ti;
          A = __ldg(tr);
          B = __ldg(tr + 1);
          C = __ldg(tr + 2);
          m = G;
          if (common) {
            const float ax = A.x - cox, ay = A.y - coy, az = A.z - coz;
            const float bx = B.x - cox, by = B.y - coy, bz = B.z - coz;
            const float cx = C.x - cox, cy = C.y - coy, cz = C.z - coz;
            m &= rays_meeting(ws.slope, sel3(ay, az, ax, kz), sel3(az, ax, ay, kz), sg * sel3(ax, ay, az, kz),
                              sel3(by, bz, bx, kz), sel3(bz, bx, by, kz), sg * sel3(bx, by, bz, kz),
                              sel3(cy, cz, cx, kz), sel3(cz, cx, cy, kz), sg * sel3(cx, cy, cz, kz));
          }
        }
        if (count_work) {
          const int tests = __reduce_add_sync(full, __popc(m));
          if (lane == 0) ws.cnt[kWTris] += tests;
        }
        // the pairs left, compacted kWarpPairs at a time: a lane tests one
        while (__any_sync(full, m != 0u)) {
          int at = __popc(m);
#pragma unroll
          for (int i = 1; i < 32; i <<= 1) {
            const int v = __shfl_up_sync(full, at, i);
            if (lane >= i) at += v;
          }
          const int pairs = min(__shfl_sync(full, at, 31), kWarpPairs);
          if (common) room = min(room + (int)(kPacketRatio * kPacketUnits) * kPacketTrial * pairs, kPacketMost);
          for (at -= __popc(m); m != 0u && at < kWarpPairs; ++at, m &= m - 1u)
            ws.pair[at] = (unsigned short)((lane << 5) | (__ffs(m) - 1));
          __syncwarp();
          for (int i = lane; i - lane < pairs; i += 32) {
            const bool have = i < pairs;
            const int pr = have ? ws.pair[i] : 0;
            const int ray = pr & 31, tri = pr >> 5;
            float4 a, b, c;
            a.x = __shfl_sync(full, A.x, tri), a.y = __shfl_sync(full, A.y, tri), a.z = __shfl_sync(full, A.z, tri);
            b.x = __shfl_sync(full, B.x, tri), b.y = __shfl_sync(full, B.y, tri), b.z = __shfl_sync(full, B.z, tri);
            c.x = __shfl_sync(full, C.x, tri), c.y = __shfl_sync(full, C.y, tri), c.z = __shfl_sync(full, C.z, tri);
            a.w = __shfl_sync(full, A.w, tri);
            b.w = c.w = 0.f;
            if (test_pairs<K>(r, key_min, tmax, kb_n, kb, kstride, ws.hits, have, ray, a, b, c,
                              common ? 0 : (int)(kPacketRatio * kPacketUnits), room))
              zcur = fminf(z1, warp_max(in ? fmaf(tmax, dk, oz) : -INFINITY) + pad);
          }
          __syncwarp();
        }
        __syncwarp();
        room -= n * kPacketUnits;
        if (room < 0 && __popc(G) > 1) {
          single = true;
          break;
        }
        continue;
      }
      if (qn >= 32 || (sp == 0 && qn > 0)) {
        // ---- a batch of leaf triangles, one a lane, against the frustum
        const int n = min(qn, 32);
        const uint32_t ti = ws.queue[(qh + lane) & (kWarpQueue - 1)];
        qh = (qh + n) & (kWarpQueue - 1);
        qn -= n;
        bool keep = false;
        if (lane < n) {
          const float4* tr = bvh.tris + 3 * (size_t)ti;
          const float4 A = __ldg(tr), B = __ldg(tr + 1), C = __ldg(tr + 2);
          const float Au = sel3(A.y, A.z, A.x, kz), Av = sel3(A.z, A.x, A.y, kz), Az = sg * sel3(A.x, A.y, A.z, kz);
          const float Bu = sel3(B.y, B.z, B.x, kz), Bv = sel3(B.z, B.x, B.y, kz), Bz = sg * sel3(B.x, B.y, B.z, kz);
          const float Cu = sel3(C.y, C.z, C.x, kz), Cv = sel3(C.z, C.x, C.y, kz), Cz = sg * sel3(C.x, C.y, C.z, kz);
          // pad covers what lies in the frustum; a vertex outside it rounds by its own size
          const float e = kVertexMargin * max3f(max3f(fabsf(Au), fabsf(Bu), fabsf(Cu)),
                                                max3f(fabsf(Av), fabsf(Bv), fabsf(Cv)),
                                                max3f(fabsf(Az), fabsf(Bz), fabsf(Cz)));
          keep = (max3f(Az, Bz, Cz) >= z0 - e) & (min3f(Az, Bz, Cz) <= zcur + e) &
                 (min3f(fmaf(-sU1, Az, Au), fmaf(-sU1, Bz, Bu), fmaf(-sU1, Cz, Cu)) <= oU1 + e) &
                 (max3f(fmaf(-sU0, Az, Au), fmaf(-sU0, Bz, Bu), fmaf(-sU0, Cz, Cu)) >= oU0 - e) &
                 (min3f(fmaf(-sV1, Az, Av), fmaf(-sV1, Bz, Bv), fmaf(-sV1, Cz, Cv)) <= oV1 + e) &
                 (max3f(fmaf(-sV0, Az, Av), fmaf(-sV0, Bz, Bv), fmaf(-sV0, Cz, Cv)) >= oV0 - e);
        }
        const unsigned km = __ballot_sync(full, keep);
        if (keep && TT_IN_BOUNDS(status, kn + __popc(km) <= kWarpKept))
          ws.kept[(kh + kn + __popc(km & lt)) & (kWarpKept - 1)] = ti;
        kn += __popc(km);
        __syncwarp();
        continue;
      }
      if (sp == 0) break;
      // ---- four nodes, eight children each: a lane tests one child box
      const int take = sp > kWarpRoom - 28 ? 1 : min(sp, 4);
      const int q = lane >> 3;
      bool on = q < take;
      uint32_t ref = 0u;
      if (on) {
        ref = ws.ref[sp - 1 - q];
        on = (int)ws.z[sp - 1 - q] <= __float_as_int(zcur - z0) >> 16 &&
             TT_IN_BOUNDS(status, ref < (uint32_t)bvh.wide_cap);
      }
      __syncwarp();
      sp -= take;
      if (count_work) {
        const unsigned nodes = __popc(__ballot_sync(full, on)) >> 3;
        if (lane == 0) {
          ws.cnt[kWNodes] += nodes * __popc(G);
          ws.cnt[kWWarpNodes] += nodes;
        }
      }
      bool hit = false;
      float za = 0.f;
      uint32_t cref = kEmptyRef;
      if (on) {
        const float* nd = reinterpret_cast<const float*>(bvh.nodes + (size_t)ref * kNodeF4) + (lane & 7);
        const int ku = kz == 2 ? 0 : kz + 1, kv = kz == 0 ? 2 : kz - 1;
        const float zl = __ldg(nd + 16 * kz), zh = __ldg(nd + 16 * kz + 8);
        const float ul = __ldg(nd + 16 * ku), uh = __ldg(nd + 16 * ku + 8);
        const float vl = __ldg(nd + 16 * kv), vh = __ldg(nd + 16 * kv + 8);
        cref = __float_as_uint(__ldg(nd + 48));
        za = fmaxf(sg > 0.f ? zl : -zh, z0);
        const float zb = fminf(sg > 0.f ? zh : -zl, zcur);
        // (no short cuts: all loads in flight at once)
        hit = (za <= zb) & (ul <= fmaxf(fmaf(sU1, za, oU1), fmaf(sU1, zb, oU1))) &
              (uh >= fminf(fmaf(sU0, za, oU0), fmaf(sU0, zb, oU0))) &
              (vl <= fmaxf(fmaf(sV1, za, oV1), fmaf(sV1, zb, oV1))) &
              (vh >= fminf(fmaf(sV0, za, oV0), fmaf(sV0, zb, oV0)));
      }
      // leaves: their triangles go to the queue
      const bool leaf = hit && ref_is_leaf(cref);
      const uint32_t cnt = leaf ? leaf_count(cref) : 0u;
      const unsigned b0 = __ballot_sync(full, cnt & 1u), b1 = __ballot_sync(full, cnt & 2u);
      if (b0 | b1) {
        const int at = qh + qn + __popc(b0 & lt) + 2 * __popc(b1 & lt);
        const uint32_t first = leaf_first(cref);
        if (leaf && TT_IN_BOUNDS(status, at + (int)cnt - qh <= kWarpQueue)) {
          const bool ok = TT_IN_BOUNDS(status, first + cnt <= (uint32_t)bvh.P);
          ws.queue[at & (kWarpQueue - 1)] = ok ? first : 0u;
          if (cnt > 1u) ws.queue[(at + 1) & (kWarpQueue - 1)] = ok ? first + 1u : 0u;
          if (cnt > 2u) ws.queue[(at + 2) & (kWarpQueue - 1)] = ok ? first + 2u : 0u;
        }
        qn += __popc(b0) + 2 * __popc(b1);
      }
      // interior children: pushed farthest first, so the nearest are popped next
      const bool inner = hit && !leaf;
      const unsigned im = __ballot_sync(full, inner);
      if (im != 0u) {
        const int nh = __popc(im);
        // distances from z0 are >= 0, so their bits order like the values; ties go by lane
        const unsigned key = inner ? ((__float_as_uint(za - z0) & ~31u) | (unsigned)lane) : 0xFFFFFFFFu;
        int rank = 0;
        for (unsigned mm = im; mm != 0u; mm &= mm - 1u) rank += __shfl_sync(full, key, __ffs(mm) - 1) < key ? 1 : 0;
        const int npush = min(nh, kWarpStack - sp);
        if (npush < nh && __popc(G) > 1) {  // no room for the packet: its rays one by one
          single = true;
          break;
        }
        if (inner && rank < npush && TT_IN_BOUNDS(status, sp >= 0 && sp + npush <= kWarpStack)) {
          ws.ref[sp + npush - 1 - rank] = cref;
          ws.z[sp + npush - 1 - rank] = (unsigned short)(__float_as_uint(za - z0) >> 16);
        }
        if (npush < nh) {
          // stack full: the farthest children are dropped; the rays only trust
          // keys nearer than the nearest of them
          const float zd = warp_min(inner && rank >= npush ? za : INFINITY) - pad;
          if (in) t_drop = fminf(t_drop, fmaxf((zd - oz) / dk * (1.0f - 1e-6f), 0.f));
        }
        sp += npush;
      }
      __syncwarp();
    }
    __syncwarp();
    if (single && __popc(G) > 1) {
      rest = G;
      ws.hits[lane] = 0;
      kb_n = 0;
      tmax = t_hi;
      __syncwarp();
    }
  }
  __syncwarp();
  const int n = min(ws.hits[lane], K + kSpare);
  kb_sort(kb, kstride, kb_n, n);
  for (int i = n; i < K; ++i) kb[i * kstride] = kEmptyKey;
}

// ---------------------------------------------------------------- pairs
// Queries of unrelated rays, a warp's worth at a time. Traversed a ray a lane,
// such rays leave most lanes idle (7 of 32 active on the spawned levels of the
// benchmark's secondary rays): they differ in when they are at a node, at a
// leaf, inserting a hit or done. Here the warp keeps one stack of (node, ray)
// pairs; a lane takes any pair, tests its ray against the node's 8 children and
// adds the entered ones, triangles to a queue of (triangle, ray) pairs that are
// tested 32 at a time.
//
// Traversal of the spawned rays of 500k triangles, 2 views of 800^2, two
// bounces (1.87M rays, 99 node visits and 58 triangle tests each): 15.2 ms a
// ray a lane, 9.9 with pairs added slot by slot, 7.9 with each lane's triangles
// in one run (26 lanes at work in a node step, 32 in a triangle step). It
// issues on half of the cycles, the rest waits on arithmetic and on L1, whose
// bandwidth is half used by the node loads. A frustum around 32 of these rays,
// or one around each ray for the whole warp, takes 38-41 ms.
constexpr int kPairStack = 512;    // (node << 5 | ray); nodes and triangles are below 2^27
constexpr int kPairReserve = 200;  // kept free for pairs taken one at a time (a depth-first walk adds 7 a level)
constexpr int kPairQueue = 512;    // (triangle << 5 | ray), ring
struct PairMem {
  uint32_t* stack;
  uint32_t* queue;
  int* hits;  // [32] keys in each lane's buffer
  int* drop;  // [32] float bits of the nearest dropped entry distance
};
constexpr size_t kPairBytes = (size_t)(kPairStack + kPairQueue + 64) * 4;
template <int K>
constexpr size_t pair_smem() {
  return (size_t)kTraceThreads * (K + kSpare) * 8 + (size_t)(kTraceThreads / 32) * kPairBytes;
}

template <int K>
__device__ __forceinline__ void pair_query(const BvhView& bvh, const RayW& r, bool want, unsigned long long key_min,
                                           float t_hi, unsigned long long* kb, int kstride, PairMem pm, float& t_drop,
                                           int* status, Counters& cnt, int count_work) {
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  float tmax = t_hi;
  const float t_lo = key_t(key_min);
  int kb_n = 0;
  const unsigned act = __ballot_sync(full, want && bvh.has_root);
  if (want) ++cnt.queries;
  pm.hits[lane] = 0;
  pm.drop[lane] = __float_as_int(INFINITY);
  if ((act >> lane) & 1u) pm.stack[__popc(act & lt)] = (uint32_t)lane;  // the root, with every ray
  int sp = __popc(act), qh = 0, qn = 0;
  __syncwarp();
  for (int steps = 0; sp + qn > 0; ++steps) {
    if (steps > kMaxSteps) {
      if (lane == 0) atomicOr(status, kStatusTimeout);
      break;
    }
    if (qn >= 32 || sp == 0) {
      const int n = min(qn, 32);
      const uint32_t e = lane < n ? pm.queue[(qh + lane) & (kPairQueue - 1)] : 0u;
      qh += n;
      qn -= n;
      const float4* tr = bvh.tris + 3 * (size_t)(e >> 5);
      const float4 a = __ldg(tr), b = __ldg(tr + 1), c = __ldg(tr + 2);
      if (count_work && lane < n) ++cnt.tris;
      int room;
      test_pairs<K>(r, key_min, tmax, kb_n, kb, kstride, pm.hits, lane < n, (int)(e & 31u), a, b, c, 0, room);
      __syncwarp();
      continue;
    }
    int m = min(min(sp, 32), max((kPairStack - kPairReserve - sp) / 7, 1));
    const uint32_t e = lane < m ? pm.stack[sp - 1 - lane] : 0u;
    const int ray = (int)(e & 31u);
    RayW q;
    q.ix = __shfl_sync(full, r.ix, ray), q.iy = __shfl_sync(full, r.iy, ray), q.iz = __shfl_sync(full, r.iz, ray);
    q.oix = __shfl_sync(full, r.oix, ray), q.oiy = __shfl_sync(full, r.oiy, ray), q.oiz = __shfl_sync(full, r.oiz, ray);
    const float lo = __shfl_sync(full, t_lo, ray), hi = __shfl_sync(full, tmax, ray);
    const bool ok = TT_IN_BOUNDS(status, (e >> 5) < (uint32_t)bvh.wide_cap);
    const float4* nd = bvh.nodes + (size_t)(ok ? e >> 5 : 0u) * kNodeF4;
    const int nx = q.ix >= 0.f ? 0 : 2, ny = q.iy >= 0.f ? 4 : 6, nz = q.iz >= 0.f ? 8 : 10;
    float tn[8], tf[8];
    const float4 r0 = __ldg(nd + 12), r1 = __ldg(nd + 13);
    slab8(nd, nx, ny, nz, q, lo, hi, tn, tf);
    const uint32_t cref[8] = {__float_as_uint(r0.x), __float_as_uint(r0.y), __float_as_uint(r0.z),
                              __float_as_uint(r0.w), __float_as_uint(r1.x), __float_as_uint(r1.y),
                              __float_as_uint(r1.z), __float_as_uint(r1.w)};
    int tris = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) tris += tn[c] <= tf[c] && ref_is_leaf(cref[c]) ? (int)leaf_count(cref[c]) : 0;
    // triangles: each lane's in one run; fewer pairs if they would not fit
    int at;
    for (;; m >>= 1) {
      if (lane >= m) tris = 0;
      at = tris;
#pragma unroll
      for (int i = 1; i < 32; i <<= 1) {
        const int u = __shfl_up_sync(full, at, i);
        if (lane >= i) at += u;
      }
      const int total = __shfl_sync(full, at, 31);
      at += qh + qn - tris;
      if (total <= kPairQueue - qn || m == 1) {
        qn += total;
        break;
      }
    }
    const bool on = lane < m;
    if (count_work && on) ++cnt.nodes;
    __syncwarp();
    sp -= m;
    unsigned inner[8];
    int more = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const bool h = on && tn[c] <= tf[c], leaf = ref_is_leaf(cref[c]);
      inner[c] = __ballot_sync(full, h && !leaf);
      more += __popc(inner[c]);
      if (h && leaf) {
        const uint32_t first = leaf_first(cref[c]), n = leaf_count(cref[c]);
        if (!TT_IN_BOUNDS(status, at + (int)n - qh <= kPairQueue)) continue;
        const uint32_t f = ((TT_IN_BOUNDS(status, first + n <= (uint32_t)bvh.P) ? first : 0u) << 5) | (uint32_t)ray;
        pm.queue[at & (kPairQueue - 1)] = f;
        if (n > 1u) pm.queue[(at + 1) & (kPairQueue - 1)] = f + 32u;
        if (n > 2u) pm.queue[(at + 2) & (kPairQueue - 1)] = f + 64u;
        at += (int)n;
      }
    }
    // interior children: slot by slot, so that rays entering the same child lie
    // side by side and share its loads
    if (sp + more <= kPairStack) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (((inner[c] >> lane) & 1u) && TT_IN_BOUNDS(status, sp >= 0 && sp + __popc(inner[c]) <= kPairStack))
          pm.stack[sp + __popc(inner[c] & lt)] = (cref[c] << 5) | (uint32_t)ray;
        sp += __popc(inner[c]);
      }
    } else {
      // no room: the rays only trust keys nearer than what they had to drop
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if ((inner[c] >> lane) & 1u) {
          const int to = sp + __popc(inner[c] & lt);
          if (to < kPairStack)
            pm.stack[to] = (cref[c] << 5) | (uint32_t)ray;
          else
            atomicMin(pm.drop + ray, __float_as_int(tn[c]));
        }
        sp = min(sp + __popc(inner[c]), kPairStack);
      }
    }
    __syncwarp();
  }
  __syncwarp();
  const int n = min(pm.hits[lane], K + kSpare);
  kb_sort(kb, kstride, kb_n, n);
  for (int i = n; i < K; ++i) kb[i * kstride] = kEmptyKey;
  t_drop = __int_as_float(pm.drop[lane]);
  __syncwarp();
}

// ---------------------------------------------------------------- shading
// Per-hit geometry. The ray/plane intersection (t and the hit point relative
// to vertex A) is solved in FP64; everything after that works in FP32 on
// triangle-sized, A-relative coordinates, where FP32 keeps ~7 digits of the
// inradius (an FP32 hit point o + t d at distance ~3 keeps only ~3).
struct Geom {
  float Cx;
  float3 n;          // unit face normal
  float phi_final, phi_max;
  float d[3];        // signed edge distances of the hit point
  float3 q;          // hit point - A
  float3 e1, e2;     // B - A, C - A
  float t;           // hit distance from the FP64 solve
};

__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator-(float3 a) { return make_float3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 operator*(float s, float3 a) { return make_float3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float fdot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 fcross(float3 a, float3 b) {
  return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float flen(float3 v) { return sqrtf(fdot(v, v)); }
__device__ __forceinline__ float3 fnormalize(float3 v) { return v * rsqrtf(fdot(v, v)); }

// FP32 operations with explicit round-to-nearest and no contraction, for
// code that repeats the reference's FP32 expression trees operation by
// operation (the sphere variants' set-up, the reference-arithmetic window
// function).
namespace vf {
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float3 add(float3 a, float3 b) { return make_float3(add(a.x, b.x), add(a.y, b.y), add(a.z, b.z)); }
__device__ __forceinline__ float3 sub(float3 a, float3 b) { return make_float3(sub(a.x, b.x), sub(a.y, b.y), sub(a.z, b.z)); }
__device__ __forceinline__ float3 scale(float3 a, float s) { return make_float3(mul(a.x, s), mul(a.y, s), mul(a.z, s)); }
__device__ __forceinline__ float dot(float3 a, float3 b) { return add(add(mul(a.x, b.x), mul(a.y, b.y)), mul(a.z, b.z)); }
__device__ __forceinline__ float3 cross(float3 a, float3 b) {
  return make_float3(sub(mul(a.y, b.z), mul(a.z, b.y)), sub(mul(a.z, b.x), mul(a.x, b.z)),
                     sub(mul(a.x, b.y), mul(a.y, b.x)));
}
__device__ __forceinline__ float3 normalize(float3 v) { return scale(v, div(1.0f, __fsqrt_rn(dot(v, v)))); }
__device__ __forceinline__ float3 neg(float3 v) { return make_float3(-v.x, -v.y, -v.z); }
// vecmath.h reflect: i - (2 n) dot(n, i)
__device__ __forceinline__ float3 reflect(float3 i, float3 n) { return sub(i, scale(scale(n, 2.0f), dot(n, i))); }

// common.h:116-141
__device__ __forceinline__ bool hit_sphere(float r, float3 cnt, float3 o, float3 d, float& t) {
  const float3 op = sub(o, cnt);
  const float a = dot(d, d);
  if (a <= 0.0f) return false;
  const float b = dot(op, d);
  const float c = sub(dot(op, op), mul(r, r));
  float det = sub(mul(b, b), mul(c, a));
  if (det < 0.0f) return false;
  det = __fsqrt_rn(det);
  t = div(sub(-b, det), a);
  if ((double)t < kStepEps) {
    t = div(add(-b, det), a);
    if ((double)t < kStepEps) return false;
  }
  return true;
}

// refract.cu:24-45, kept as written (square roots where Snell's law has
// squares; the same double/float mix)
__device__ __forceinline__ bool refract_dir(float3& out, float3 in, float3 n, float eta_org) {
  const float cos_i = dot(in, n);
  float eta = eta_org;
  if ((double)cos_i > 0.0) {
    eta = __double2float_rn(__drcp_rn((double)eta_org));
    n = neg(n);
  }
  const float sin2_i = __double2float_rn(fmax(0.0, __dsub_rn(1.0, (double)sqrtf(cos_i))));
  const float sin2_t = div(sin2_i, __fsqrt_rn(eta));
  if (sin2_t >= 1.0f) return false;
  const float cos_t = __double2float_rn(sqrt(fmax(0.0, __dsub_rn(1.0, (double)sin2_t))));
  out = add(scale(in, div(1.0f, eta)), scale(n, sub(div(-cos_i, eta), cos_t)));
  return true;
}

// envlight.cu:25-51
__device__ __forceinline__ float lcg(uint32_t& u) {
  u = u * 1664525u + 1013904223u;
  return mul((float)(u & 0x00FFFFFFu), 1.0f / 16777216.0f);
}
__device__ __forceinline__ float3 cosine_hemisphere(uint32_t& seed, float3 n) {
  const float u = lcg(seed);
  const float v = lcg(seed);
  const float z = __fsqrt_rn(u);
  const float rr = __fsqrt_rn(fmaxf(0.0f, __double2float_rn(__dsub_rn(1.0, (double)mul(z, z)))));
  const float phi = mul(v, 6.2831853071795864769f);
  const float3 dir = make_float3(mul(rr, cosf(phi)), mul(rr, sinf(phi)), z);
  const float3 up = fabsf(n.z) < 0.999f ? make_float3(0.f, 0.f, 1.f) : make_float3(0.f, 1.f, 0.f);
  const float3 t = normalize(cross(up, n));
  const float3 b = normalize(cross(n, t));
  return normalize(add(add(scale(t, dir.x), scale(b, dir.y)), scale(n, dir.z)));
}
}  // namespace vf

// Window function of tritracer/common.h:57-114: edge normals
// normalize(edge_cross x (p_i - p_{i+1})), edge 0 oriented by the incenter,
// phi = max edge distance, phi_final = phi / dist(incenter, edge 0),
// Cx = max(0, phi_final^sigma) with a negative base giving 0.
__device__ __forceinline__ Geom window_fn(float4 a, float4 b, float4 c, float3 o, float3 d, float sigma) {
  Geom g;
  const double e1x = (double)b.x - a.x, e1y = (double)b.y - a.y, e1z = (double)b.z - a.z;
  const double e2x = (double)c.x - a.x, e2y = (double)c.y - a.y, e2z = (double)c.z - a.z;
  const double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
  const double ox = (double)o.x - a.x, oy = (double)o.y - a.y, oz = (double)o.z - a.z;  // o - A
  const double t = -(ox * nx + oy * ny + oz * nz) / ((double)d.x * nx + (double)d.y * ny + (double)d.z * nz);
  g.t = (float)t;
  g.q = make_float3((float)(ox + t * d.x), (float)(oy + t * d.y), (float)(oz + t * d.z));
  g.e1 = make_float3((float)e1x, (float)e1y, (float)e1z);
  g.e2 = make_float3((float)e2x, (float)e2y, (float)e2z);
  const float3 e1 = g.e1, e2 = g.e2;
  const float la = flen(e1 - e2), lb = flen(e2), lc = flen(e1);
  const float3 inc = (lb * e1 + lc * e2) * (1.0f / (la + lb + lc));  // A is the origin
  const float3 ec = fcross(e1, e2);
  g.n = fnormalize(ec);
  float3 en0 = fnormalize(fcross(ec, -e1));
  float dist = fdot(en0, inc);
  if (dist > 0.0f) {
    en0 = -en0;
    dist = -dist;
  }
  const float3 en1 = fnormalize(fcross(ec, e1 - e2));
  const float3 en2 = fnormalize(fcross(ec, e2));
  g.d[0] = fdot(en0, g.q);
  g.d[1] = fdot(en1, g.q - e1);
  g.d[2] = fdot(en2, g.q - e2);
  g.phi_max = fmaxf(fmaxf(g.d[0], g.d[1]), g.d[2]);
  g.phi_final = g.phi_max / dist;
  // __powf of the reference is NaN for a negative base and then clamped to 0
  g.Cx = (g.phi_final >= 0.0f) ? powf(g.phi_final, sigma) : 0.0f;
  return g;
}

// The window function in the reference's own FP32 arithmetic
// (tritracer/common.h:57-114 on the hit point o + t d of forward.cu:118, t
// the FP32 hit distance): absolute coordinates, each operation rounded to
// nearest in the order of the reference's expressions, no multiply-add
// fusion. It reproduces the reference's FP32 results, including the noise of
// its edge distances (dot(n, hit) + offset cancels most of its digits on
// small triangles far from the origin), for direct comparison with the
// reference's code; the default mode solves the hit point in FP64 instead.
__device__ __forceinline__ Geom window_fn_ref(float4 a4, float4 b4, float4 c4, float3 o, float3 d, float t,
                                              float sigma) {
  using namespace vf;
  Geom g;
  const float3 A = make_float3(a4.x, a4.y, a4.z), B = make_float3(b4.x, b4.y, b4.z), C = make_float3(c4.x, c4.y, c4.z);
  const float3 hit = add(o, scale(d, t));
  const float la = __fsqrt_rn(dot(sub(B, C), sub(B, C)));
  const float lb = __fsqrt_rn(dot(sub(A, C), sub(A, C)));
  const float lc = __fsqrt_rn(dot(sub(A, B), sub(A, B)));
  const float3 num = add(add(scale(A, la), scale(B, lb)), scale(C, lc));
  const float3 inc = scale(num, div(1.0f, add(add(la, lb), lc)));
  const float3 ec = cross(sub(B, A), sub(C, A));
  g.n = normalize(ec);
  const float3 P[3] = {A, B, C};
  float dist = 0.f, phi = -INFINITY;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float3 p1 = P[i], p2 = P[(i + 1) % 3];
    float3 en = normalize(cross(ec, sub(p1, p2)));
    float offset = -dot(en, p1);
    if (i == 0) {
      dist = add(dot(en, inc), offset);
      if (dist > 0.0f) {
        en = neg(en);
        offset = -offset;
        dist = -dist;
      }
    }
    const float ed = add(dot(en, hit), offset);
    phi = fmaxf(phi, ed);
    g.d[i] = ed;
  }
  g.phi_max = phi;
  g.phi_final = div(phi, dist);
  g.Cx = (g.phi_final >= 0.0f) ? powf(g.phi_final, sigma) : 0.0f;
  g.q = sub(hit, A);
  g.e1 = sub(B, A);
  g.e2 = sub(C, A);
  g.t = t;
  return g;
}

// Geometry of a hit in the given shading mode.
template <int MODE>
__device__ __forceinline__ Geom shade_geom(float4 a, float4 b, float4 c, float3 o, float3 d, float t, float sigma) {
  if constexpr (MODE == kShadeRefArith)
    return window_fn_ref(a, b, c, o, d, t, sigma);
  else
    return window_fn(a, b, c, o, d, sigma);
}

__device__ __constant__ float c_sh2[5] = {1.0925484305920792f, -1.0925484305920792f, 0.31539156525252005f,
                                          -1.0925484305920792f, 0.5462742152960396f};
__device__ __constant__ float c_sh3[7] = {-0.5900435899266435f, 2.890611442640554f, -0.4570457994644658f,
                                          0.3731763325901154f, -0.4570457994644658f, 1.445305721320277f,
                                          -0.5900435899266435f};
constexpr float kSH0 = 0.28209479177387814f;
constexpr float kSH1 = 0.4886025119029199f;

// Degree-<=3 SH basis (tritracer/common.h:16-55, auxiliary.h:13-30).
__device__ __forceinline__ void sh_basis(float3 u, int deg, float (&B)[16]) {
  const float x = u.x, y = u.y, z = u.z;
  B[0] = kSH0;
  if (deg > 0) {
    B[1] = -kSH1 * y;
    B[2] = kSH1 * z;
    B[3] = -kSH1 * x;
  }
  if (deg > 1) {
    const float xx = x * x, yy = y * y, zz = z * z, xy = x * y, yz = y * z, xz = x * z;
    B[4] = c_sh2[0] * xy;
    B[5] = c_sh2[1] * yz;
    B[6] = c_sh2[2] * (2.0f * zz - xx - yy);
    B[7] = c_sh2[3] * xz;
    B[8] = c_sh2[4] * (xx - yy);
    if (deg > 2) {
      B[9] = c_sh3[0] * y * (3.0f * xx - yy);
      B[10] = c_sh3[1] * xy * z;
      B[11] = c_sh3[2] * y * (4.0f * zz - xx - yy);
      B[12] = c_sh3[3] * z * (2.0f * zz - 3.0f * xx - 3.0f * yy);
      B[13] = c_sh3[4] * x * (4.0f * zz - xx - yy);
      B[14] = c_sh3[5] * z * (xx - yy);
      B[15] = c_sh3[6] * x * (xx - 3.0f * yy);
    }
  }
}

__device__ __forceinline__ int sh_count(int deg) { return (deg + 1) * (deg + 1); }

// 16 coefficients of 3 channels are rows of 192 bytes, taken 16 bytes at a time
// where the array starts on such a boundary: a caller's may start at any float.
__device__ __forceinline__ bool on_16_bytes(const float* a) { return (reinterpret_cast<uintptr_t>(a) & 15u) == 0; }

// RGB = sum_k B_k * sh_k + 0.5 (before the clamp at 0).
__device__ __forceinline__ float3 sh_raw(const float* __restrict__ shs, int M, int prim, int deg, const float (&B)[16]) {
  const float* base = shs + (size_t)prim * M * 3;
  float r = 0.f, g = 0.f, b = 0.f;
  if (M == 16 && deg == 3 && on_16_bytes(shs)) {
    const float4* q = reinterpret_cast<const float4*>(base);
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const float4 w = __ldg(q + i);
      const float v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int idx = 4 * i + j, k = idx / 3, ch = idx % 3;
        if (ch == 0) r = fmaf(B[k], v[j], r);
        else if (ch == 1) g = fmaf(B[k], v[j], g);
        else b = fmaf(B[k], v[j], b);
      }
    }
  } else {
    const int n = sh_count(deg);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      if (k < n) {
        r = fmaf(B[k], __ldg(base + 3 * k), r);
        g = fmaf(B[k], __ldg(base + 3 * k + 1), g);
        b = fmaf(B[k], __ldg(base + 3 * k + 2), b);
      }
    }
  }
  return make_float3(r + 0.5f, g + 0.5f, b + 0.5f);
}

__device__ __forceinline__ float3 unit(float3 d) {
  const float inv = 1.0f / sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
  return make_float3(d.x * inv, d.y * inv, d.z * inv);
}

// computeScaling of tritracer/forward.cu:25-74 (first blending ray records the
// largest angle the vertices subtend around the centroid direction), in FP64.
__device__ __noinline__ void compute_scaling(float* __restrict__ scaling, const float* __restrict__ verts,
                                             const int* __restrict__ cumsum, const int* __restrict__ num_points,
                                             int prim, float3 of) {
  if (scaling[prim] > 0.0f) return;
  const int off = cumsum[prim], np = num_points[prim];
  const d3 o = mkd(of.x, of.y, of.z);
  d3 cen = mkd(0, 0, 0);
  for (int i = 0; i < np; ++i) {
    const float* v = verts + 3 * (size_t)(off + i);
    cen = cen + mkd(v[0], v[1], v[2]);
  }
  cen = cen * (1.0 / (double)np);
  const d3 t2o = cen - o;
  double best = 0.0;
  for (int i = 0; i < np; ++i) {
    const float* v = verts + 3 * (size_t)(off + i);
    const d3 a = mkd(v[0], v[1], v[2]) - o;
    const double lab = len(a) * len(t2o);
    double ang = 0.0;
    if (!(lab < 1e-12)) ang = acos(fmax(-1.0, fmin(1.0, dot(a, t2o) / lab)));
    best = fmax(ang, best);
  }
  scaling[prim] = (float)best;
}

// computeScaling in the reference's own FP32 arithmetic (forward.cu:25-74:
// centroid as a sum times 1/n, angle = acos of the clamped cosine), for the
// reference-arithmetic mode; the default computes it in FP64 above.
__device__ __noinline__ void compute_scaling_ref(float* __restrict__ scaling, const float* __restrict__ verts,
                                                 const int* __restrict__ cumsum, const int* __restrict__ num_points,
                                                 int prim, float3 o) {
  using namespace vf;
  if (scaling[prim] > 0.0f) return;
  const int off = cumsum[prim], np = num_points[prim];
  float3 cen = make_float3(0.f, 0.f, 0.f);
  for (int i = 0; i < np; ++i) {
    const float* v = verts + 3 * (size_t)(off + i);
    cen = add(cen, make_float3(v[0], v[1], v[2]));
  }
  cen = scale(cen, div(1.0f, (float)np));
  const float3 t2o = sub(cen, o);
  const float lt = __fsqrt_rn(dot(t2o, t2o));
  float best = 0.0f;
  for (int i = 0; i < np; ++i) {
    const float* v = verts + 3 * (size_t)(off + i);
    const float3 a = sub(make_float3(v[0], v[1], v[2]), o);
    const float lab = mul(__fsqrt_rn(dot(a, a)), lt);
    float ang = 0.0f;
    if (!(lab < 1e-12f)) ang = acosf(fmaxf(-1.0f, fminf(1.0f, div(dot(a, t2o), lab))));
    best = fmaxf(ang, best);
  }
  scaling[prim] = best;
}

// ---------------------------------------------------------------- the march
// Per-thread shared memory: the traversal stack and the 16 keys of the
// current chunk (staged out of registers before shading starts).
struct Smem {
  Stack st;
  unsigned long long* keys;
  int stride;
};

template <int SD>
__device__ __forceinline__ Smem thread_smem() {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem s;
  const int nt = blockDim.x;
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem_raw);
  uint32_t* refs = reinterpret_cast<uint32_t*>(smem_raw + (size_t)kChunk * nt * 8);
  float* tns = reinterpret_cast<float*>(refs + (size_t)SD * nt);
  s.keys = keys + threadIdx.x;
  s.stride = nt;
  s.st.ref = refs + threadIdx.x;
  s.st.tn = tns + threadIdx.x;
  s.st.stride = nt;
  return s;
}

// Where a ray's next k-closest query starts, where it is inside the
// reference's 16-hit chunk, and the far bound of its queries (the far plane,
// or the end of a proposed interval until the ray leaves it).
struct Cursor {
  unsigned long long key_min;
  float last_hit_t;
  float t_hi;
  int ref_pos;
  int chunks;
};

__device__ __forceinline__ unsigned long long first_key(int tmin_inclusive) {
  return tmin_inclusive ? 0ull : (1ull << 32);
}

__device__ __forceinline__ Cursor first_cursor(int tmin_inclusive) {
  Cursor c;
  c.key_min = first_key(tmin_inclusive);
  c.last_hit_t = 0.f;
  c.t_hi = kFar;
  c.ref_pos = 0;
  c.chunks = 0;
  return c;
}

// Clips a ray's first query to the proposed interval [t_near, t_far]
// (interval planes [2][H][W]); a NaN or out-of-range bound falls back to the
// plain one.
__device__ __forceinline__ void clip_cursor(Cursor& c, const float* interval, int HW, int pix) {
  const float tn = __ldg(interval + pix), tf = __ldg(interval + HW + pix);
  if (tn > 0.f && tn < kFar) c.key_min = max(c.key_min, (unsigned long long)__float_as_uint(tn) << 32);
  if (tf >= 0.f && tf < kFar) c.t_hi = tf;
}

// Visits the keys of one query (K keys, ascending, staged in shared memory)
// in the reference's chunk order (forward.cu:99-154), each hit at or beyond the
// near plane; consume_chunk calls sh.visit(prim) for it, which returns true to
// end the ray (transmittance cut-off), and returns true when the ray is
// finished, else leaves in `cur` where the next query starts.
//
// The reference re-traces after every 16th visited hit from last_hit_t
// (closed interval: the hit(s) at last_hit_t come again) or just after it
// (open). A query buffer holds EVERY key between its lower bound and its last
// key, so the position "first key >= the new bound" is found inside the
// buffer whenever the buffer reaches it, and only otherwise does the next
// query start at that bound; after a full or truncated buffer the stream
// resumes right after the last key taken. The query size K is therefore a
// performance choice that never changes the visited sequence.
//
// Proposed intervals: when a clipped stream runs out (no key left below
// cur.t_hi) before the ray terminated, the ray is not finished: its queries go
// on from the next key with the far plane as bound (a continuation, counted
// in cnt.cont), or, if the interval held no hit at all, from the start of the
// ray (a plain re-trace, cnt.restart). Either way every hit at or beyond
// t_near is visited in the plain order.
//
// March: the position inside a query's buffer; next() moves to the next hit
// to visit (its slot in m.i) or to the buffer's end.
struct March {
  unsigned long long last_key = 0;
  int i = 0;
  int boundaries = 0;
  bool any = false;
  bool visited = false;  // slot i was handed out by the last call
};
constexpr int kMarchVisit = 0;  // visit slot m.i
constexpr int kMarchQuery = 1;  // the next query starts at cur.key_min
constexpr int kMarchDone = 2;   // the ray is finished

template <int K, bool kStopsAtClip, class Cnt>
__device__ __forceinline__ int march_next(const Smem& sm, float t_drop, March& m, Cursor& cur, int tmin_inclusive, int P,
                                          int* status, Cnt& cnt) {
  const bool truncated = t_drop < INFINITY;
  auto trusted = [&](unsigned long long key) {
    return key != kEmptyKey && !(truncated && key_t(key) >= t_drop);
  };
  // the stream ran out below cur.t_hi; `next` is where it would resume. The
  // collecting pass (kStopsAtClip) cannot end a ray and stops there too: the
  // shading pass decides on continuations and re-traces.
  auto exhausted = [&](unsigned long long next) {
    if (cur.t_hi >= kFar || kStopsAtClip) return kMarchDone;
    cur.t_hi = kFar;
    if (!m.any && cur.chunks == 0) {
      cur.key_min = first_key(tmin_inclusive);
      cnt.add_restart();
    } else {
      cur.key_min = next;
      cnt.add_cont();
    }
    return kMarchQuery;
  };
  for (;;) {
    if (m.visited) {
      m.visited = false;
      if (cur.ref_pos == kChunk) {
        // the reference's next optixTrace starts at last_hit_t
        cur.ref_pos = 0;
        const unsigned long long tb = __float_as_uint(cur.last_hit_t);
        const unsigned long long bound = tmin_inclusive ? (tb << 32) : ((tb + 1ull) << 32);
        if (++m.boundaries > K) {  // 16+ hits at one t under the closed interval: no progress
          atomicOr(status, kStatusTimeout);
          return kMarchDone;
        }
        int j = 0;
        while (j < K && trusted(sm.keys[j * sm.stride]) && sm.keys[j * sm.stride] < bound) ++j;
        if (j < K && trusted(sm.keys[j * sm.stride])) {
          m.i = j;  // continue inside the buffer
          continue;
        }
        if (j < K && sm.keys[j * sm.stride] == kEmptyKey && !truncated) return exhausted(bound);
        cur.key_min = bound;
        return kMarchQuery;
      }
      ++m.i;
    }
    if (m.i >= K) break;
    const unsigned long long key = sm.keys[m.i * sm.stride];
    if (!trusted(key)) break;
    m.any = true;
    m.last_key = key;
    const float t = key_t(key);
    // fmaxf(last + STEP_EPSILON, t) with the sum in double (forward.cu:111)
    cur.last_hit_t = fmaxf(__double2float_rn(__dadd_rn((double)cur.last_hit_t, kStepEps)), t);
    ++cur.ref_pos;
    if (!TT_IN_BOUNDS(status, key_prim(key) < (uint32_t)P)) return kMarchDone;
    m.visited = true;
    if (t >= kNear) return kMarchVisit;
  }
  if (m.i < K && sm.keys[m.i * sm.stride] == kEmptyKey && !truncated)
    return exhausted(m.any ? m.last_key + 1ull : cur.key_min);
  if (!m.any) {
    atomicOr(status, kStatusStack);  // a truncated query that trusted nothing
    return kMarchDone;
  }
  cur.key_min = m.last_key + 1ull;
  return kMarchQuery;
}

template <int K, class Shader, class Cnt>
__device__ __forceinline__ bool consume_chunk(const Smem& sm, float t_drop, Cursor& cur, int tmin_inclusive,
                                              int* status, Shader& sh, Cnt& cnt) {
  March m;
  sh.prepare();
  for (;;) {
    const int r = march_next<K, Shader::kStopsAtClip>(sm, t_drop, m, cur, tmin_inclusive, sh.p.bvh.P, status, cnt);
    if (r != kMarchVisit) return r == kMarchDone;
    const unsigned long long key = sm.keys[m.i * sm.stride];
    if (visit_slot(sh, key_prim(key), key_t(key), m.i, 0)) return true;
  }
}

// View holding global tile `tile` (views are stored in tile order).
__device__ __forceinline__ int find_view(const TraceParams& p, int tile) {
  int lo = 0, hi = p.nviews - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (p.views[mid].tile_begin <= tile)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// Hit cache (HitCacheHeader): the forward stores every query of a ray, the
// adjoint replays them. Rows are written and read once, so they bypass L2
// residency (streaming stores / loads) and leave it to the BVH.
__device__ __forceinline__ HitCacheHeader* cache_header_ptr(const TraceParams& p) {
  return static_cast<HitCacheHeader*>(p.hit_cache);
}
__device__ __forceinline__ unsigned long long* cache_main(const TraceParams& p) {
  return reinterpret_cast<unsigned long long*>(static_cast<char*>(p.hit_cache) + sizeof(HitCacheHeader));
}
template <int K>
__device__ __forceinline__ unsigned long long* cache_pool(const TraceParams& p) {
  return cache_main(p) + (size_t)(K + 1) * p.cache_rays;
}

template <int K>
__device__ __forceinline__ bool cache_replays(const TraceParams& p) {
  if (p.cache_mode != kCacheRead && p.cache_mode != kCacheFill) return false;
  const HitCacheHeader* h = cache_header_ptr(p);
  return h->magic == kHitCacheMagic && (h->k & ~kCacheColorsFlag) == (uint32_t)K && h->rays == p.cache_rays &&
         h->gen == p.cache_gen && h->pool_cap == p.cache_pool_cap;
}

// The forward stored every query it made: no pool entry was refused (a
// missing query always follows a refusal, and pool_used counts refused
// requests too). The adjoint can then replay every query of every march.
template <int K>
__device__ __forceinline__ bool cache_complete(const TraceParams& p) {
  return cache_replays<K>(p) && cache_header_ptr(p)->pool_used <= p.cache_pool_cap;
}

// Hit colours beside the queries (plain forward / adjoint of the packet
// drivers): the forward's shading kernels store them, the adjoint reads them
// when the header says they were written.
__device__ __forceinline__ bool cache_colors_on(const TraceParams& p) {
  if (!p.cache_colors || p.cols) return false;
  return p.cache_mode != kCacheRead || (cache_header_ptr(p)->k & kCacheColorsFlag) != 0u;
}
// Colours of the main-part entry of ray g or of pool entry e (slot i's three
// channels at i * stride). Three times either count fits an int, or there are no rows.
template <int K>
__device__ __forceinline__ float* cache_color_rows(const TraceParams& p, bool main_part, long long g, uint32_t e,
                                                   int& stride) {
  if (main_part) {
    stride = 3 * (int)p.cache_rays;
    return p.cache_colors + 3 * (size_t)g;
  }
  stride = 3 * (int)p.cache_pool_cap;
  return p.cache_colors + (size_t)3 * K * p.cache_rays + 3 * (size_t)e;
}

// Shaders that use the colour rows take them and the hit's slot; the others
// ignore both.
template <class S>
__device__ __forceinline__ auto set_color_rows(S& sh, float* rows, int stride, int) -> decltype(sh.set_colors(rows, stride)) {
  sh.set_colors(rows, stride);
}
template <class S>
__device__ __forceinline__ void set_color_rows(S&, float*, int, long) {}
template <class S>
__device__ __forceinline__ auto visit_slot(S& sh, uint32_t prim, float t, int slot, int) -> decltype(sh.visit(prim, t, slot)) {
  return sh.visit(prim, t, slot);
}
template <class S>
__device__ __forceinline__ bool visit_slot(S& sh, uint32_t prim, float t, int, long) {
  return sh.visit(prim, t);
}

// Forward, first query of ray g. Returns where the entry of its next query
// gets linked (the high half of row k).
template <int K>
__device__ __forceinline__ uint32_t* cache_put_first(const TraceParams& p, long long g, const Smem& sm, float t_drop) {
  unsigned long long* rows = cache_main(p) + g;
  const size_t R = (size_t)p.cache_rays;
#pragma unroll 4
  for (int i = 0; i < K; ++i) __stcs(rows + i * R, sm.keys[i * sm.stride]);
  unsigned long long* w = rows + K * R;
  __stcs(w, ((unsigned long long)kNoEntry << 32) | __float_as_uint(t_drop));
  return reinterpret_cast<uint32_t*>(w) + 1;
}

// Forward, a later query into pool entry e (< pool_cap), linked from `link`.
template <int K>
__device__ __forceinline__ uint32_t* cache_put_more(const TraceParams& p, uint32_t e, unsigned long long key_min,
                                                    const Smem& sm, float t_drop, uint32_t* link) {
  unsigned long long* rows = cache_pool<K>(p) + e;
  const size_t C = p.cache_pool_cap;
#pragma unroll 4
  for (int i = 0; i < K; ++i) __stcs(rows + i * C, sm.keys[i * sm.stride]);
  unsigned long long* w = rows + K * C;
  __stcs(w, ((unsigned long long)kNoEntry << 32) | __float_as_uint(t_drop));
  __stcs(rows + (K + 1) * C, key_min);
  *link = e;
  return reinterpret_cast<uint32_t*>(w) + 1;
}

// Forward: pool entries for the lanes in `want` (one atomic per warp).
__device__ __forceinline__ uint32_t cache_alloc(const TraceParams& p, bool want) {
  const unsigned m = __ballot_sync(0xFFFFFFFFu, want);
  if (m == 0u) return kNoEntry;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  uint32_t base = 0u;
  if (lane == leader) base = atomicAdd(&cache_header_ptr(p)->pool_used, (uint32_t)__popc(m));
  base = __shfl_sync(0xFFFFFFFFu, base, leader);
  return want ? base + (uint32_t)__popc(m & ((1u << lane) - 1u)) : kNoEntry;
}

// Adjoint: fills the lane's query buffer from the first query of ray g or
// from pool entry e; returns t_drop and the entry of the next query.
template <int K>
__device__ __forceinline__ float cache_get(const TraceParams& p, bool first, long long g, uint32_t e, const Smem& sm,
                                           uint32_t& next) {
  const unsigned long long* rows = first ? cache_main(p) + g : cache_pool<K>(p) + e;
  const size_t S = first ? (size_t)p.cache_rays : (size_t)p.cache_pool_cap;
#pragma unroll 4
  for (int i = 0; i < K; ++i) sm.keys[i * sm.stride] = __ldcs(rows + i * S);
  const unsigned long long w = __ldcs(rows + K * S);
  next = (uint32_t)(w >> 32);
  return __uint_as_float((uint32_t)w);
}

// Fill mode: the word where the entry of the query after the one replayed
// from the main part (first) or from pool entry e gets linked.
template <int K>
__device__ __forceinline__ uint32_t* cache_link_of(const TraceParams& p, bool first, long long g, uint32_t e) {
  unsigned long long* w = first ? cache_main(p) + g + (size_t)K * p.cache_rays
                                : cache_pool<K>(p) + e + (size_t)K * p.cache_pool_cap;
  return reinterpret_cast<uint32_t*>(w) + 1;
}

// Adjoint: does pool entry e hold the query that starts at key_min?
template <int K>
__device__ __forceinline__ bool cache_has(const TraceParams& p, uint32_t e, unsigned long long key_min) {
  return e < p.cache_pool_cap && __ldcs(cache_pool<K>(p) + (size_t)(K + 1) * p.cache_pool_cap + e) == key_min;
}

template <int K>
__device__ __forceinline__ void cache_header(const TraceParams& p, bool colors = false) {
  if (p.cache_mode == kCacheWrite && blockIdx.x == 0 && threadIdx.x == 0) {
    HitCacheHeader* h = cache_header_ptr(p);  // pool_used was zeroed by the host
    h->magic = kHitCacheMagic;
    h->k = K | (colors ? kCacheColorsFlag : 0u);  // colours: the shading kernels store them
    h->rays = p.cache_rays;
    h->gen = p.cache_gen;
    h->pool_cap = p.cache_pool_cap;
  }
}

// Persistent warp driver. Each round: lanes without a ray take the next rays
// of the tile-ordered image (8x4 pixels per 32 slots) from the global counter,
// then every lane holding a ray runs its k-closest query, then every such lane
// shades its chunk. Traversal and shading never mix inside a warp, and lanes
// whose ray finished are refilled instead of idling.
// With SD = 0 (no hit cache) the queries go through the warp's pair stack `pm`
// instead of a stack a lane.
template <int SD, class Shader>
__device__ __forceinline__ void drive(const TraceParams& p, const Smem& sm, Shader& sh, Counters& cnt,
                                      PairMem pm = PairMem{}) {
  constexpr int K = kChunk;  // hits per per-lane query
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int total = p.ntiles * 32;
  bool have = false, exhausted = false;
  Cursor cur = first_cursor(p.tmin_inclusive);
  float3 o = make_float3(0.f, 0.f, 0.f), d = o;
  long long g = 0;              // hit cache index of the lane's ray
  uint32_t* link = nullptr;     // forward: where the entry of the ray's next query gets linked
  uint32_t next = kNoEntry;     // adjoint: entry of the ray's next query
  const bool replay = cache_replays<K>(p);
  for (;;) {
    const unsigned need = __ballot_sync(full, !have && !exhausted);
    if (need) {
      const int leader = __ffs(need) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(p.work, __popc(need));
      base = __shfl_sync(full, base, leader);
      if (!have && !exhausted) {
        const int slot = base + __popc(need & lt);
        if (slot >= total) {
          exhausted = true;
        } else {
          const int tile = slot >> 5, l = slot & 31;
          const ViewDesc& v = p.views[find_view(p, tile)];
          const int lt = tile - v.tile_begin;
          const int px = (lt % v.ntx) * 8 + (l & 7), py = (lt / v.ntx) * 4 + (l >> 3);
          if (px < v.W && py < v.H) {
            const int pix = py * v.W + px;
            o = make_float3(v.ray_o[3 * pix], v.ray_o[3 * pix + 1], v.ray_o[3 * pix + 2]);
            d = make_float3(v.ray_d[3 * pix], v.ray_d[3 * pix + 1], v.ray_d[3 * pix + 2]);
            g = v.ray_begin + pix;
            cur = first_cursor(p.tmin_inclusive);
            if (v.interval) clip_cursor(cur, v.interval, v.H * v.W, pix);
            if (sh.begin(&v, pix, o, d))
              have = true;
            else
              sh.end();
          }
        }
      }
    }
    if (__ballot_sync(full, have) == 0) {
      if (__all_sync(full, exhausted)) break;
      continue;
    }
    float t_drop = INFINITY;
    if constexpr (SD == 0) {
      pair_query<K>(p.bvh, make_ray(o, d), have, cur.key_min, cur.t_hi, sm.keys, sm.stride, pm, t_drop, p.status, cnt,
                    p.count_work);
    } else if (have) {
      const bool first = cur.chunks == 0;  // the ray's queries are numbered by its chunks
      if (replay && (first || cache_has<K>(p, next, cur.key_min))) {  // as the forward found it
        if (p.cache_mode == kCacheFill) link = cache_link_of<K>(p, first, g, next);
        t_drop = cache_get<K>(p, first, g, next, sm, next);
        ++cnt.replays;
      } else {
        next = kNoEntry;
        const RayW r = make_ray(o, d);
        query<SD>(p.bvh, r, cur.key_min, cur.t_hi, sm.keys, sm.stride, sm.st, t_drop, p.status, cnt, p.count_work);
        if (p.cache_mode == kCacheWrite || p.cache_mode == kCacheFill) {
          if (first) {
            link = cache_put_first<K>(p, g, sm, t_drop);
          } else if (link) {
            const uint32_t e = atomicAdd(&cache_header_ptr(p)->pool_used, 1u);
            link = e < p.cache_pool_cap ? cache_put_more<K>(p, e, cur.key_min, sm, t_drop, link) : nullptr;
          }
        }
      }
    }
    __syncwarp();
    if (have) {
      bool done = consume_chunk<K>(sm, t_drop, cur, p.tmin_inclusive, p.status, sh, cnt);
      if (!done && ++cur.chunks >= kMaxChunks) {
        atomicOr(p.status, kStatusTimeout);
        done = true;
      }
      // the collecting pass stores at most collect_queries queries a ray
      if (Shader::kStopsAtClip && p.collect_queries > 0 && cur.chunks >= p.collect_queries) done = true;
      if (done) {
        if (sh.next(o, d)) {  // another ray of the same pixel (envlight samples)
          cur = first_cursor(p.tmin_inclusive);
        } else {
          sh.end();
          have = false;
        }
      }
    }
  }
}

__device__ __forceinline__ PairMem pair_mem(unsigned char* base) {
  PairMem pm;
  pm.stack = reinterpret_cast<uint32_t*>(base + (size_t)(threadIdx.x >> 5) * kPairBytes);
  pm.queue = pm.stack + kPairStack;
  pm.hits = reinterpret_cast<int*>(pm.queue + kPairQueue);
  pm.drop = pm.hits + 32;
  return pm;
}

// Packet driver: a warp takes an 8x4-pixel tile (or, of a small image, a part
// of one: p.parts_log), then runs rounds of one packet query (all lanes whose
// ray is unfinished) and one shading pass until every ray of it is done.
__device__ __forceinline__ WarpStack warp_stack(unsigned char* base) {
  base += (size_t)(threadIdx.x >> 5) * kWarpBytes;
  WarpStack ws;
  ws.slope = reinterpret_cast<float4*>(base);
  ws.ref = reinterpret_cast<uint32_t*>(ws.slope + 16);
  ws.queue = ws.ref + kWarpStack;
  ws.kept = ws.queue + kWarpQueue;
  ws.hits = reinterpret_cast<int*>(ws.kept + kWarpKept);
  ws.cnt = reinterpret_cast<unsigned*>(ws.hits + 32);
  ws.scene = reinterpret_cast<float*>(ws.cnt + kWCounters);
  ws.pair = reinterpret_cast<unsigned short*>(ws.scene + 8);
  ws.z = ws.pair + kWarpPairs;
  return ws;
}

// kReplayOnly: every query comes from the hit cache (the adjoint given a
// complete cache); the build carries no traversal code, which leaves the
// shading arithmetic more registers. A query the cache lacks (which a
// complete cache never does) ends that ray and sets kStatusCacheMiss.
template <int K, class Shader, bool kReplayOnly = false>
__device__ __forceinline__ void drive_packets(const TraceParams& p, const Smem& sm, WarpStack ws, Shader& sh,
                                              Counters& cnt) {
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const bool replay = cache_replays<K>(p);
  const bool colors = cache_colors_on(p);
  if (lane < kWCounters) ws.cnt[lane] = 0u;
  if constexpr (!kReplayOnly) warp_scene(p.bvh, ws);
  __syncwarp();
  WarpCounters wc{ws.cnt};
  for (;;) {
    int tile = 0;
    if (lane == 0) tile = atomicAdd(p.work, 1);
    tile = __shfl_sync(full, tile, 0);
    const int part = tile & ((1 << p.parts_log) - 1);
    tile >>= p.parts_log;
    if (tile >= p.ntiles) break;
    const ViewDesc& v = p.views[find_view(p, tile)];
    const int lt = tile - v.tile_begin;
    const int px = (lt % v.ntx) * 8 + (lane & 7), py = (lt / v.ntx) * 4 + (lane >> 3);
    bool active = px < v.W && py < v.H && (lane << p.parts_log) >> 5 == part;
    float3 o = make_float3(0.f, 0.f, 1.f), d = make_float3(0.f, 0.f, 1.f);
    Cursor cur = first_cursor(p.tmin_inclusive);
    long long g = 0;  // hit cache index of the lane's ray
    if (active) {
      const int pix = py * v.W + px;
      g = v.ray_begin + pix;
      o = make_float3(v.ray_o[3 * pix], v.ray_o[3 * pix + 1], v.ray_o[3 * pix + 2]);
      d = make_float3(v.ray_d[3 * pix], v.ray_d[3 * pix + 1], v.ray_d[3 * pix + 2]);
      if (v.interval) clip_cursor(cur, v.interval, v.H * v.W, pix);
      sh.begin(&v, pix, o, d);  // the plain shaders always trace their one ray
    }
    const RayW r = make_ray(o, d);
    uint32_t* link = nullptr;  // forward: where the entry of the ray's next query gets linked
    uint32_t next = kNoEntry;  // adjoint: entry of the ray's next query
    for (bool first = true; __any_sync(full, active); first = false) {
      float t_drop = INFINITY;
      // lanes whose query the forward stored replay it; the others traverse
      const bool rep = replay && active && (first || cache_has<K>(p, next, cur.key_min));
      const bool trav = active && !rep;
      if constexpr (kReplayOnly) {
        if (trav) {
          atomicOr(p.status, kStatusCacheMiss);
          active = false;
        }
      } else {
        if (__any_sync(full, trav))
          packet_query<K>(p.bvh, r, trav, cur.key_min, cur.t_hi, sm.keys, sm.stride, ws, t_drop, p.status,
                          p.count_work);
      }
      const unsigned nrep = __popc(__ballot_sync(full, rep));
      if (lane == 0) ws.cnt[kWReplays] += nrep;
      // the cache entry holding this query, if any: its colour rows
      bool in_main = false;
      uint32_t entry = kNoEntry;
      if (rep) {
        in_main = first;
        entry = next;
        if (p.cache_mode == kCacheFill) link = cache_link_of<K>(p, first, g, next);
        t_drop = cache_get<K>(p, first, g, next, sm, next);
      } else {
        next = kNoEntry;
      }
      if (p.cache_mode == kCacheWrite || p.cache_mode == kCacheFill) {
        if (first) {
          if (trav) {
            link = cache_put_first<K>(p, g, sm, t_drop);
            in_main = true;
          }
        } else {
          const bool more = trav && link != nullptr;
          const uint32_t e = cache_alloc(p, more);
          if (more) {
            link = e < p.cache_pool_cap ? cache_put_more<K>(p, e, cur.key_min, sm, t_drop, link) : nullptr;
            if (e < p.cache_pool_cap) entry = e;
          }
        }
      }
      if (colors) {
        int stride = 0;
        float* rows = (in_main || entry != kNoEntry) ? cache_color_rows<K>(p, in_main, g, entry, stride) : nullptr;
        set_color_rows(sh, rows, stride, 0);
      }
      if (active) {
        bool done = consume_chunk<K>(sm, t_drop, cur, p.tmin_inclusive, p.status, sh, wc);
        if (!done && ++cur.chunks >= kMaxChunks) {
          atomicOr(p.status, kStatusTimeout);
          done = true;
        }
        // the collecting pass stores at most collect_queries queries a ray
        if (Shader::kStopsAtClip && p.collect_queries > 0 && cur.chunks >= p.collect_queries) done = true;
        if (done) {
          sh.end();
          active = false;
        }
      }
    }
  }
  // the warp's counters into lane 0's Counters (summed over the warp later)
  __syncwarp();
  if (lane == 0) {
    cnt.nodes += ws.cnt[kWNodes];
    cnt.tris += ws.cnt[kWTris];
    cnt.warp_nodes += ws.cnt[kWWarpNodes];
    cnt.queries += ws.cnt[kWQueries];
    cnt.replays += ws.cnt[kWReplays];
    cnt.cont += ws.cnt[kWCont];
    cnt.restart += ws.cnt[kWRestart];
  }
}

template <int K, bool kReplayOnly = false>
__device__ __forceinline__ Smem packet_smem(unsigned char*& rest) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem s;
  s.keys = reinterpret_cast<unsigned long long*>(smem_raw) + threadIdx.x;
  s.stride = blockDim.x;
  s.st.ref = nullptr;
  s.st.tn = nullptr;
  s.st.stride = 0;
  rest = smem_raw + (size_t)(K + (kReplayOnly ? 0 : kSpare)) * blockDim.x * 8;
  return s;
}

// Traversal configurations the kernels are instantiated for (the autotuner
// picks one per workload): warp packets with 16 or 32 hits per query, or
// independent lanes with a 32- or 24-entry stack per ray.
constexpr int kMaxPartsLog = 5;  // parts of one ray
template <int CFG>
struct TraversalCfg;
template <>
struct TraversalCfg<kCfgLanes32> {
  static constexpr bool packets = false;
  static constexpr int K = 16, SD = 32;
};
template <>
struct TraversalCfg<kCfgPackets16> {
  static constexpr bool packets = true;
  static constexpr int K = 16, SD = 0;
};
template <>
struct TraversalCfg<kCfgPackets32> {
  static constexpr bool packets = true;
  static constexpr int K = 32, SD = 0;
};
template <>
struct TraversalCfg<kCfgLanes24> {
  static constexpr bool packets = false;
  static constexpr int K = 16, SD = 24;
};

template <int CFG, bool kReplayOnly = false>
constexpr size_t smem_bytes_for() {
  using C = TraversalCfg<CFG>;
  if (kReplayOnly) return (size_t)kTraceThreads * C::K * 8 + (size_t)(kTraceThreads / 32) * kWCounters * 4;
  return C::packets ? (size_t)kTraceThreads * (C::K + kSpare) * 8 + (size_t)(kTraceThreads / 32) * kWarpBytes
                    : (size_t)kTraceThreads * (C::SD * 8 + kChunk * 8);
}

// Exact-adjoint forward: per-thread shared-memory words after the traversal's
// shared memory (FwdShader<true>).
constexpr int kXD = 0, kXWsum = 1, kXWt2 = 2, kXMid = 3, kXDist2 = 4, kXMidSet = 5, kExactSlots = 6;
constexpr size_t kExactSmemBytes = (size_t)kTraceThreads * kExactSlots * 4;

template <int CFG, class Shader, bool kReplayOnly = false>
__device__ __forceinline__ void run(const TraceParams& p, Shader& sh, Counters& cnt) {
  using C = TraversalCfg<CFG>;
  if constexpr (C::packets) {
    unsigned char* rest;
    const Smem sm = packet_smem<C::K, kReplayOnly>(rest);
    WarpStack ws;
    if constexpr (kReplayOnly) {
      ws = WarpStack{};
      ws.cnt = reinterpret_cast<unsigned*>(rest) + (threadIdx.x >> 5) * kWCounters;
    } else {
      ws = warp_stack(rest);
    }
    drive_packets<C::K, Shader, kReplayOnly>(p, sm, ws, sh, cnt);
  } else {
    drive<C::SD>(p, thread_smem<C::SD>(), sh, cnt);
  }
}

// ---------------------------------------------------------------- forward
__device__ __forceinline__ void add_stats(unsigned long long* stats, unsigned rays, unsigned evals, unsigned blends,
                                          const Counters& c) {
  const unsigned v[kNumStats] = {rays,         evals,   blends,    c.nodes,   c.tris,
                                 c.queries,    c.warp_nodes, c.cont, c.restart, c.replays};
#pragma unroll
  for (int i = 0; i < kNumStats; ++i) {
    const unsigned s = __reduce_add_sync(0xFFFFFFFFu, v[i]);
    if ((threadIdx.x & 31) == 0) atomicAdd(stats + i, (unsigned long long)s);
  }
}

// forward.cu:109-152 per hit and :204-214 per ray. EXACT (no reference
// counterpart) also fills the channels the reference leaves at 0: depth
// sum w t, middepth (t of the hit after which T <= 0.5) and distortion
// sum_{i<j} w_i w_j (t_i - t_j)^2 (running sums of w and w t^2).
template <int MODE>
struct FwdShader {
  static constexpr bool EXACT = MODE == kShadeExact;
  static constexpr bool kStopsAtClip = false;
  const TraceParams& p;
  const ViewDesc* v;
  int pix;
  float3 o, d;
  float C0, C1, C2, N0, N1, N2, T;
  // EXACT only: the ray's depth sums, middepth and distortion live in a
  // per-thread shared-memory slot (kExactSlots words, stride blockDim.x), so
  // the traversal between two shading passes does not carry them in registers
  float* xs = nullptr;
  // colours of the current query's hit-cache entry (raw colour of the hit in
  // slot i at i * cstride), or nullptr
  float* crow = nullptr;
  int cstride = 0;
  unsigned n_rays = 0, n_eval = 0, n_blend = 0;
  unsigned first_eval = 0;  // value of n_eval at the ray's first hit (record only)

  __device__ FwdShader(const TraceParams& params, size_t exact_offset) : p(params) {
    if (EXACT) {
      extern __shared__ __align__(16) unsigned char smem_raw[];
      xs = reinterpret_cast<float*>(smem_raw + exact_offset) + threadIdx.x;
    }
  }
  __device__ __forceinline__ float& x(int i) { return xs[i * blockDim.x]; }

  __device__ __forceinline__ bool begin(const ViewDesc* view, int pixel, float3 ro, float3 rd) {
    v = view;
    pix = pixel;
    o = ro;
    d = rd;
    C0 = C1 = C2 = N0 = N1 = N2 = 0.f;
    if (EXACT) {
#pragma unroll
      for (int i = 0; i < kExactSlots; ++i) x(i) = 0.f;
    }
    T = 1.0f;
    ++n_rays;
    if (v->record) {
      // t of the first and last hit visited, and whether the ray terminated
      const int HW = v->H * v->W;
      v->record[pix] = INFINITY;
      v->record[HW + pix] = INFINITY;
      v->record[2 * HW + pix] = 0.0f;
      first_eval = n_eval + 1;
    }
    return true;
  }

  __device__ __forceinline__ bool next(float3&, float3&) { return false; }

  __device__ __forceinline__ void prepare() {}

  __device__ __forceinline__ void set_colors(float* rows, int stride) {
    crow = rows;
    cstride = stride;
  }

  __device__ __forceinline__ bool visit(uint32_t prim, float t) { return visit(prim, t, -1); }

  // `slot`: the hit's position in its query (colour rows), -1 if unknown
  __device__ __forceinline__ bool visit(uint32_t prim, float t, int slot) {
    const float4* tr = p.bvh.tri_prim + 3 * (size_t)prim;
    const Geom g = shade_geom<MODE>(__ldg(tr), __ldg(tr + 1), __ldg(tr + 2), o, d, t, __ldg(p.sigma + prim));
    ++n_eval;
    float* rec = v->record;
    const int HW = v->H * v->W;
    if (rec) {
      if (n_eval == first_eval) rec[pix] = t;
      rec[HW + pix] = t;
    }
    const float alpha = fminf(kAlphaMax, __ldg(p.opac + prim) * g.Cx);
    if (alpha < kAlphaMin) return false;
    const float test_T = T * (1.0f - alpha);
    if (test_T < kTMin) {
      if (rec) rec[2 * HW + pix] = 1.0f;
      return true;
    }
    ++n_blend;
    p.density[prim] = 1.0f;
    if constexpr (MODE == kShadeRefArith)
      compute_scaling_ref(p.scaling, p.verts, p.cumsum, p.num_points, (int)prim, o);
    else
      compute_scaling(p.scaling, p.verts, p.cumsum, p.num_points, (int)prim, o);
    const float w = alpha * T;
    atomicMax(reinterpret_cast<int*>(p.max_blending) + prim, __float_as_int(w));
    N0 += g.n.x * w;
    N1 += g.n.y * w;
    N2 += g.n.z * w;
    if (EXACT) {
      const float ht = g.t;
      const float D = x(kXD), Wsum = x(kXWsum), Wt2 = x(kXWt2);
      x(kXDist2) += w * (ht * ht * Wsum - 2.0f * ht * D + Wt2);
      x(kXWsum) = Wsum + w;
      x(kXD) = D + w * ht;
      x(kXWt2) = Wt2 + w * ht * ht;
      if (x(kXMidSet) == 0.f && test_T <= 0.5f) {
        x(kXMid) = ht;
        x(kXMidSet) = 1.f;
      }
    }
    float3 c;
    if (p.cols) {  // precomputed colours in place of SH
      c = make_float3(__ldg(p.cols + 3 * prim), __ldg(p.cols + 3 * prim + 1), __ldg(p.cols + 3 * prim + 2));
    } else {
      float B[16];
      sh_basis(unit(d), p.sh_degree, B);
      const float3 raw = sh_raw(p.shs, p.M, (int)prim, p.sh_degree, B);
      c = make_float3(fmaxf(raw.x, 0.f), fmaxf(raw.y, 0.f), fmaxf(raw.z, 0.f));
      if (crow && slot >= 0) {  // for the adjoint, which then reads it instead of the SH
        crow[(size_t)slot * cstride] = raw.x;
        crow[(size_t)slot * cstride + 1] = raw.y;
        crow[(size_t)slot * cstride + 2] = raw.z;
      }
    }
    C0 += c.x * w;
    C1 += c.y * w;
    C2 += c.z * w;
    T = test_T;
    return false;
  }

  __device__ __forceinline__ void end() {
    const int HW = v->H * v->W;
    v->out_color[pix] = C0 + T * p.bg[0];
    v->out_color[HW + pix] = C1 + T * p.bg[1];
    v->out_color[2 * HW + pix] = C2 + T * p.bg[2];
    v->out_others[kDepthCh * HW + pix] = EXACT ? x(kXD) : 0.0f;  // the reference never accumulates depth
    v->out_others[kAlphaCh * HW + pix] = 1.0f - T;
    v->out_others[(kNormalCh + 0) * HW + pix] = N0;
    v->out_others[(kNormalCh + 1) * HW + pix] = N1;
    v->out_others[(kNormalCh + 2) * HW + pix] = N2;
    v->out_others[kMidDepthCh * HW + pix] = EXACT ? x(kXMid) : 0.0f;
    v->out_others[kDistortionCh * HW + pix] = EXACT ? x(kXDist2) : 0.0f;
  }
};

// Blocks per SM the replay-only builds are compiled for (shading pass and
// adjoint): 4, as the traversing builds; at 5 the adjoint spilled 240 bytes
// a thread and took 5.4 ms instead of 5.0 on C2.
#ifndef TT_REPLAY_BLOCKS
#define TT_REPLAY_BLOCKS 4
#endif
constexpr int kReplayBlocks = TT_REPLAY_BLOCKS;

// REPLAY: the replay-only build for the shading pass of a split forward
// whose traversal-only pass stored every query of every march; launched as a
// pair with the traversing build (p.fwd_pair), like the adjoint.
template <int CFG, int MODE, bool REPLAY = false>
__global__ void __launch_bounds__(kTraceThreads, REPLAY ? kReplayBlocks : kMinBlocks) k_forward(const __grid_constant__ TraceParams p) {
  if (p.fwd_pair && cache_complete<TraversalCfg<CFG>::K>(p) != REPLAY) return;
  cache_header<TraversalCfg<CFG>::K>(p, TraversalCfg<CFG>::packets && p.cache_colors != nullptr);
  Counters cnt;
  FwdShader<MODE> sh(p, smem_bytes_for<CFG, REPLAY>());
  run<CFG, FwdShader<MODE>, REPLAY>(p, sh, cnt);
  // queries = those the march used, traversed here or replayed from the
  // collecting pass; hit_cache_replays counts the adjoint's replays only
  cnt.queries += cnt.replays;
  cnt.replays = 0;
  add_stats(p.stats, sh.n_rays, sh.n_eval, sh.n_blend, cnt);
}

// ---------------------------------------------------------------- collect
// Traversal-only pass of the split forward (plain program with a hit cache).
// It runs every ray's march with a shader that shades nothing and never ends
// a ray early, so it makes, and stores in the hit cache, every k-closest
// query the plain march would make. The shading pass (k_forward reading the
// cache) then replays each query its own march asks for; a ray that ends on
// the transmittance cut-off simply leaves its later queries unread, and a
// query the cache could not hold (pool full) is traversed again there. With
// no shading state or code the pass needs far fewer registers than the fused
// kernel, so more warps per SM hide the latency of the node and triangle
// loads, which is what bounds the traversal.
// Warps per SM decide it (the pass waits on loads). 32-hit packets: 5 blocks
// of 128 threads, what their buffers leave of shared memory (3.3 ms on 1M
// triangles, 4 x 800^2 rays; 3.9 at 4 blocks). 16-hit packets: 6 blocks at 80
// registers (3M triangles at 1080p 2.6 ms; 2.8 at 5 and at 7, 3.3 at 4).
#ifndef TT_COLLECT_BLOCKS
#define TT_COLLECT_BLOCKS 6
#endif
constexpr int kCollectBlocks = TT_COLLECT_BLOCKS;

struct MarchShader {
  static constexpr bool kStopsAtClip = true;
  const TraceParams& p;
  __device__ explicit MarchShader(const TraceParams& params) : p(params) {}
  __device__ __forceinline__ bool begin(const ViewDesc*, int, float3, float3) { return true; }
  __device__ __forceinline__ bool next(float3&, float3&) { return false; }
  __device__ __forceinline__ void prepare() {}
  __device__ __forceinline__ bool visit(uint32_t, float) { return false; }
  __device__ __forceinline__ void end() {}
};

template <int CFG>
__global__ void __launch_bounds__(kTraceThreads, CFG == kCfgPackets32 ? 5 : kCollectBlocks) k_collect(const __grid_constant__ TraceParams p) {
  cache_header<TraversalCfg<CFG>::K>(p, TraversalCfg<CFG>::packets && p.cache_colors != nullptr);
  Counters cnt;
  MarchShader sh(p);
  run<CFG>(p, sh, cnt);
  // the traversal work (node visits, triangle tests) only: rays, hits and the
  // queries the march used are counted by the shading pass
  cnt.queries = 0;
  add_stats(p.stats, 0u, 0u, 0u, cnt);
}

// ---------------------------------------------------------------- variants
// Sphere variants of the reference (tritracer/reflect.cu, refract.cu,
// envlight.cu, common.h:116-148), forward only as there. The analytic sphere
// is extra = [r, cx, cy, cz, samples]. The secondary-ray set-up repeats the
// reference's FP32 expressions with explicit round-to-nearest operations (no
// contraction), so the bent rays equal the oracle's.

struct VarShader {
  static constexpr bool kStopsAtClip = false;
  const TraceParams& p;
  const ViewDesc* v;
  int pix;
  float3 o, d;
  float C0, C1, C2, T;
  // envlight: the bent surface point, sample index and running radiance
  bool env;
  int sample;
  float3 so;
  float A0, A1, A2;
  unsigned n_rays = 0, n_eval = 0, n_blend = 0;

  __device__ explicit VarShader(const TraceParams& params) : p(params) {}

  __device__ __forceinline__ void env_ray(float3& ro, float3& rd) {
    const float3 cnt = make_float3(p.sph_cx, p.sph_cy, p.sph_cz);
    const float3 n = vf::normalize(vf::sub(so, cnt));
    uint32_t seed = ((uint32_t)(pix + 1u) * 9781u) ^ ((uint32_t)(sample + 1u) * 6271u);
    rd = vf::cosine_hemisphere(seed, n);
    ro = vf::add(so, vf::scale(rd, (float)kStepEps));
  }

  __device__ __forceinline__ bool begin(const ViewDesc* view, int pixel, float3& ro, float3& rd) {
    v = view;
    pix = pixel;
    C0 = C1 = C2 = 0.f;
    T = 1.0f;
    env = false;
    A0 = A1 = A2 = 0.f;
    ++n_rays;
    const float3 cnt = make_float3(p.sph_cx, p.sph_cy, p.sph_cz);
    const float eps = (float)kStepEps;
    float st;
    const bool hit = vf::hit_sphere(p.sph_r, cnt, ro, rd, st);
    if (p.variant == 1) {  // reflect.cu:42-48
      if (hit) {
        ro = vf::add(ro, vf::scale(rd, st));
        const float3 n = vf::normalize(vf::sub(ro, cnt));
        ro = vf::add(ro, vf::scale(n, eps));
        rd = vf::reflect(vf::normalize(rd), n);
      }
    } else if (p.variant == 2) {  // refract.cu:47-71
      if (hit) {
        const float3 hp = vf::add(ro, vf::scale(rd, st));
        const float3 n = vf::normalize(vf::sub(hp, cnt));
        const float3 in = vf::normalize(rd);
        const float ior = vf::div(1.5f, 1.0003f);
        float3 nd = in;
        if (!vf::refract_dir(nd, in, n, ior)) nd = vf::reflect(in, vf::dot(in, n) < 0.0f ? n : vf::neg(n));
        ro = vf::add(hp, vf::scale(n, eps));
        rd = nd;
      }
    } else if (hit) {  // envlight.cu:116-166
      so = vf::add(ro, vf::scale(rd, st));
      so = vf::add(so, vf::scale(vf::normalize(vf::sub(so, cnt)), eps));
      env = true;
      sample = 0;
      if (p.samples <= 0) return false;
      env_ray(ro, rd);
    }
    o = ro;
    d = rd;
    return true;
  }

  __device__ __forceinline__ void prepare() {}

  __device__ __forceinline__ bool visit(uint32_t prim, float) {
    const float4* tr = p.bvh.tri_prim + 3 * (size_t)prim;
    const Geom g = window_fn(__ldg(tr), __ldg(tr + 1), __ldg(tr + 2), o, d, __ldg(p.sigma + prim));
    ++n_eval;
    const float alpha = fminf(kAlphaMax, __ldg(p.opac + prim) * g.Cx);
    if (alpha < kAlphaMin) return false;
    const float test_T = T * (1.0f - alpha);
    if (test_T < kTMin) return true;
    ++n_blend;
    const float w = alpha * T;
    float B[16];
    sh_basis(unit(d), p.sh_degree, B);
    const float3 c = sh_raw(p.shs, p.M, (int)prim, p.sh_degree, B);
    C0 += fmaxf(c.x, 0.f) * w;
    C1 += fmaxf(c.y, 0.f) * w;
    C2 += fmaxf(c.z, 0.f) * w;
    T = test_T;
    return false;
  }

  __device__ __forceinline__ bool next(float3& ro, float3& rd) {
    if (!env) return false;
    A0 += C0 + T * p.bg[0];
    A1 += C1 + T * p.bg[1];
    A2 += C2 + T * p.bg[2];
    if (++sample >= p.samples) return false;
    C0 = C1 = C2 = 0.f;
    T = 1.0f;
    env_ray(ro, rd);
    o = ro;
    d = rd;
    return true;
  }

  __device__ __forceinline__ void end() {
    const int HW = v->H * v->W;
    if (env) {  // mean sample radiance; transmittance 0
      const float inv = 1.0f / (float)p.samples;
      C0 = A0 * inv;
      C1 = A1 * inv;
      C2 = A2 * inv;
      T = 0.0f;
    }
    v->out_color[pix] = C0 + T * p.bg[0];
    v->out_color[HW + pix] = C1 + T * p.bg[1];
    v->out_color[2 * HW + pix] = C2 + T * p.bg[2];
#pragma unroll
    for (int c = 0; c < 7; ++c) v->out_others[c * HW + pix] = 0.0f;  // variants write colour only
  }
};

// Bent and sampled rays share no direction: they are traced as pairs
// (environment lighting with 8 samples, 100k triangles, 400 x 400: 3.25 ms a ray
// a lane, 1.70 as pairs; 2.1 at 5 blocks per SM, 2.4 at 6, which spill). But most
// rays of an image miss the sphere, and pinhole rays that visit few nodes each gain
// nothing from being paired; once the image fills the chip, a ray a lane is faster on
// small trees. A ray a lane against pairs (ms), clouds of small triangles:
//   reflect   500^2   1k 0.087 / 0.097   5k 0.138 / 0.148   20k 0.257 / 0.249
//             800^2   1k 0.128 / 0.173   20k 0.447 / 0.508  60k 0.849 / 0.860  150k 1.58 / 1.40
//             1080^2  1k 0.196 / 0.278   20k 0.728 / 0.879  60k 1.41 / 1.51    150k 2.65 / 2.46
//   lighting  1080^2, 4 samples  1k 0.285 / 0.345  5k 0.558 / 0.604  20k 1.10 / 1.04
//             1080^2, 8 samples  1k 0.421 / 0.431  5k 0.882 / 0.752
// and below 131k pixels pairs always. Large triangles make long hit lists, for which
// pairs are better again: refract at 1080^2, 1k 0.82 / 0.99, 5k 6.4 / 5.4 ms, with 0.6 and 3
// hits expected a ray.
constexpr int kVariantStack = 16;
__device__ __forceinline__ bool variant_lanes(const TraceParams& p) {
  if (!p.bvh.has_root) return false;
  const SceneStats st = scene_stats(p.bvh);
  const float x = st.hi[0] - st.lo[0], y = st.hi[1] - st.lo[1], z = st.hi[2] - st.lo[2];
  const float hits = 0.75f * (float)p.bvh.P * st.extent * st.extent / (x * y + y * z + z * x);
  return hits < 1.0f;
}
// Where the sizes leave the choice to the hits to expect (p.fwd_pair), both
// kernels are launched and one returns at once.
template <bool kLanes>
__global__ void __launch_bounds__(kTraceThreads, 4) k_variant(const __grid_constant__ TraceParams p) {
  if (p.fwd_pair && variant_lanes(p) != kLanes) return;
  Counters cnt;
  VarShader sh(p);
  if constexpr (kLanes) {
    drive<kVariantStack>(p, thread_smem<kVariantStack>(), sh, cnt);
  } else {
    unsigned char* rest;
    const Smem sm = packet_smem<kChunk>(rest);
    drive<0>(p, sm, sh, cnt, pair_mem(rest));
  }
  add_stats(p.stats, sh.n_rays, sh.n_eval, sh.n_blend, cnt);
}

// ---------------------------------------------------------------- adjoint
// Gradient of phi_max through the unit edge normal of each edge at the maximum
// (|d_k - phi_max| <= 1e-6) and of the face normal, as in
// tritracer/backward.cu:104-189, in A-relative FP32 coordinates. Returns the
// 9 vertex gradients summed over both terms.
__device__ __forceinline__ void window_bwd(const Geom& g, float dL_dphi, float3 dL_dn3, float3 (&gv)[3]) {
  const float3 V[3] = {make_float3(0.f, 0.f, 0.f), g.e1, g.e2};
  gv[0] = gv[1] = gv[2] = make_float3(0.f, 0.f, 0.f);
  unsigned at_max = 0u;
#pragma unroll
  for (int k = 0; k < 3; ++k) at_max |= fabsf(g.d[k] - g.phi_max) > 1e-6f ? 0u : 1u << k;
  // nearly always one edge, but another one in every lane: the edge's vertices
  // are selected instead of running one copy of the body per edge
  for (; at_max != 0u; at_max &= at_max - 1u) {
    const int k = __ffs(at_max) - 1;
    const float3 p1 = k == 0 ? V[0] : (k == 1 ? V[1] : V[2]);
    const float3 p2 = k == 0 ? V[1] : (k == 1 ? V[2] : V[0]);
    const float3 p3 = k == 0 ? V[2] : (k == 1 ? V[0] : V[1]);
    const float3 aa = p1 - p3, bb = p2 - p3, cc = p1 - p2;
    const float3 n = fcross(aa, bb);
    const float3 ne = fcross(n, cc);
    const float inv = 1.0f / flen(ne);
    const float3 Ne = ne * inv;
    // dL/dne = (I - Ne Ne^T) dL/dNe / |ne|
    const float3 dL_dNe = dL_dphi * (g.q - p1);
    const float3 v = (dL_dNe - Ne * fdot(Ne, dL_dNe)) * inv;
    // ne = ((p1-p3) x (p2-p3)) x (p1-p2); Jacobians in the form of
    // vecmath.h:2808-2859, with v^T [u]x = v x u for the skew terms
    const float3 axb = n;
    const float3 g1 = fdot(v, bb) * cc - fdot(bb, cc) * v + fcross(v, axb) - dL_dphi * Ne;
    const float3 g2 = fdot(aa, cc) * v - fdot(v, aa) * cc - fcross(v, axb);
    const float3 g3 = fdot(v, cc) * cc - fdot(cc, cc) * v;
    gv[0] = gv[0] + (k == 0 ? g1 : (k == 1 ? g3 : g2));
    gv[1] = gv[1] + (k == 0 ? g2 : (k == 1 ? g1 : g3));
    gv[2] = gv[2] + (k == 0 ? g3 : (k == 1 ? g2 : g1));
  }
  {
    // n = (p1-p3) x (p2-p3): dn/dp1 = [p3-p2]x etc.; v^T [u]x = v x u
    const float3 n = fcross(V[0] - V[2], V[1] - V[2]);
    const float inv = 1.0f / flen(n);
    const float3 Nn = n * inv;
    const float3 v = (dL_dn3 - Nn * fdot(Nn, dL_dn3)) * inv;
    gv[0] = gv[0] + fcross(v, V[2] - V[1]);
    gv[1] = gv[1] + fcross(v, V[0] - V[2]);
    gv[2] = gv[2] + fcross(v, V[1] - V[0]);
  }
}

// Exact adjoint of the window function (no reference counterpart), written
// from its definition in A-relative coordinates (P0 = 0, P1 = e1, P2 = e2,
// hit point q): edge k's unit normal en_k = s_k normalize(nc x (P_k - P_k+1))
// with nc = e1 x e2, d_k = en_k . (q - P_k), phi = max d_k,
// dist = en_0 . (I - P0), I the incenter, phi_final = phi / dist; the face
// normal normalize(nc); q = o - A + t dir with t solving q . nc = 0. Inputs:
// dL/dphi, dL/dCx sigma Cx (for dist), dL/dn and the depth term dL/dt.
__device__ __noinline__ void window_bwd_exact(const Geom& g, float3 dir, float dL_dphi, float G, float3 dL_dn3,
                                              float dL_dt_depth, float3 (&gv)[3]) {
  const float3 P[3] = {make_float3(0.f, 0.f, 0.f), g.e1, g.e2};
  const float3 nc = fcross(g.e1, g.e2);
  const float la = flen(g.e1 - g.e2), lb = flen(g.e2), lc = flen(g.e1), sum = la + lb + lc;
  const float3 inc = (lb * g.e1 + lc * g.e2) * (1.0f / sum);
  float3 en[3];
  en[0] = fnormalize(fcross(nc, -g.e1));
  float dist = fdot(en[0], inc);
  const bool flip0 = dist > 0.0f;
  if (flip0) {
    en[0] = -en[0];
    dist = -dist;
  }
  en[1] = fnormalize(fcross(nc, g.e1 - g.e2));
  en[2] = fnormalize(fcross(nc, g.e2));
  const float dL_ddist = -G / dist;
  gv[0] = gv[1] = gv[2] = make_float3(0.f, 0.f, 0.f);
  float3 g_nc = make_float3(0.f, 0.f, 0.f);
  auto edge_bwd = [&](int k, float3 g_en) {
    const float3 e = P[k] - P[(k + 1) % 3];
    const float3 ne = fcross(nc, e);
    const float inv = 1.0f / flen(ne);
    const float3 raw = ne * inv;
    const float3 gr = (k == 0 && flip0) ? -g_en : g_en;
    const float3 v = (gr - raw * fdot(raw, gr)) * inv;  // dL/d(ne)
    g_nc = g_nc + fcross(e, v);
    const float3 ge = fcross(v, nc);
    gv[k] = gv[k] + ge;
    gv[(k + 1) % 3] = gv[(k + 1) % 3] - ge;
  };
  float3 g_p = make_float3(0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (fabsf(g.d[k] - g.phi_max) > 1e-6f) continue;
    edge_bwd(k, dL_dphi * (g.q - P[k]));
    g_p = g_p + dL_dphi * en[k];
    gv[k] = gv[k] - dL_dphi * en[k];
  }
  {
    edge_bwd(0, dL_ddist * inc);
    const float3 gI = dL_ddist * en[0];
    gv[0] = gv[0] - gI;
    gv[0] = gv[0] + (la / sum) * gI;
    gv[1] = gv[1] + (lb / sum) * gI;
    gv[2] = gv[2] + (lc / sum) * gI;
    const float ga = fdot(gI, P[0] - inc) / sum, gb = fdot(gI, P[1] - inc) / sum, gc = fdot(gI, P[2] - inc) / sum;
    const float3 bc = P[1] - P[2], ca = P[2] - P[0], ab = P[0] - P[1];
    gv[1] = gv[1] + (ga / la) * bc;
    gv[2] = gv[2] - (ga / la) * bc;
    gv[2] = gv[2] + (gb / lb) * ca;
    gv[0] = gv[0] - (gb / lb) * ca;
    gv[0] = gv[0] + (gc / lc) * ab;
    gv[1] = gv[1] - (gc / lc) * ab;
  }
  {
    const float inv = 1.0f / flen(nc);
    const float3 n = nc * inv;
    g_nc = g_nc + (dL_dn3 - n * fdot(n, dL_dn3)) * inv;
  }
  {
    const float dL_dt = fdot(g_p, dir) + dL_dt_depth;
    const float sc = -dL_dt / fdot(dir, nc);
    const float3 fB = fcross(g.e2, g.q), fC = fcross(g.q, g.e1);
    gv[0] = gv[0] + sc * (-nc - fB - fC);
    gv[1] = gv[1] + sc * fB;
    gv[2] = gv[2] + sc * fC;
  }
  {
    const float3 g1 = fcross(g.e2, g_nc), g2 = fcross(g_nc, g.e1);
    gv[1] = gv[1] + g1;
    gv[2] = gv[2] + g2;
    gv[0] = gv[0] - g1 - g2;
  }
}

// Upstream gradients of one ray and what its adjoint needs of the forward's
// outputs.
struct RayGrads {
  float g0, g1, g2, gD, gN0, gN1, gN2;
  float Cf0, Cf1, Cf2, Df, Nf0, Nf1, Nf2;
  // EXACT: middepth / distortion
  float Wf, distf, gMid, gDist;
};

template <bool EXACT>
__device__ __forceinline__ RayGrads load_ray_grads(const ViewDesc& v, int pix) {
  const int HW = v.H * v.W;
  RayGrads r;
  r.g0 = __ldg(v.dL_dpix + pix);
  r.g1 = __ldg(v.dL_dpix + HW + pix);
  r.g2 = __ldg(v.dL_dpix + 2 * HW + pix);
  r.gD = __ldg(v.dL_doth + kDepthCh * HW + pix);
  r.gN0 = __ldg(v.dL_doth + (kNormalCh + 0) * HW + pix);
  r.gN1 = __ldg(v.dL_doth + (kNormalCh + 1) * HW + pix);
  r.gN2 = __ldg(v.dL_doth + (kNormalCh + 2) * HW + pix);
  r.Cf0 = __ldg(v.colors + pix);
  r.Cf1 = __ldg(v.colors + HW + pix);
  r.Cf2 = __ldg(v.colors + 2 * HW + pix);
  r.Df = __ldg(v.others + kDepthCh * HW + pix);
  r.Nf0 = __ldg(v.others + (kNormalCh + 0) * HW + pix);
  r.Nf1 = __ldg(v.others + (kNormalCh + 1) * HW + pix);
  r.Nf2 = __ldg(v.others + (kNormalCh + 2) * HW + pix);
  if (EXACT) {
    r.Wf = __ldg(v.others + kAlphaCh * HW + pix);
    r.distf = __ldg(v.others + kDistortionCh * HW + pix);
    r.gMid = __ldg(v.dL_doth + kMidDepthCh * HW + pix);
    r.gDist = __ldg(v.dL_doth + kDistortionCh * HW + pix);
  }
  return r;
}

// backward.cu:296-312 forms dL/dalpha per channel as
// g (T x - (X_final - X) / (1 - alpha)), X the channel's running sum of w x up to
// and with the current hit. Each X repeats the forward's additions in the forward's
// order, so its rounding cancels against X_final's and the rest behind the hit is
// as good as its own terms; one sum over the channels, or another order, leaves
// that rounding in, multiplied by up to 100 (L2 error of dL/dalpha against FP64
// 1.6 to 2.2 times as large).
struct RaySums {
  float C0 = 0.f, C1 = 0.f, C2 = 0.f, N0 = 0.f, N1 = 0.f, N2 = 0.f, D = 0.f;
  __device__ __forceinline__ void add(float c0, float c1, float c2, float3 n, float t, float w) {
    C0 += c0 * w;
    C1 += c1 * w;
    C2 += c2 * w;
    N0 += n.x * w;
    N1 += n.y * w;
    N2 += n.z * w;
    D += w * t;
  }
};
__device__ __forceinline__ float alpha_grad_color(float g0, float g1, float g2, float c0, float c1, float c2, float b0,
                                                  float b1, float b2, float T, float inv1a) {
  return g0 * (T * c0 - b0 * inv1a) + g1 * (T * c1 - b1 * inv1a) + g2 * (T * c2 - b2 * inv1a);
}

// One blended hit's opacity and sigma gradients, scattered, and its vertex
// gradients, given dL/dalpha (and, EXACT, dL/dt).
template <int MODE>
__device__ __forceinline__ void hit_grads(const TraceParams& p, uint32_t prim, const Geom& g, float3 d, float sig,
                                          float opacity, float dL_dalpha, float dL_dt, float3 dL_dn, float3 (&gv)[3]) {
  constexpr bool EXACT = MODE == kShadeExact;
  const bool live = !EXACT || opacity * g.Cx < kAlphaMax;
  const float dL_dC = live ? opacity * dL_dalpha : 0.0f;
  if (live) red_add(p.d_opac + prim, dL_dalpha * g.Cx);
  if (g.phi_final > 0.0f) red_add(p.d_sigma + prim, dL_dC * g.Cx * logf(g.phi_final));
  const float dL_dphi = sig / g.phi_max * dL_dC * g.Cx;
  if (EXACT)
    window_bwd_exact(g, d, dL_dphi, dL_dC * sig * g.Cx, dL_dn, dL_dt, gv);
  else
    window_bwd(g, dL_dphi, dL_dn, gv);
}

__device__ __forceinline__ void scatter_vertices(const TraceParams& p, uint32_t prim, const float3 (&gv)[3]) {
  float* dt = p.d_tri + 3 * (size_t)__ldg(p.cumsum + prim);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    red_add(dt + 3 * k + 0, gv[k].x);
    red_add(dt + 3 * k + 1, gv[k].y);
    red_add(dt + 3 * k + 2, gv[k].z);
  }
}

// Scatters one blended hit's vertex and colour gradients.
__device__ __forceinline__ void scatter_hit(const TraceParams& p, uint32_t prim, float w, float g0, float g1, float g2,
                                            float3 raw, const float (&B)[16], const float3 (&gv)[3]) {
  scatter_vertices(p, prim, gv);
  if (p.cols) {
    red_add(p.d_cols + 3 * prim + 0, g0 * w);
    red_add(p.d_cols + 3 * prim + 1, g1 * w);
    red_add(p.d_cols + 3 * prim + 2, g2 * w);
    return;
  }
  // SH: dRGB/dsh_k = B_k, masked where the colour was clamped at 0
  const float e0 = raw.x < 0.f ? 0.f : g0 * w, e1 = raw.y < 0.f ? 0.f : g1 * w, e2 = raw.z < 0.f ? 0.f : g2 * w;
  float* dsh = p.d_sh + (size_t)prim * p.M * 3;
  const int n = sh_count(p.sh_degree);
  if (p.M == 16 && n == 16 && on_16_bytes(p.d_sh)) {
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      float v4[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int idx = 4 * q + j, k = idx / 3, ch = idx % 3;
        v4[j] = B[k] * (ch == 0 ? e0 : (ch == 1 ? e1 : e2));
      }
      red_add4(dsh + 4 * q, v4[0], v4[1], v4[2], v4[3]);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      if (k < n) {
        red_add(dsh + 3 * k + 0, B[k] * e0);
        red_add(dsh + 3 * k + 1, B[k] * e1);
        red_add(dsh + 3 * k + 2, B[k] * e2);
      }
    }
  }
}

// backward.cu:191-350: the same march, dL/dalpha from the final values and the
// running sums, scattered gradients. EXACT: the full chain rule of
// window_bwd_exact, and no gradient through a clamped alpha.
template <int MODE>
struct BwdShader {
  static constexpr bool EXACT = MODE == kShadeExact;
  static constexpr bool kStopsAtClip = false;
  const TraceParams& p;
  const ViewDesc* v;
  int pix;
  float3 o, d;
  // upstream gradients and finals, loaded for each chunk (so they do not
  // occupy registers during traversal)
  RayGrads r;
  RaySums x;
  float T;
  float Sd;  // EXACT: running sum of the distortion's w E
  bool mid_seen;

  __device__ explicit BwdShader(const TraceParams& params) : p(params) {}

  __device__ __forceinline__ bool begin(const ViewDesc* view, int pixel, float3 ro, float3 rd) {
    v = view;
    pix = pixel;
    o = ro;
    d = rd;
    x = RaySums{};
    T = 1.0f;
    Sd = 0.f;
    mid_seen = false;
    return true;
  }

  __device__ __forceinline__ bool next(float3&, float3&) { return false; }

  __device__ __forceinline__ void prepare() { r = load_ray_grads<EXACT>(*v, pix); }

  // colour rows of the current query's hit-cache entry (the forward's raw
  // colour of each blended hit), or nullptr: then the SH are evaluated
  float* crow = nullptr;
  int cstride = 0;
  __device__ __forceinline__ void set_colors(float* rows, int stride) {
    crow = rows;
    cstride = stride;
  }

  __device__ __forceinline__ bool visit(uint32_t prim, float t) { return visit(prim, t, -1); }

  __device__ __forceinline__ bool visit(uint32_t prim, float t, int slot) {
    const float4* tr = p.bvh.tri_prim + 3 * (size_t)prim;
    const float sig = __ldg(p.sigma + prim);
    const Geom g = shade_geom<MODE>(__ldg(tr), __ldg(tr + 1), __ldg(tr + 2), o, d, t, sig);
    const float opacity = __ldg(p.opac + prim);
    const float alpha = fminf(kAlphaMax, opacity * g.Cx);
    if (alpha < kAlphaMin) return false;
    const float test_T = T * (1.0f - alpha);
    if (test_T < kTMin) return true;
    const float w = alpha * T;
    float B[16];
    float3 raw;
    if (p.cols) {  // precomputed colours in place of SH
      raw = make_float3(__ldg(p.cols + 3 * prim), __ldg(p.cols + 3 * prim + 1), __ldg(p.cols + 3 * prim + 2));
    } else {
      sh_basis(unit(d), p.sh_degree, B);
      if (crow && slot >= 0)
        raw = make_float3(crow[(size_t)slot * cstride], crow[(size_t)slot * cstride + 1],
                          crow[(size_t)slot * cstride + 2]);
      else
        raw = sh_raw(p.shs, p.M, (int)prim, p.sh_degree, B);
    }
    const float c0 = p.cols ? raw.x : fmaxf(raw.x, 0.f), c1 = p.cols ? raw.y : fmaxf(raw.y, 0.f),
                c2 = p.cols ? raw.z : fmaxf(raw.z, 0.f);
    x.add(c0, c1, c2, g.n, g.t, w);
    const float inv1a = 1.0f / (1.0f - alpha);
    float dL_dalpha = alpha_grad_color(r.g0, r.g1, r.g2, c0, c1, c2, r.Cf0 - x.C0, r.Cf1 - x.C1, r.Cf2 - x.C2, T, inv1a);
    dL_dalpha += r.gD * (T * g.t - (r.Df - x.D) * inv1a);
    dL_dalpha += alpha_grad_color(r.gN0, r.gN1, r.gN2, g.n.x, g.n.y, g.n.z, r.Nf0 - x.N0, r.Nf1 - x.N1, r.Nf2 - x.N2, T,
                                  inv1a);
    float dL_dt = r.gD * w;
    if (EXACT) {
      // distortion: dD/dalpha_k = T_k E_k - (2 D_f - S_k) / (1 - alpha_k),
      // E_k = t^2 W_f - 2 t B_f + C_f, C_f = (D_f + B_f^2) / W_f; dD/dt_k = 2 w (t W_f - B_f)
      const float Cf = r.Wf > 0.f ? (r.distf + r.Df * r.Df) / r.Wf : 0.f;
      const float E = g.t * g.t * r.Wf - 2.0f * g.t * r.Df + Cf;
      Sd += w * E;
      dL_dalpha += r.gDist * (T * E - (2.0f * r.distf - Sd) * inv1a);
      dL_dt += r.gDist * 2.0f * w * (g.t * r.Wf - r.Df);
      if (!mid_seen && test_T <= 0.5f) {
        mid_seen = true;
        dL_dt += r.gMid;
      }
    }
    float3 gv[3];
    hit_grads<MODE>(p, prim, g, d, sig, opacity, dL_dalpha, dL_dt, make_float3(r.gN0 * w, r.gN1 * w, r.gN2 * w), gv);
    scatter_hit(p, prim, w, r.g0, r.g1, r.g2, raw, B, gv);
    T = test_T;
    return false;
  }

  __device__ __forceinline__ void end() {}
};

// The adjoint that marches ray by ray: re-traversing, or with the queries of
// an incomplete hit cache. Given a cache, the packet configurations launch
// k_adjoint first (p.bwd_pair): it works when the cache is complete and this
// kernel otherwise, and the other returns at once; the choice is read on the
// device, so nothing synchronises.
template <int CFG, int MODE>
__global__ void __launch_bounds__(kTraceThreads, kMinBlocks) k_backward(const __grid_constant__ TraceParams p) {
  if (p.bwd_pair && cache_complete<TraversalCfg<CFG>::K>(p)) return;
  Counters cnt;
  BwdShader<MODE> sh(p);
  run<CFG>(p, sh, cnt);
  const unsigned s = __reduce_add_sync(0xFFFFFFFFu, cnt.replays);
  if ((threadIdx.x & 31) == 0 && s != 0u) atomicAdd(p.stats + kStatReplays, (unsigned long long)s);
}

// The adjoint over a complete hit cache, a lane per hit instead of per ray.
// Ray by ray, a warp's lanes run as many steps as its longest ray, 17 of 32
// lanes at work on the benchmark's clouds, each step waiting on its gathers.
// Here each ray's march only lists its next hits (kVisits a round); the lists
// of the tile's rays are laid end to end and taken 32 at a time, and what a
// hit needs of the ones before it on its ray, the transmittance and the channels'
// running sums, run along the ray's lanes and are carried from one step to the next
// in shared memory. A ray ends at the first hit whose transmittance falls below
// the cut-off; the transmittance is multiplied hit by hit, in the forward's
// order, because a product that rounds differently ends a ray that lies on the
// cut-off elsewhere than the forward did, where the cache holds no next query. The
// sums follow the forward hit by hit too (RaySums says why); depth and normals
// are summed only where one of the tile's rays has a gradient there.
// A ray has at most kVisits lanes of a step, so those chains are short.
//
// What bounds it then is L2's handling of the reductions: 23 a hit (12 of 16
// bytes, the others of 4), each a request and a sector of its own when every
// lane scatters its own hit. So the gradients are staged in shared memory and
// the lanes regrouped: 12 neighbouring lanes add a hit's 192 bytes of SH
// gradient and 9 its vertices, which the load/store unit merges into whole
// sectors, ~5 requests and 10 sectors a hit.
//
// Measured (ms; ray by ray / a lane per hit / regrouped reductions): 1M
// triangles, 4 views of 800^2, 28M blended hits 4.2 / 4.3 / 2.9; 3M triangles,
// 16 views, 180M hits 39.0 / 38.6 / 20.5; exact adjoint of 200k triangles
// 0.24 / 0.18 / 0.18. (Scans over the whole warp instead of a ray's lanes: 3.2 and
// 22.1.) These are with one sum over all channels; the channels' own sums made a step
// of the 1M triangles 9.49 instead of 9.20 ms, of the exact 200k 0.59 instead of 0.57.
// It issues on 48 % of the cycles, with L2 38 and DRAM 15 % busy: bound by
// instructions and their latency at 16 warps per SM. Its loop is as long as the
// instruction cache: waits for instructions were 1.6 instead of 1.0 of ~9 cycles an
// instruction with the sums' chain unrolled and the SH evaluation inlined, 9.76 ms a step.
constexpr int kVisits = 6;

// Inclusive sum over the lanes of a segment (first lane `seg`) of at most 8.
__device__ __forceinline__ float seg_sum(float v, int lane, int seg) {
  static_assert(kVisits <= 8, "a segment is a ray's hits of one round");
#pragma unroll
  for (int i = 1; i < 8; i <<= 1) {
    const float u = __shfl_up_sync(0xFFFFFFFFu, v, i);
    if (lane - i >= seg) v += u;
  }
  return v;
}

// (out of line: only an adjoint whose cache has no colours evaluates them)
__device__ __noinline__ float3 sh_raw_cold(const float* shs, int M, int deg, int prim, const float* basis) {
  float B[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) B[i] = basis[i];
  return sh_raw(shs, M, prim, deg, B);
}
struct AdjointMem {
  // [4][32]: d, gD | g, T | N, D or Cf, o.x | C, gN0 (T < 0: the ray has ended); [32]: gN1, gN2 or o.y, o.z.
  // A tile without gradients of depth and normals keeps its rays' colours and
  // origins where their sums and gradients would lie; one with them reads both from
  // memory (18 floats a ray are what leaves 4 blocks of 32-hit queries an SM).
  float4* ray;
  float2* gn12;
  float* exact;         // [3][32] EXACT: gDist, gMid, Sd
  float* basis;         // [32][16] SH basis
  float* stage;         // [32][8] e0 e1 e2 e0 e1, prim, ray | [32][9] vertex gradients, [32] first vertex
  unsigned short* list; // [32 * kVisits]: ray << 8 | slot
};
template <int MODE>
constexpr size_t adjoint_warp_bytes() {
  return (size_t)32 * (16 * (4 + 4) + 8 + (MODE == kShadeExact ? 12 : 0)) + 32 * 10 * 4 + 32 * kVisits * 2;
}
template <int K, int MODE>
constexpr size_t adjoint_smem() {
  return (size_t)kTraceThreads * K * 8 + (size_t)(kTraceThreads / 32) * adjoint_warp_bytes<MODE>();
}

#ifndef TT_ADJOINT_BLOCKS
#define TT_ADJOINT_BLOCKS 4
#endif
constexpr int kAdjointBlocks = TT_ADJOINT_BLOCKS;

template <int K, int MODE>
__global__ void __launch_bounds__(kTraceThreads, kAdjointBlocks) k_adjoint(const __grid_constant__ TraceParams p) {
  if (!cache_complete<K>(p)) return;
  constexpr bool EXACT = MODE == kShadeExact;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  Smem sm;
  sm.keys = reinterpret_cast<unsigned long long*>(smem_raw) + threadIdx.x;
  sm.stride = blockDim.x;
  AdjointMem am;
  {
    unsigned char* base = smem_raw + (size_t)K * blockDim.x * 8 + (threadIdx.x >> 5) * adjoint_warp_bytes<MODE>();
    am.ray = reinterpret_cast<float4*>(base);
    am.basis = reinterpret_cast<float*>(am.ray + 4 * 32);
    am.stage = am.basis + 16 * 32;
    am.gn12 = reinterpret_cast<float2*>(am.stage + 32 * 10);
    am.exact = reinterpret_cast<float*>(am.gn12 + 32);
    am.list = reinterpret_cast<unsigned short*>(am.exact + (EXACT ? 3 * 32 : 0));
  }
  const bool colors = cache_colors_on(p);
  const bool sh16 = !p.cols && p.M == 16 && p.sh_degree == 3 && on_16_bytes(p.d_sh);
  const int row = p.cols ? 3 : 3 * sh_count(p.sh_degree);  // colour gradients of a hit
  unsigned replays = 0;
  Counters cnt;  // (interval continuations and re-traces are the forward's to count)
  for (;;) {
    int tile = 0;
    if (lane == 0) tile = atomicAdd(p.work, 1);
    tile = __shfl_sync(full, tile, 0);
    const int part = tile & ((1 << p.parts_log) - 1);
    tile >>= p.parts_log;
    if (tile >= p.ntiles) break;
    const ViewDesc& v = p.views[find_view(p, tile)];
    const int lt = tile - v.tile_begin;
    const int px = (lt % v.ntx) * 8 + (lane & 7), py = (lt / v.ntx) * 4 + (lane >> 3);
    bool active = px < v.W && py < v.H && (lane << p.parts_log) >> 5 == part;
    const int pix0 = (lt / v.ntx) * 4 * v.W + (lt % v.ntx) * 8, HW = v.H * v.W;
    bool other = false;  // the ray has a gradient of depth or normals
    Cursor cur = first_cursor(p.tmin_inclusive);
    long long ray_g = 0;
    if (active) {
      const int pix = py * v.W + px;
      ray_g = v.ray_begin + pix;
      const float3 d = make_float3(v.ray_d[3 * pix], v.ray_d[3 * pix + 1], v.ray_d[3 * pix + 2]);
      if (v.interval) clip_cursor(cur, v.interval, HW, pix);
      const float gD = __ldg(v.dL_doth + kDepthCh * HW + pix);
      const float gN0 = __ldg(v.dL_doth + (kNormalCh + 0) * HW + pix);
      const float gN1 = __ldg(v.dL_doth + (kNormalCh + 1) * HW + pix);
      const float gN2 = __ldg(v.dL_doth + (kNormalCh + 2) * HW + pix);
      other = gD != 0.f || gN0 != 0.f || gN1 != 0.f || gN2 != 0.f;
      am.ray[lane] = make_float4(d.x, d.y, d.z, gD);
      am.ray[32 + lane] =
          make_float4(__ldg(v.dL_dpix + pix), __ldg(v.dL_dpix + HW + pix), __ldg(v.dL_dpix + 2 * HW + pix), 1.0f);
      am.ray[96 + lane] = make_float4(0.f, 0.f, 0.f, gN0);
      am.gn12[lane] = make_float2(gN1, gN2);
      if (EXACT) {
        am.exact[lane] = __ldg(v.dL_doth + kDistortionCh * HW + pix);
        am.exact[32 + lane] = __ldg(v.dL_doth + kMidDepthCh * HW + pix);
        am.exact[64 + lane] = 0.0f;
      }
      if (!p.cols) {
        float B[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) B[i] = 0.f;
        sh_basis(unit(d), p.sh_degree, B);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          reinterpret_cast<float4*>(am.basis + 16 * lane)[i] = make_float4(B[4 * i], B[4 * i + 1], B[4 * i + 2], B[4 * i + 3]);
      }
    }
    const bool others = __any_sync(full, other);
    if (others) {
      am.ray[64 + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else if (active) {
      const int pix = py * v.W + px;
      am.ray[64 + lane] =
          make_float4(__ldg(v.colors + pix), __ldg(v.colors + HW + pix), __ldg(v.colors + 2 * HW + pix), v.ray_o[3 * pix]);
      am.gn12[lane] = make_float2(v.ray_o[3 * pix + 1], v.ray_o[3 * pix + 2]);
    }
    uint32_t next = kNoEntry;
    for (bool first = true; __any_sync(full, active); first = false) {
      // the cache holds every query of every march
      bool have = active && (first || cache_has<K>(p, next, cur.key_min));
      if (active && !have) {
        atomicOr(p.status, kStatusCacheMiss);
        active = false;
      }
      replays += __popc(__ballot_sync(full, have));
      float t_drop = INFINITY;
      float* rows = nullptr;
      int rstride = 0;
      if (have) {
        if (colors) rows = cache_color_rows<K>(p, first, ray_g, next, rstride);
        t_drop = cache_get<K>(p, first, ray_g, next, sm, next);
      }
      March m;
      bool marching = have;
      while (__any_sync(full, marching)) {
        // ---- each ray lists its next hits
        unsigned long long slots = 0ull;
        int count = 0, state = kMarchVisit;
        while (marching && count < kVisits) {
          state = march_next<K, false>(sm, t_drop, m, cur, p.tmin_inclusive, p.bvh.P, p.status, cnt);
          if (state != kMarchVisit) break;
          slots |= (unsigned long long)m.i << (8 * count);
          ++count;
        }
        if (marching && state != kMarchVisit) {
          marching = false;
          if (state == kMarchDone) {
            active = false;
          } else if (++cur.chunks >= kMaxChunks) {
            atomicOr(p.status, kStatusTimeout);
            active = false;
          }
        }
        int at = count;
#pragma unroll
        for (int i = 1; i < 32; i <<= 1) {
          const int u = __shfl_up_sync(full, at, i);
          if (lane >= i) at += u;
        }
        const int total = __shfl_sync(full, at, 31);
        at -= count;
        for (int i = 0; i < count && TT_IN_BOUNDS(p.status, at + i < 32 * kVisits); ++i)
          am.list[at + i] = (unsigned short)((lane << 8) | (int)((slots >> (8 * i)) & 0xFFu));
        __syncwarp();
        // ---- the hits of all rays, 32 at a time
        for (int base = 0; base < total; base += 32) {
          const bool on = base + lane < total;
          const int e = on ? am.list[base + lane] : (32 << 8);
          const int ray = e >> 8, slot = e & 0xFF;
          const int before = __shfl_up_sync(full, ray, 1);
          const unsigned heads = __ballot_sync(full, lane == 0 || ray != before);
          const int seg = 31 - __clz(heads & (full >> (31 - lane)));
          const bool tail = on && (lane == 31 || ((heads >> (lane + 1)) & 1u));
          float* crow = reinterpret_cast<float*>(
              __shfl_sync(full, reinterpret_cast<unsigned long long>(rows), ray & 31));
          const int cstride = __shfl_sync(full, rstride, ray & 31);
          float T0 = -1.0f;
          float4 q0, q1;  // d, gD | g, T
          const int pix = pix0 + ((ray & 31) >> 3) * v.W + (ray & 7);  // the ray's
          Geom g;
          float alpha = 0.f, opacity = 0.f, sig = 0.f;
          uint32_t prim = 0;
          float3 raw = make_float3(0.f, 0.f, 0.f);
          if (on && TT_IN_BOUNDS(p.status, slot < K && ray < 32)) {
            const unsigned long long key = sm.keys[slot * sm.stride + (ray - lane)];
            prim = key_prim(key);
            const float4* tr = p.bvh.tri_prim + 3 * (size_t)prim;
            const float4 a = __ldg(tr), b = __ldg(tr + 1), c = __ldg(tr + 2);
            sig = __ldg(p.sigma + prim);
            opacity = __ldg(p.opac + prim);
            if (p.cols)
              raw = make_float3(__ldg(p.cols + 3 * prim), __ldg(p.cols + 3 * prim + 1), __ldg(p.cols + 3 * prim + 2));
            else if (crow)
              raw = make_float3(crow[(size_t)slot * cstride], crow[(size_t)slot * cstride + 1],
                                crow[(size_t)slot * cstride + 2]);
            float3 o;
            if (others) {
              o = make_float3(__ldg(v.ray_o + 3 * pix), __ldg(v.ray_o + 3 * pix + 1), __ldg(v.ray_o + 3 * pix + 2));
            } else {
              const float2 yz = am.gn12[ray];
              o = make_float3(reinterpret_cast<const float*>(am.ray + 64 + ray)[3], yz.x, yz.y);
            }
            q0 = am.ray[ray];
            q1 = am.ray[32 + ray];
            T0 = q1.w;
            g = shade_geom<MODE>(a, b, c, o, make_float3(q0.x, q0.y, q0.z), key_t(key), sig);
            alpha = fminf(kAlphaMax, opacity * g.Cx);
            if (alpha < kAlphaMin) alpha = 0.f;
          }
          // transmittance in front of and behind the hit
          float T = T0, test_T = T0 * (1.0f - alpha);
#pragma unroll
          for (int i = 1; i < kVisits; ++i) {
            const float u = __shfl_up_sync(full, test_T, 1);
            if (lane - seg == i) {
              T = u;
              test_T = T * (1.0f - alpha);
            }
          }
          const unsigned ended = __ballot_sync(full, on && test_T < kTMin);
          const bool dead = (ended & (full << seg) & (full >> (31 - lane))) != 0u;
          const bool blend = on && alpha > 0.f && !dead;
          const float w = blend ? alpha * T : 0.f;
          float c0 = 0.f, c1 = 0.f, c2 = 0.f, E = 0.f;
          float Cf0, Cf1, Cf2;                    // the ray's outputs
          float Df = 0.f, Wf = 0.f, distf = 0.f;  // EXACT
          float4 x = make_float4(0.f, 0.f, 0.f, 0.f);  // running sums of the colour, gN0
          if (on) x = am.ray[96 + ray];
          if (blend) {
            if (others) {
              Cf0 = __ldg(v.colors + pix);
              Cf1 = __ldg(v.colors + HW + pix);
              Cf2 = __ldg(v.colors + 2 * HW + pix);
            } else {
              const float4 y = am.ray[64 + ray];
              Cf0 = y.x;
              Cf1 = y.y;
              Cf2 = y.z;
            }
            if (!p.cols && !crow) raw = sh_raw_cold(p.shs, p.M, p.sh_degree, (int)prim, am.basis + 16 * ray);
            c0 = p.cols ? raw.x : fmaxf(raw.x, 0.f);
            c1 = p.cols ? raw.y : fmaxf(raw.y, 0.f);
            c2 = p.cols ? raw.z : fmaxf(raw.z, 0.f);
            if (EXACT) {
              Df = __ldg(v.others + kDepthCh * HW + pix);
              Wf = __ldg(v.others + kAlphaCh * HW + pix);
              distf = __ldg(v.others + kDistortionCh * HW + pix);
              const float Cf = Wf > 0.f ? (distf + Df * Df) / Wf : 0.f;
              E = g.t * g.t * Wf - 2.0f * g.t * Df + Cf;
            }
          }
          // the running sums, hit by hit like the transmittance
          const float w0 = c0 * w, w1 = c1 * w, w2 = c2 * w;
          x.x += w0, x.y += w1, x.z += w2;
#pragma unroll 1  // (unrolled, the kernel's code passes the instruction cache)
          for (int i = 1; i < kVisits; ++i) {
            const float u0 = __shfl_up_sync(full, x.x, 1), u1 = __shfl_up_sync(full, x.y, 1),
                        u2 = __shfl_up_sync(full, x.z, 1);
            if (lane - seg == i) x.x = u0 + w0, x.y = u1 + w1, x.z = u2 + w2;
          }
          float Sd = 0.f;
          if (EXACT) Sd = (on ? am.exact[64 + ray] : 0.f) + seg_sum(w * E, lane, seg);
          const float inv1a = 1.0f / (1.0f - alpha);
          float dL_dalpha = 0.f;
          if (blend)
            dL_dalpha = alpha_grad_color(q1.x, q1.y, q1.z, c0, c1, c2, Cf0 - x.x, Cf1 - x.y, Cf2 - x.z, T, inv1a);
          float3 dL_dn = make_float3(0.f, 0.f, 0.f);
          if (others) {
            float4 y = on ? am.ray[64 + ray] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float n0 = blend ? g.n.x * w : 0.f, n1 = blend ? g.n.y * w : 0.f, n2 = blend ? g.n.z * w : 0.f,
                        nD = blend ? w * g.t : 0.f;
            y.x += n0, y.y += n1, y.z += n2, y.w += nD;
#pragma unroll 1
            for (int i = 1; i < kVisits; ++i) {
              const float u0 = __shfl_up_sync(full, y.x, 1), u1 = __shfl_up_sync(full, y.y, 1),
                          u2 = __shfl_up_sync(full, y.z, 1), uD = __shfl_up_sync(full, y.w, 1);
              if (lane - seg == i) y.x = u0 + n0, y.y = u1 + n1, y.z = u2 + n2, y.w = uD + nD;
            }
            if (blend) {
              const float2 gn = am.gn12[ray];
              dL_dn = make_float3(x.w * w, gn.x * w, gn.y * w);
              const float D = EXACT ? Df : __ldg(v.others + kDepthCh * HW + pix);
              const float Nf0 = __ldg(v.others + (kNormalCh + 0) * HW + pix);
              const float Nf1 = __ldg(v.others + (kNormalCh + 1) * HW + pix);
              const float Nf2 = __ldg(v.others + (kNormalCh + 2) * HW + pix);
              dL_dalpha += q0.w * (T * g.t - (D - y.w) * inv1a);
              dL_dalpha += alpha_grad_color(x.w, gn.x, gn.y, g.n.x, g.n.y, g.n.z, Nf0 - y.x, Nf1 - y.y, Nf2 - y.z, T, inv1a);
            }
            __syncwarp();
            if (tail) am.ray[64 + ray] = y;
          }
          const unsigned bm = __ballot_sync(full, blend);
          const int nb = __popc(bm), rank = __popc(bm & ((1u << lane) - 1u));
          float3 gv[3];
          if (blend) {
            float dL_dt = q0.w * w;
            if (EXACT) {
              const float gDist = am.exact[ray];
              dL_dalpha += gDist * (T * E - (2.0f * distf - Sd) * inv1a);
              dL_dt += gDist * 2.0f * w * (g.t * Wf - Df);
              if (T > 0.5f && test_T <= 0.5f) dL_dt += am.exact[32 + ray];
            }
            hit_grads<MODE>(p, prim, g, make_float3(q0.x, q0.y, q0.z), sig, opacity, dL_dalpha, dL_dt,
                            dL_dn, gv);
            // colour gradients: dRGB/dsh_k = B_k, masked where the colour was clamped at 0
            const bool m0 = !p.cols && raw.x < 0.f, m1 = !p.cols && raw.y < 0.f, m2 = !p.cols && raw.z < 0.f;
            const float e0 = m0 ? 0.f : q1.x * w, e1 = m1 ? 0.f : q1.y * w, e2 = m2 ? 0.f : q1.z * w;
            float4* st = reinterpret_cast<float4*>(am.stage) + 2 * rank;
            st[0] = make_float4(e0, e1, e2, e0);
            st[1] = make_float4(e1, __uint_as_float(prim), __int_as_float(ray), 0.f);
          }
          __syncwarp();
          if (sh16) {
            // two hits of 12 chunks at a time; chunk j holds the products of
            // coefficients k = 4j / 3 and k + 1, starting at channel j % 3
            if (lane < 24) {
              const int j = lane % 12, k = 4 * j / 3, c = j % 3;
              for (int h = lane / 12; h < nb; h += 2) {
                const float* st = am.stage + 8 * h;
                const float* B = am.basis + 16 * __float_as_int(st[6]) + k;
                const float b0 = B[0], b1 = B[1];
                const float ea = st[c], eb = st[c + 1], ec = st[c + 2];
                red_add4(p.d_sh + (size_t)__float_as_uint(st[5]) * 48 + 4 * j, b0 * ea, (c == 2 ? b1 : b0) * eb,
                         (c == 0 ? b0 : b1) * ec, b1 * ea);
              }
            }
          } else {
            for (int i = lane; i < nb * row; i += 32) {
              const int h = i / row, c = i - h * row;
              const float* st = am.stage + 8 * h;
              const uint32_t pr = __float_as_uint(st[5]);
              if (p.cols)
                red_add(p.d_cols + 3 * (size_t)pr + c, st[c]);
              else
                red_add(p.d_sh + (size_t)pr * p.M * 3 + c, am.basis[16 * __float_as_int(st[6]) + c / 3] * st[c % 3]);
            }
          }
          __syncwarp();
          if (blend) {
            float* st = am.stage + 9 * rank;
            st[0] = gv[0].x, st[1] = gv[0].y, st[2] = gv[0].z;
            st[3] = gv[1].x, st[4] = gv[1].y, st[5] = gv[1].z;
            st[6] = gv[2].x, st[7] = gv[2].y, st[8] = gv[2].z;
            am.stage[9 * 32 + rank] = __int_as_float(__ldg(p.cumsum + prim));
          }
          __syncwarp();
          if (lane < 27) {
            const int c = lane % 9;
            for (int h = lane / 9; h < nb; h += 3)
              red_add(p.d_tri + 3 * (size_t)__float_as_int(am.stage[9 * 32 + h]) + c, am.stage[9 * h + c]);
          }
          __syncwarp();
          if (tail) {
            reinterpret_cast<float*>(am.ray + 32 + ray)[3] = dead ? -1.0f : test_T;
            am.ray[96 + ray] = x;
            if (EXACT) am.exact[64 + ray] = Sd;
          }
          __syncwarp();
        }
        if (marching || active) {
          if (reinterpret_cast<const float*>(am.ray + 32 + lane)[3] < 0.f) marching = active = false;
        }
      }
    }
    __syncwarp();
  }
  if (lane == 0 && replays != 0u) atomicAdd(p.stats + kStatReplays, (unsigned long long)replays);
}

// ---------------------------------------------------------------- secondary rays
// Secondary-ray passes over a device ray queue (no reference counterpart; the
// reference bends rays only at one analytic sphere). Per pixel a tree of
// rays: the first blended hit of a ray of depth < max_depth on a triangle of
// material 1 spawns a reflected and (unless totally reflected) a refracted
// ray from the exact hit point, and that hit's colour is
// F L(reflected) + (1 - F) L(refracted) instead of its SH colour; rays that
// leave the scene see a lat-long environment map in place of bg. One launch
// per level traces the level's rays from its queue and appends their
// children to the next level's queue (atomic slot counter); resolve launches
// then add each child's radiance to its parent, deepest level first, and
// write the pixel colours. The adjoint traces every ray of every level in one
// launch with upstream gradient tau dL/dpixel, taking the spawning hit's
// colour from the children's resolved radiance.

// Per-lane persistent driver over `total` queue items (item order = record
// order); lanes refill as their rays finish. With SD = 0 the queries go through
// the warp's pair stack `pm` instead of a stack a lane.
template <int SD, class Shader>
__device__ __forceinline__ void drive_items(const TraceParams& p, const Smem& sm, Shader& sh, Counters& cnt,
                                            int total, PairMem pm = PairMem{}) {
  constexpr int K = kChunk;
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  bool have = false, exhausted = false;
  Cursor cur = first_cursor(p.tmin_inclusive);
  float3 o = make_float3(0.f, 0.f, 0.f), d = o;
  uint32_t* link = nullptr;  // forward: where the entry of the ray's next query gets linked
  uint32_t next = kNoEntry;  // adjoint: entry of the ray's next query
  const bool replay = cache_replays<K>(p);
  for (;;) {
    const unsigned need = __ballot_sync(full, !have && !exhausted);
    if (need) {
      const int leader = __ffs(need) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(p.work, __popc(need));
      base = __shfl_sync(full, base, leader);
      if (!have && !exhausted) {
        const int item = base + __popc(need & lt);
        if (item >= total) {
          exhausted = true;
        } else {
          sh.begin_item(item, o, d);
          cur = first_cursor(p.tmin_inclusive);
          have = true;
        }
      }
    }
    if (__ballot_sync(full, have) == 0) {
      if (__all_sync(full, exhausted)) break;
      continue;
    }
    float t_drop = INFINITY;
    if constexpr (SD == 0)  // (no queries to replay where pairs are used)
      pair_query<K>(p.bvh, make_ray(o, d), have, cur.key_min, cur.t_hi, sm.keys, sm.stride, pm, t_drop, p.status, cnt,
                    p.count_work);
    if (have) {
      // Hit cache: a level-0 ray (record = pixel) keeps its first query in
      // the main part; a deeper ray starts its chain in the pool, linked from
      // its queue record
      const bool first = cur.chunks == 0;
      const bool main_part = first && sh.ridx < p.cache_rays;
      uint32_t* rec_link = &p.sec.rec[sh.ridx].cache_link;
      if (replay && first && !main_part) next = __ldcg(rec_link);
      if (replay && (main_part || cache_has<K>(p, next, cur.key_min))) {
        if (p.cache_mode == kCacheFill) link = cache_link_of<K>(p, main_part, sh.ridx, next);
        t_drop = cache_get<K>(p, main_part, sh.ridx, next, sm, next);
        ++cnt.replays;
      } else {
        next = kNoEntry;
        if constexpr (SD != 0) {
          const RayW r = make_ray(o, d);
          query<SD>(p.bvh, r, cur.key_min, cur.t_hi, sm.keys, sm.stride, sm.st, t_drop, p.status, cnt, p.count_work);
        }
        if (p.cache_mode == kCacheWrite || p.cache_mode == kCacheFill) {
          if (main_part) {
            link = cache_put_first<K>(p, sh.ridx, sm, t_drop);
          } else {
            if (first) link = rec_link;
            if (link) {
              const uint32_t e = atomicAdd(&cache_header_ptr(p)->pool_used, 1u);
              link = e < p.cache_pool_cap ? cache_put_more<K>(p, e, cur.key_min, sm, t_drop, link) : nullptr;
            }
          }
        }
      }
    }
    __syncwarp();
    if (have) {
      bool done = consume_chunk<K>(sm, t_drop, cur, p.tmin_inclusive, p.status, sh, cnt);
      if (!done && ++cur.chunks >= kMaxChunks) {
        atomicOr(p.status, kStatusTimeout);
        done = true;
      }
      // the collecting pass stores at most collect_queries queries a ray
      if (Shader::kStopsAtClip && p.collect_queries > 0 && cur.chunks >= p.collect_queries) done = true;
      if (done) {
        sh.end();
        have = false;
      }
    }
  }
}

// FP64 with explicit round-to-nearest operations (no contraction), in the
// oracle's operation order, so both spawn the same FP32 rays.
namespace sd {
struct V {
  double x, y, z;
};
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ V vsub(V a, V b) { return {sub(a.x, b.x), sub(a.y, b.y), sub(a.z, b.z)}; }
__device__ __forceinline__ V vadd(V a, V b) { return {add(a.x, b.x), add(a.y, b.y), add(a.z, b.z)}; }
__device__ __forceinline__ V vscale(V a, double s) { return {mul(a.x, s), mul(a.y, s), mul(a.z, s)}; }
__device__ __forceinline__ double dot(V a, V b) { return add(add(mul(a.x, b.x), mul(a.y, b.y)), mul(a.z, b.z)); }
__device__ __forceinline__ V cross(V a, V b) {
  return {sub(mul(a.y, b.z), mul(a.z, b.y)), sub(mul(a.z, b.x), mul(a.x, b.z)), sub(mul(a.x, b.y), mul(a.y, b.x))};
}
__device__ __forceinline__ V from(float4 v) { return {(double)v.x, (double)v.y, (double)v.z}; }
__device__ __forceinline__ V from(float3 v) { return {(double)v.x, (double)v.y, (double)v.z}; }
__device__ __forceinline__ float3 to_f(V v) {
  return make_float3(__double2float_rn(v.x), __double2float_rn(v.y), __double2float_rn(v.z));
}
}  // namespace sd

struct SpawnDev {
  float3 o, r, t;
  bool refracts;
  float F;
};

// Reflected / refracted rays at the hit of (o, d) on the triangle (a, b, c)
// with index of refraction ior: Schlick's Fresnel term, the exact hit point
// of an FP64 plane solve.
__device__ __noinline__ SpawnDev spawn_rays(float4 a4, float4 b4, float4 c4, float3 of, float3 df, float ior_f) {
  using namespace sd;
  const V A = from(a4), B = from(b4), C = from(c4), o = from(of), d = from(df);
  const V nc = cross(vsub(B, A), vsub(C, A));
  const double te = __ddiv_rn(dot(vsub(A, o), nc), dot(d, nc));
  const V x = vadd(o, vscale(d, te));
  const V n = vscale(nc, __ddiv_rn(1.0, __dsqrt_rn(dot(nc, nc))));
  const V du = vscale(d, __ddiv_rn(1.0, __dsqrt_rn(dot(d, d))));
  const double ior = (double)ior_f;
  const double cosi = dot(du, n);
  const bool entering = cosi < 0.0;
  const V nf = entering ? n : V{-n.x, -n.y, -n.z};
  const double c = entering ? -cosi : cosi;
  const double ei = entering ? 1.0 : ior, et = entering ? ior : 1.0;
  const double eta = __ddiv_rn(ei, et);
  const double q = __ddiv_rn(sub(ei, et), add(ei, et));
  const double r0 = mul(q, q);
  const double k = sub(1.0, mul(mul(eta, eta), sub(1.0, mul(c, c))));
  SpawnDev sp;
  sp.o = to_f(x);
  sp.r = to_f(vadd(du, vscale(nf, mul(2.0, c))));
  sp.refracts = k >= 0.0;
  double F = 1.0;
  V t = du;
  if (sp.refracts) {
    const double m = sub(1.0, c);
    const double m2 = mul(m, m);
    F = add(r0, mul(sub(1.0, r0), mul(mul(m2, m2), m)));
    t = vadd(vscale(du, eta), vscale(nf, sub(mul(eta, c), __dsqrt_rn(k))));
  }
  sp.t = to_f(t);
  sp.F = __double2float_rn(F);
  return sp;
}

// Lat-long lookup: longitude atan2(d.z, d.x) over the columns (wrapping),
// colatitude acos(d.y) over the rows (clamped), bilinear between texel centres.
// env_texels gives the four texels (word offsets of their RGB) and the
// bilinear fractions; the adjoint scatters into the same four.
struct EnvTexels {
  size_t t00, t01, t10, t11;
  float ax, ay;
};

__device__ __forceinline__ EnvTexels env_texels(const SecParams& s, float3 d) {
  const float kPi = 3.14159265358979f;
  const float len = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
  const float u = atan2f(d.z, d.x) * (0.5f / kPi) + 0.5f;
  const float v = acosf(fminf(1.f, fmaxf(-1.f, d.y / len))) * (1.0f / kPi);
  float fx = u * (float)s.env_w - 0.5f, fy = v * (float)s.env_h - 0.5f;
  if (!(fabsf(fx) <= (float)s.env_w)) fx = 0.f;  // NaN direction: any texel, never out of bounds
  if (!(fabsf(fy) <= (float)s.env_h)) fy = 0.f;
  const float x0f = floorf(fx), y0f = floorf(fy);
  const int W = s.env_w, H = s.env_h;
  const int x0 = (((int)x0f % W) + W) % W, x1 = (x0 + 1) % W;
  const int y0 = max(0, min(H - 1, (int)y0f)), y1 = max(0, min(H - 1, (int)y0f + 1));
  EnvTexels t;
  t.ax = fx - x0f;
  t.ay = fy - y0f;
  t.t00 = ((size_t)y0 * W + x0) * 3;
  t.t01 = ((size_t)y0 * W + x1) * 3;
  t.t10 = ((size_t)y1 * W + x0) * 3;
  t.t11 = ((size_t)y1 * W + x1) * 3;
  return t;
}

__device__ __forceinline__ float3 env_lookup(const SecParams& s, float3 d) {
  const EnvTexels t = env_texels(s, d);
  const float ax = t.ax, ay = t.ay;
  const float* e = s.env;
  float out[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float t00 = __ldg(e + t.t00 + c), t01 = __ldg(e + t.t01 + c);
    const float t10 = __ldg(e + t.t10 + c), t11 = __ldg(e + t.t11 + c);
    out[c] = (1.f - ay) * ((1.f - ax) * t00 + ax * t01) + ay * ((1.f - ax) * t10 + ax * t11);
  }
  return make_float3(out[0], out[1], out[2]);
}

// Adjoint of T env(d) in a ray's radiance: dL/d(texel) += g T (bilinear weight).
__device__ __forceinline__ void env_lookup_bwd(const SecParams& s, float3 d, float T, float g0, float g1, float g2) {
  const EnvTexels t = env_texels(s, d);
  const float ax = t.ax, ay = t.ay;
  const float wt[4] = {(1.f - ay) * (1.f - ax), (1.f - ay) * ax, ay * (1.f - ax), ay * ax};
  const size_t at[4] = {t.t00, t.t01, t.t10, t.t11};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float f = T * wt[k];
    red_add(s.d_env + at[k] + 0, g0 * f);
    red_add(s.d_env + at[k] + 1, g1 * f);
    red_add(s.d_env + at[k] + 2, g2 * f);
  }
}

// d F / d ior of Schlick's reflected share F at a refracting hit:
// F = r0 + (1 - r0) (1 - cos)^5 with r0 = ((ior - 1) / (ior + 1))^2 (either
// side of the interface), so dF/dior = dr0/dior (1 - F) / (1 - r0) and
// dr0/dior = 4 (ior - 1) / (ior + 1)^3.
__device__ __forceinline__ float fresnel_dF_dior(float n, float F) {
  const float q = (n - 1.f) / (n + 1.f);
  const float n1 = n + 1.f;
  return 4.f * (n - 1.f) / (n1 * n1 * n1) * (1.f - F) / (1.f - q * q);
}

// The rays of one level: trace, composite, spawn children into the next level.
struct SecShader {
  static constexpr bool kStopsAtClip = false;
  const TraceParams& p;
  const ViewDesc* v;
  int ridx, pix, level;
  float3 o, d;
  float C0, C1, C2, N0, N1, N2, T, tau;
  bool spawned;
  unsigned n_rays = 0, n_eval = 0, n_blend = 0;

  __device__ explicit SecShader(const TraceParams& params) : p(params), v(&params.views[0]), level(params.sec.level) {}

  __device__ __forceinline__ void begin_item(int i, float3& ro, float3& rd) {
    const SecParams& s = p.sec;
    ridx = s.base[level] + (level > 0 && s.order ? (int)__ldg(s.order + i) : i);
    SecRecord* r = s.rec + ridx;
    if (level == 0) {
      pix = i;
      ro = make_float3(v->ray_o[3 * pix], v->ray_o[3 * pix + 1], v->ray_o[3 * pix + 2]);
      rd = make_float3(v->ray_d[3 * pix], v->ray_d[3 * pix + 1], v->ray_d[3 * pix + 2]);
      tau = 1.0f;
      r->pixel = pix;
      r->tau = 1.0f;
    } else {
      ro = make_float3(r->o[0], r->o[1], r->o[2]);
      rd = make_float3(r->d[0], r->d[1], r->d[2]);
      pix = r->pixel;
      tau = r->tau;
    }
    r->child_r = r->child_t = -1;
    r->F = r->w = 0.f;
    o = ro;
    d = rd;
    C0 = C1 = C2 = N0 = N1 = N2 = 0.f;
    T = 1.0f;
    spawned = false;
    ++n_rays;
  }

  // The packet driver's entry (level 0): the primary ray of `pixel`.
  __device__ __forceinline__ bool begin(const ViewDesc*, int pixel, float3, float3) {
    float3 ro, rd;
    begin_item(pixel, ro, rd);
    return true;
  }

  __device__ __forceinline__ void prepare() {}

  __device__ __forceinline__ int push_child(float3 co, float3 cd, float ctau) {
    const SecParams& s = p.sec;
    const int slot = atomicAdd(s.count + level + 1, 1);
    if (slot >= s.cap[level + 1]) {
      atomicOr(p.status, kStatusStack);
      return -1;
    }
    SecRecord* c = s.rec + s.base[level + 1] + slot;
    c->o[0] = co.x;
    c->o[1] = co.y;
    c->o[2] = co.z;
    c->d[0] = cd.x;
    c->d[1] = cd.y;
    c->d[2] = cd.z;
    c->pixel = pix;
    c->tau = ctau;
    c->cache_link = kNoEntry;
    return slot;
  }

  __device__ __forceinline__ bool visit(uint32_t prim, float) {
    const float4* tr = p.bvh.tri_prim + 3 * (size_t)prim;
    const float4 a = __ldg(tr), b = __ldg(tr + 1), c = __ldg(tr + 2);
    const Geom g = window_fn(a, b, c, o, d, __ldg(p.sigma + prim));
    ++n_eval;
    const float alpha = fminf(kAlphaMax, __ldg(p.opac + prim) * g.Cx);
    if (alpha < kAlphaMin) return false;
    const float test_T = T * (1.0f - alpha);
    if (test_T < kTMin) return true;
    ++n_blend;
    const float w = alpha * T;
    if (level == 0) {
      p.density[prim] = 1.0f;
      compute_scaling(p.scaling, p.verts, p.cumsum, p.num_points, (int)prim, o);
      atomicMax(reinterpret_cast<int*>(p.max_blending) + prim, __float_as_int(w));
      N0 += g.n.x * w;
      N1 += g.n.y * w;
      N2 += g.n.z * w;
    }
    const SecParams& s = p.sec;
    if (!spawned && level < s.max_depth && __ldg(s.material + prim) == 1) {
      // the hit's colour comes from its children at the resolve
      spawned = true;
      const SpawnDev sp = spawn_rays(a, b, c, o, d, __ldg(s.ior + prim));
      SecRecord* r = s.rec + ridx;
      r->F = sp.F;
      r->w = w;
      r->child_r = push_child(sp.o, sp.r, tau * w * sp.F);
      if (sp.refracts) r->child_t = push_child(sp.o, sp.t, tau * w * (1.0f - sp.F));
    } else {
      float B[16];
      sh_basis(unit(d), p.sh_degree, B);
      const float3 col = sh_raw(p.shs, p.M, (int)prim, p.sh_degree, B);
      C0 += fmaxf(col.x, 0.f) * w;
      C1 += fmaxf(col.y, 0.f) * w;
      C2 += fmaxf(col.z, 0.f) * w;
    }
    T = test_T;
    return false;
  }

  __device__ __forceinline__ void end() {
    const float3 e = env_lookup(p.sec, d);
    SecRecord* r = p.sec.rec + ridx;
    r->L[0] = C0 + T * e.x;
    r->L[1] = C1 + T * e.y;
    r->L[2] = C2 + T * e.z;
    if (level == 0) {
      const int HW = v->H * v->W;
      v->out_others[kDepthCh * HW + pix] = 0.0f;
      v->out_others[kAlphaCh * HW + pix] = 1.0f - T;
      v->out_others[(kNormalCh + 0) * HW + pix] = N0;
      v->out_others[(kNormalCh + 1) * HW + pix] = N1;
      v->out_others[(kNormalCh + 2) * HW + pix] = N2;
      v->out_others[kMidDepthCh * HW + pix] = 0.0f;
      v->out_others[kDistortionCh * HW + pix] = 0.0f;
    }
  }
};

__device__ __forceinline__ int sec_level_size(const TraceParams& p, int level) {
  return level == 0 ? p.views[0].H * p.views[0].W : min(__ldcg(p.sec.count + level), p.sec.cap[level]);
}

// Level 0: the primary rays are camera-coherent, so they are traced as warp
// packets of 8x4 pixels (with the hit cache's 16 hits per query), in a kernel
// of their own (the lane driver's registers would spill in the same kernel).
__global__ void __launch_bounds__(kTraceThreads, kMinBlocks) k_sec_primary(const __grid_constant__ TraceParams p) {
  cache_header<kChunk>(p);  // the deeper levels append to the same cache
  Counters cnt;
  SecShader sh(p);
  unsigned char* rest;
  const Smem sm = packet_smem<kChunk>(rest);
  drive_packets<kChunk>(p, sm, warp_stack(rest), sh, cnt);
  cnt.queries += cnt.replays;  // replayed from the traversal pass (split schedule): used by the march all the same
  cnt.replays = 0;
  add_stats(p.stats, sh.n_rays, sh.n_eval, sh.n_blend, cnt);
}

// Levels >= 1: spawned rays, shaded one a lane. Their queries come from the
// traversal pass before (pairs, k_sec_collect); a query it did not store, and every
// one with TT_OPT_SPLIT_FORWARD off, is traversed here with a kSecStack-entry
// stack in shared memory per lane (continued in local memory), kSecBlocks blocks
// per SM.
#ifndef TT_SEC_STACK
#define TT_SEC_STACK 32
#endif
#ifndef TT_SEC_BLOCKS
#define TT_SEC_BLOCKS 4
#endif
constexpr int kSecStack = TT_SEC_STACK, kSecBlocks = TT_SEC_BLOCKS;
constexpr size_t sec_trace_smem() { return (size_t)kTraceThreads * (kSecStack * 8 + kChunk * 8); }

__global__ void __launch_bounds__(kTraceThreads, kSecBlocks) k_sec_trace(const __grid_constant__ TraceParams p) {
  Counters cnt;
  SecShader sh(p);
  drive_items<kSecStack>(p, thread_smem<kSecStack>(), sh, cnt, sec_level_size(p, p.sec.level));
  cnt.queries += cnt.replays;  // replayed from the traversal pass (split schedule): used by the march all the same
  cnt.replays = 0;
  add_stats(p.stats, sh.n_rays, sh.n_eval, sh.n_blend, cnt);
}

// Traversal pass of a spawned level (split schedule): the level's rays, in
// the same order, with a shader that shades and spawns nothing, storing every
// query in the ray tree's hit cache (the chain starts at the ray's record);
// k_sec_trace then replays them in fill mode. Like k_collect for primary
// rays, it needs fewer registers without the shading and spawning code; its
// rays are traced as pairs. 5 blocks per SM (96 registers): 7.9 ms on the
// workload above, 8.0 at 4.
#ifndef TT_SEC_COLLECT_BLOCKS
#define TT_SEC_COLLECT_BLOCKS 5
#endif
constexpr int kSecCollectBlocks = TT_SEC_COLLECT_BLOCKS;
constexpr size_t sec_collect_smem() { return pair_smem<kChunk>(); }

struct SecMarchShader {
  static constexpr bool kStopsAtClip = true;
  const TraceParams& p;
  int ridx = 0;
  __device__ explicit SecMarchShader(const TraceParams& params) : p(params) {}
  __device__ __forceinline__ void begin_item(int i, float3& ro, float3& rd) {
    const SecParams& s = p.sec;
    ridx = s.base[s.level] + (s.order ? (int)__ldg(s.order + i) : i);
    const SecRecord* r = s.rec + ridx;
    ro = make_float3(r->o[0], r->o[1], r->o[2]);
    rd = make_float3(r->d[0], r->d[1], r->d[2]);
  }
  __device__ __forceinline__ void prepare() {}
  __device__ __forceinline__ bool visit(uint32_t, float) { return false; }
  __device__ __forceinline__ void end() {}
};

__global__ void __launch_bounds__(kTraceThreads, kSecCollectBlocks) k_sec_collect(const __grid_constant__ TraceParams p) {
  Counters cnt;
  SecMarchShader sh(p);
  unsigned char* rest;
  const Smem sm = packet_smem<kChunk>(rest);
  drive_items<0>(p, sm, sh, cnt, sec_level_size(p, p.sec.level), pair_mem(rest));
  cnt.queries = 0;  // counted by the shading pass (k_sec_trace), like k_collect
  add_stats(p.stats, 0u, 0u, 0u, cnt);
}

// Sort keys of the spawned rays of level p.sec.level: the direction in 16 x
// 16 octahedral bins (8 bits) over the Morton code of the origin, 7 bits an
// axis, within the root box of the BVH (21 bits); slots past the level's
// count get 0xFFFFFFFF and sort after every ray. The order was chosen when these
// rays were traversed one a lane (500k triangles, 2 views of 800^2, two bounces, a
// step): 29.9 ms, against 30.7 with the direction octant over a 27-bit Morton code and
// 32.5 with the origin first; finer direction bins (1024, 4096) or coarser origins
// were slower. Pairs depend on it less (TT_OPT_SORT_SECONDARY).
__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // 9 bits -> every third of 27
  v &= 0x1FFu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

__global__ void k_sec_sort_keys(const __grid_constant__ TraceParams p, uint32_t* __restrict__ keys,
                                uint32_t* __restrict__ vals) {
  const SecParams& s = p.sec;
  const int level = s.level, cap = s.cap[level];
  const int n = min(__ldcg(s.count + level), cap);
  // the root's box: the union of its 8 child boxes (empty slots are inverted)
  float lo[3] = {0.f, 0.f, 0.f}, ext[3] = {1.f, 1.f, 1.f};
  if (p.bvh.has_root && p.bvh.P >= 2) {
    const float* nd = reinterpret_cast<const float*>(p.bvh.nodes);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float l = INFINITY, h = -INFINITY;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        l = fminf(l, __ldg(nd + 16 * a + c));
        h = fmaxf(h, __ldg(nd + 16 * a + 8 + c));
      }
      if (l < h) {
        lo[a] = l;
        ext[a] = h - l;
      }
    }
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += gridDim.x * blockDim.x) {
    uint32_t key = 0xFFFFFFFFu;
    if (i < n) {
      const SecRecord& r = s.rec[s.base[level] + i];
      uint32_t q[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) q[a] = (uint32_t)fminf(fmaxf((r.o[a] - lo[a]) / ext[a] * 512.f, 0.f), 511.f);
      // octahedral map of the direction onto [-1, 1]^2 (lower hemisphere folded out)
      const float ad = fabsf(r.d[0]) + fabsf(r.d[1]) + fabsf(r.d[2]);
      float ux = ad > 0.f ? r.d[0] / ad : 0.f, uy = ad > 0.f ? r.d[1] / ad : 0.f;
      if (r.d[2] < 0.f) {
        const float fx = (1.f - fabsf(uy)) * (ux >= 0.f ? 1.f : -1.f);
        const float fy = (1.f - fabsf(ux)) * (uy >= 0.f ? 1.f : -1.f);
        ux = fx;
        uy = fy;
      }
      const uint32_t bx = (uint32_t)fminf(fmaxf((ux * 0.5f + 0.5f) * 16.f, 0.f), 15.f);
      const uint32_t by = (uint32_t)fminf(fmaxf((uy * 0.5f + 0.5f) * 16.f, 0.f), 15.f);
      key = (((bx << 4) | by) << 21) | (spread3(q[0] >> 2) << 2) | (spread3(q[1] >> 2) << 1) | spread3(q[2] >> 2);
    }
    keys[i] = key;
    vals[i] = (uint32_t)i;
  }
}

// Adds each record's children's radiance to it (their level is complete) and,
// for level 0, writes the pixel colours.
__global__ void k_sec_resolve(const __grid_constant__ TraceParams p) {
  const SecParams& s = p.sec;
  const int level = s.level;
  const int n = sec_level_size(p, level);
  const ViewDesc& v = p.views[0];
  const int HW = v.H * v.W;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    SecRecord* r = s.rec + s.base[level] + i;
    float L0 = r->L[0], L1 = r->L[1], L2 = r->L[2];
    if (r->child_r >= 0 || r->child_t >= 0) {
      float lr[3] = {0.f, 0.f, 0.f}, lt[3] = {0.f, 0.f, 0.f};
      if (r->child_r >= 0) {
        const SecRecord* c = s.rec + s.base[level + 1] + r->child_r;
        lr[0] = c->L[0];
        lr[1] = c->L[1];
        lr[2] = c->L[2];
      }
      if (r->child_t >= 0) {
        const SecRecord* c = s.rec + s.base[level + 1] + r->child_t;
        lt[0] = c->L[0];
        lt[1] = c->L[1];
        lt[2] = c->L[2];
      }
      const float F = r->F, w = r->w;
      L0 += w * (F * lr[0] + (1.0f - F) * lt[0]);
      L1 += w * (F * lr[1] + (1.0f - F) * lt[1]);
      L2 += w * (F * lr[2] + (1.0f - F) * lt[2]);
      r->L[0] = L0;
      r->L[1] = L1;
      r->L[2] = L2;
    }
    if (level == 0) {
      v.out_color[i] = L0;
      v.out_color[HW + i] = L1;
      v.out_color[2 * HW + i] = L2;
    }
  }
}

// Adjoint of every ray of every level (backward.cu's per-hit formulas with
// upstream gradient tau dL/dpixel; the spawning hit's colour is the
// children's resolved radiance and it has no SH gradient).
struct SecBwdShader {
  static constexpr bool kStopsAtClip = false;
  const TraceParams& p;
  const ViewDesc* v;
  int ridx, pix, level;
  float3 o, d;
  float Cf0, Cf1, Cf2, Df, Nf0, Nf1, Nf2;  // finals and upstream gradients as in RayGrads
  float g0, g1, g2, gD, gN0, gN1, gN2;
  RaySums x;
  float T;
  bool spawned;

  __device__ explicit SecBwdShader(const TraceParams& params) : p(params), v(&params.views[0]) {}

  __device__ __forceinline__ void begin_item(int item, float3& ro, float3& rd) {
    const SecParams& s = p.sec;
    level = 0;
    int i = item;
    while (level < s.max_depth && i >= sec_level_size(p, level)) {
      i -= sec_level_size(p, level);
      ++level;
    }
    // spawned levels in the order the forward traced them (neighbouring
    // items then gather the same triangles)
    const uint32_t* ord = level > 0 ? s.bwd_order[level] : nullptr;
    ridx = s.base[level] + (ord ? (int)__ldg(ord + i) : i);
    const SecRecord* r = s.rec + ridx;
    const int HW = v->H * v->W;
    float tau;
    if (level == 0) {
      pix = i;
      ro = make_float3(v->ray_o[3 * pix], v->ray_o[3 * pix + 1], v->ray_o[3 * pix + 2]);
      rd = make_float3(v->ray_d[3 * pix], v->ray_d[3 * pix + 1], v->ray_d[3 * pix + 2]);
      tau = 1.0f;
      // The exact adjoint differentiates the outputs the passes compute: the
      // depth channel is 0 there (as in the reference), so it has no gradient
      gD = p.mode == kShadeExact ? 0.f : __ldg(v->dL_doth + kDepthCh * HW + pix);
      gN0 = __ldg(v->dL_doth + (kNormalCh + 0) * HW + pix);
      gN1 = __ldg(v->dL_doth + (kNormalCh + 1) * HW + pix);
      gN2 = __ldg(v->dL_doth + (kNormalCh + 2) * HW + pix);
      Df = __ldg(v->others + kDepthCh * HW + pix);
      Nf0 = __ldg(v->others + (kNormalCh + 0) * HW + pix);
      Nf1 = __ldg(v->others + (kNormalCh + 1) * HW + pix);
      Nf2 = __ldg(v->others + (kNormalCh + 2) * HW + pix);
    } else {
      ro = make_float3(r->o[0], r->o[1], r->o[2]);
      rd = make_float3(r->d[0], r->d[1], r->d[2]);
      pix = r->pixel;
      tau = r->tau;
      Df = Nf0 = Nf1 = Nf2 = gD = gN0 = gN1 = gN2 = 0.f;
    }
    g0 = tau * __ldg(v->dL_dpix + pix);
    g1 = tau * __ldg(v->dL_dpix + HW + pix);
    g2 = tau * __ldg(v->dL_dpix + 2 * HW + pix);
    Cf0 = r->L[0];
    Cf1 = r->L[1];
    Cf2 = r->L[2];
    o = ro;
    d = rd;
    x = RaySums{};
    T = 1.0f;
    spawned = false;
  }

  __device__ __forceinline__ void prepare() {}

  __device__ __forceinline__ bool visit(uint32_t prim, float) {
    const float4* tr = p.bvh.tri_prim + 3 * (size_t)prim;
    const float sig = __ldg(p.sigma + prim);
    const Geom g = window_fn(__ldg(tr), __ldg(tr + 1), __ldg(tr + 2), o, d, sig);
    const float opacity = __ldg(p.opac + prim);
    const float alpha = fminf(kAlphaMax, opacity * g.Cx);
    if (alpha < kAlphaMin) return false;
    const float test_T = T * (1.0f - alpha);
    if (test_T < kTMin) return true;
    const float w = alpha * T;
    const SecParams& s = p.sec;
    float c0, c1, c2;
    float3 raw = make_float3(0.f, 0.f, 0.f);
    float B[16];
    const bool spawn = !spawned && level < s.max_depth && __ldg(s.material + prim) == 1;
    if (spawn) {
      spawned = true;
      const SecRecord* r = s.rec + ridx;
      const float Fr = r->F;
      float lr[3] = {0.f, 0.f, 0.f}, lt[3] = {0.f, 0.f, 0.f};
      if (r->child_r >= 0) {
        const SecRecord* c = s.rec + s.base[level + 1] + r->child_r;
        lr[0] = c->L[0];
        lr[1] = c->L[1];
        lr[2] = c->L[2];
      }
      if (r->child_t >= 0) {
        const SecRecord* c = s.rec + s.base[level + 1] + r->child_t;
        lt[0] = c->L[0];
        lt[1] = c->L[1];
        lt[2] = c->L[2];
      }
      c0 = Fr * lr[0] + (1.0f - Fr) * lt[0];
      c1 = Fr * lr[1] + (1.0f - Fr) * lt[1];
      c2 = Fr * lr[2] + (1.0f - Fr) * lt[2];
      if (s.d_ior && r->child_t >= 0) {  // a refracting hit: the colour depends on ior through F
        const float dL_dF = w * (g0 * (lr[0] - lt[0]) + g1 * (lr[1] - lt[1]) + g2 * (lr[2] - lt[2]));
        red_add(s.d_ior + prim, dL_dF * fresnel_dF_dior(__ldg(s.ior + prim), Fr));
      }
    } else {
      sh_basis(unit(d), p.sh_degree, B);
      raw = sh_raw(p.shs, p.M, (int)prim, p.sh_degree, B);
      c0 = fmaxf(raw.x, 0.f);
      c1 = fmaxf(raw.y, 0.f);
      c2 = fmaxf(raw.z, 0.f);
    }
    x.add(c0, c1, c2, g.n, g.t, w);
    const float inv1a = 1.0f / (1.0f - alpha);
    float dL_dalpha = alpha_grad_color(g0, g1, g2, c0, c1, c2, Cf0 - x.C0, Cf1 - x.C1, Cf2 - x.C2, T, inv1a);
    if (level == 0) {  // spawned rays only pass colour on
      dL_dalpha += gD * (T * g.t - (Df - x.D) * inv1a);
      dL_dalpha += alpha_grad_color(gN0, gN1, gN2, g.n.x, g.n.y, g.n.z, Nf0 - x.N0, Nf1 - x.N1, Nf2 - x.N2, T, inv1a);
    }
    const float3 dL_dn = make_float3(gN0 * w, gN1 * w, gN2 * w);
    float3 gv[3];
    if (p.mode == kShadeExact)  // the full chain rule of the window function and the face normal; spawn geometry held constant
      hit_grads<kShadeExact>(p, prim, g, d, sig, opacity, dL_dalpha, 0.0f, dL_dn, gv);
    else
      hit_grads<kShadeRef>(p, prim, g, d, sig, opacity, dL_dalpha, 0.0f, dL_dn, gv);
    if (spawn)
      scatter_vertices(p, prim, gv);
    else
      scatter_hit(p, prim, w, g0, g1, g2, raw, B, gv);
    T = test_T;
    return false;
  }

  // the environment term T env(d) of the ray's radiance
  __device__ __forceinline__ void end() {
    if (p.sec.d_env) env_lookup_bwd(p.sec, d, T, g0, g1, g2);
  }
};

__global__ void __launch_bounds__(kTraceThreads, 4) k_sec_backward(const __grid_constant__ TraceParams p) {
  Counters cnt;
  SecBwdShader sh(p);
  int total = 0;
  for (int l = 0; l <= p.sec.max_depth; ++l) total += sec_level_size(p, l);
  drive_items<32>(p, thread_smem<32>(), sh, cnt, total);
  const unsigned s = __reduce_add_sync(0xFFFFFFFFu, cnt.replays);
  if ((threadIdx.x & 31) == 0 && s != 0u) atomicAdd(p.stats + kStatReplays, (unsigned long long)s);
}

// ---------------------------------------------------------------- zero
__global__ void __launch_bounds__(256) k_zero(const __grid_constant__ ZeroList z) {
  const size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  for (int r = 0; r < z.n; ++r) {
    uint32_t* p = z.p[r];
    const size_t words = z.words[r];
    // 16-byte stores between the ragged ends
    const size_t head = min(words, (size_t)((4u - (((uintptr_t)p >> 2) & 3u)) & 3u)), quads = (words - head) / 4;
    uint4* q = reinterpret_cast<uint4*>(p + head);
    for (size_t i = i0; i < quads; i += step) q[i] = make_uint4(0u, 0u, 0u, 0u);
    const size_t ragged = words - 4 * quads;
    if (i0 < ragged) p[i0 < head ? i0 : i0 + 4 * quads] = 0u;
  }
}

// ---------------------------------------------------------------- hit stream
__global__ void __launch_bounds__(kTraceThreads) k_hit_stream(HitStreamParams p) {
  const Smem sm = thread_smem<kStackDepth>();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.R) return;
  const float3 o = make_float3(p.ray_o[3 * i], p.ray_o[3 * i + 1], p.ray_o[3 * i + 2]);
  const float3 d = make_float3(p.ray_d[3 * i], p.ray_d[3 * i + 1], p.ray_d[3 * i + 2]);
  const RayW r = make_ray(o, d);
  unsigned long long key_min = 0ull;
  int count = 0;
  for (int chunk = 0; chunk < kMaxChunks; ++chunk) {
    float t_drop;
    Counters cnt;
    query<kStackDepth>(p.bvh, r, key_min, kFar, sm.keys, sm.stride, sm.st, t_drop, p.status, cnt, 0);
    int consumed = 0;
    unsigned long long last = 0;
#pragma unroll
    for (int j = 0; j < kChunk; ++j) {
      const unsigned long long key = sm.keys[j * sm.stride];
      if (key == kEmptyKey || key_t(key) >= t_drop) break;
      if (count < p.max_hits) {
        p.ids[(size_t)i * p.max_hits + count] = key_prim(key);
        p.ts[(size_t)i * p.max_hits + count] = key_t(key);
      }
      ++count;
      ++consumed;
      last = key;
    }
    if (t_drop == INFINITY && consumed < kChunk) break;
    if (consumed == 0) {
      atomicOr(p.status, kStatusStack);
      break;
    }
    key_min = last + 1ull;
  }
  p.counts[i] = count;
}

}  // namespace

bool variant_may_go_by_lanes(const TraceParams& p) {
  if (p.variant == 0) return false;
  const long long samples = p.variant == 3 ? std::max(p.samples, 1) : 1;
  return 32ll * p.ntiles > (1 << 17) + 10ll * p.bvh.P + 300000 * (samples - 1);
}

cudaError_t launch_zero(const ZeroList& z, cudaStream_t s) {
  size_t most = 0;
  for (int i = 0; i < z.n; ++i) most = std::max(most, (size_t)z.words[i]);
  if (most == 0) return cudaSuccess;
  const int grid = (int)std::min<size_t>((most / 4 + 255) / 256 + 1, 148 * 8);
  k_zero<<<grid, 256, 0, s>>>(z);
  return cudaGetLastError();
}

size_t trace_smem_bytes(int cfg) {
  switch (cfg) {
    case kCfgPackets16: return smem_bytes_for<kCfgPackets16>();
    case kCfgPackets32: return smem_bytes_for<kCfgPackets32>();
    case kCfgLanes24: return smem_bytes_for<kCfgLanes24>();
    default: return smem_bytes_for<kCfgLanes32>();
  }
}

namespace {
template <int CFG>
const void* fwd_fn() { return (const void*)k_forward<CFG, kShadeRef>; }
template <int CFG>
const void* bwd_fn() { return (const void*)k_backward<CFG, kShadeRef>; }
const void* collect_fn(int cfg) {
  switch (cfg) {
    case kCfgPackets16: return (const void*)k_collect<kCfgPackets16>;
    case kCfgPackets32: return (const void*)k_collect<kCfgPackets32>;
    case kCfgLanes24: return (const void*)k_collect<kCfgLanes24>;
    default: return (const void*)k_collect<kCfgLanes32>;
  }
}
const void* kernel_for(int which, int cfg) {
  switch (cfg) {
    case kCfgPackets16: return which == 0 ? fwd_fn<kCfgPackets16>() : bwd_fn<kCfgPackets16>();
    case kCfgPackets32: return which == 0 ? fwd_fn<kCfgPackets32>() : bwd_fn<kCfgPackets32>();
    case kCfgLanes24: return which == 0 ? fwd_fn<kCfgLanes24>() : bwd_fn<kCfgLanes24>();
    default: return which == 0 ? fwd_fn<kCfgLanes32>() : bwd_fn<kCfgLanes32>();
  }
}
}  // namespace

int trace_blocks_per_sm(int which, int cfg) {
  int n = 0;
  const void* fn = which == 2 ? (const void*)k_variant<false> : (which == 3 ? collect_fn(cfg) : kernel_for(which, cfg));
  const size_t smem = which == 2 ? pair_smem<kChunk>() : trace_smem_bytes(cfg);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kTraceThreads, smem) != cudaSuccess) n = 1;
  return n > 0 ? n : 1;
}

// Opts the kernels of a traversal configuration and shading mode in to their
// dynamic shared memory where it passes the default 48 KB: the buffers of
// 32-hit packets, and the exact-adjoint forward's accumulators
// (kExactSmemBytes after the traversal's). Only the configuration a handle
// uses: an attribute call loads its kernel.
template <int CFG, int MODE>
cudaError_t opt_in_kernels() {
  cudaError_t e = cudaSuccess;
  auto opt_in = [&](const void* fn, size_t bytes) {
    if (e == cudaSuccess && bytes > 48 * 1024)
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  const size_t extra = MODE == kShadeExact ? kExactSmemBytes : 0;
  opt_in((const void*)k_collect<CFG>, smem_bytes_for<CFG>());
  opt_in((const void*)k_forward<CFG, MODE>, smem_bytes_for<CFG>() + extra);
  opt_in((const void*)k_backward<CFG, MODE>, smem_bytes_for<CFG>());
  if constexpr (TraversalCfg<CFG>::packets)
    opt_in((const void*)k_adjoint<TraversalCfg<CFG>::K, MODE>, adjoint_smem<TraversalCfg<CFG>::K, MODE>());
  return e;
}

template <int MODE>
cudaError_t trace_init_t(int cfg) {
  switch (cfg) {
    case kCfgPackets16: return opt_in_kernels<kCfgPackets16, MODE>();
    case kCfgPackets32: return opt_in_kernels<kCfgPackets32, MODE>();
    case kCfgLanes24: return opt_in_kernels<kCfgLanes24, MODE>();
    default: return opt_in_kernels<kCfgLanes32, MODE>();
  }
}

cudaError_t trace_init(int cfg, int mode) {
  switch (mode) {
    case kShadeExact: return trace_init_t<kShadeExact>(cfg);
    case kShadeRefArith: return trace_init_t<kShadeRefArith>(cfg);
    default: return trace_init_t<kShadeRef>(cfg);
  }
}

// The replay-only builds' shared memory (keys and counters, and the exact
// forward's accumulators) stays within the default.
static_assert(smem_bytes_for<kCfgPackets32, true>() + kExactSmemBytes <= 48 * 1024, "replay builds need no opt-in");

// Grid of a replay-only build: the traversing build's grid (SMs x its blocks
// per SM) at the replay build's blocks per SM.
inline int replay_grid(int grid) { return grid / kMinBlocks * kReplayBlocks; }
inline int adjoint_grid(int grid) { return grid / kMinBlocks * kAdjointBlocks; }

// Parts a tile is taken in (log2): an image with fewer tiles than the grid has
// warps leaves warps without work, and a warp with a few of a tile's rays walks
// less for a narrower frustum. Whole tiles / parts: 3M triangles, 64 x 64
// 7.8 / 1.2 ms; 616k, 31 x 38 3.4 / 0.28 ms; training step of 1M, 128 x 160
// 3.9 / 1.9 ms; parts of at least 8 rays 2.4, 1.1 and 1.9 ms.
inline TraceParams with_parts(const TraceParams& p, int grid) {
  TraceParams q = p;
  const long long warps = (long long)grid * (kTraceThreads / 32);
  while (q.parts_log < kMaxPartsLog && ((long long)q.ntiles << (q.parts_log + 1)) <= warps) ++q.parts_log;
  return q;
}

template <int MODE>
cudaError_t launch_forward_t(const TraceParams& in, int grid, cudaStream_t s) {
  const TraceParams p = with_parts(in, grid);
  const size_t extra = MODE == kShadeExact ? kExactSmemBytes : 0;
  if (p.fwd_pair) {
    if (p.cfg == kCfgPackets16)
      k_forward<kCfgPackets16, MODE, true><<<replay_grid(grid), kTraceThreads, smem_bytes_for<kCfgPackets16, true>() + extra, s>>>(p);
    else
      k_forward<kCfgPackets32, MODE, true><<<replay_grid(grid), kTraceThreads, smem_bytes_for<kCfgPackets32, true>() + extra, s>>>(p);
  }
  switch (p.cfg) {
    case kCfgPackets16: k_forward<kCfgPackets16, MODE><<<grid, kTraceThreads, smem_bytes_for<kCfgPackets16>() + extra, s>>>(p); break;
    case kCfgPackets32: k_forward<kCfgPackets32, MODE><<<grid, kTraceThreads, smem_bytes_for<kCfgPackets32>() + extra, s>>>(p); break;
    case kCfgLanes24: k_forward<kCfgLanes24, MODE><<<grid, kTraceThreads, smem_bytes_for<kCfgLanes24>() + extra, s>>>(p); break;
    default: k_forward<kCfgLanes32, MODE><<<grid, kTraceThreads, smem_bytes_for<kCfgLanes32>() + extra, s>>>(p); break;
  }
  return cudaGetLastError();
}

template <int MODE>
cudaError_t launch_backward_t(const TraceParams& in, int grid, cudaStream_t s) {
  const TraceParams p = with_parts(in, grid);
  if (p.bwd_pair) {
    if (p.cfg == kCfgPackets16)
      k_adjoint<16, MODE><<<adjoint_grid(grid), kTraceThreads, adjoint_smem<16, MODE>(), s>>>(p);
    else
      k_adjoint<32, MODE><<<adjoint_grid(grid), kTraceThreads, adjoint_smem<32, MODE>(), s>>>(p);
  }
  switch (p.cfg) {
    case kCfgPackets16: k_backward<kCfgPackets16, MODE><<<grid, kTraceThreads, smem_bytes_for<kCfgPackets16>(), s>>>(p); break;
    case kCfgPackets32: k_backward<kCfgPackets32, MODE><<<grid, kTraceThreads, smem_bytes_for<kCfgPackets32>(), s>>>(p); break;
    case kCfgLanes24: k_backward<kCfgLanes24, MODE><<<grid, kTraceThreads, smem_bytes_for<kCfgLanes24>(), s>>>(p); break;
    default: k_backward<kCfgLanes32, MODE><<<grid, kTraceThreads, smem_bytes_for<kCfgLanes32>(), s>>>(p); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_collect(const TraceParams& in, int grid, cudaStream_t s) {
  const TraceParams p = with_parts(in, grid);
  switch (p.cfg) {
    case kCfgPackets16: k_collect<kCfgPackets16><<<grid, kTraceThreads, smem_bytes_for<kCfgPackets16>(), s>>>(p); break;
    case kCfgPackets32: k_collect<kCfgPackets32><<<grid, kTraceThreads, smem_bytes_for<kCfgPackets32>(), s>>>(p); break;
    case kCfgLanes24: k_collect<kCfgLanes24><<<grid, kTraceThreads, smem_bytes_for<kCfgLanes24>(), s>>>(p); break;
    default: k_collect<kCfgLanes32><<<grid, kTraceThreads, smem_bytes_for<kCfgLanes32>(), s>>>(p); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_forward(const TraceParams& p, int grid, cudaStream_t s) {
  if (p.variant != 0) {
    if (p.fwd_pair) k_variant<true><<<grid, kTraceThreads, (size_t)kTraceThreads * (kVariantStack + kChunk) * 8, s>>>(p);
    k_variant<false><<<grid, kTraceThreads, pair_smem<kChunk>(), s>>>(p);
    return cudaGetLastError();
  }
  switch (p.mode) {
    case kShadeExact: return launch_forward_t<kShadeExact>(p, grid, s);
    case kShadeRefArith: return launch_forward_t<kShadeRefArith>(p, grid, s);
    default: return launch_forward_t<kShadeRef>(p, grid, s);
  }
}

cudaError_t launch_backward(const TraceParams& p, int grid, cudaStream_t s) {
  switch (p.mode) {
    case kShadeExact: return launch_backward_t<kShadeExact>(p, grid, s);
    case kShadeRefArith: return launch_backward_t<kShadeRefArith>(p, grid, s);
    default: return launch_backward_t<kShadeRef>(p, grid, s);
  }
}

int sec_blocks_per_sm(int which) {
  int n = 0;
  const void* fn = which == 0 ? (const void*)k_sec_trace
                              : (which == 1 ? (const void*)k_sec_backward
                                            : (which == 2 ? (const void*)k_sec_primary : (const void*)k_sec_collect));
  const size_t smem = which == 2 ? smem_bytes_for<kCfgPackets16>()
                                 : (which == 0 ? sec_trace_smem()
                                               : (which == 3 ? sec_collect_smem() : smem_bytes_for<kCfgLanes32>()));
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kTraceThreads, smem) != cudaSuccess) n = 1;
  return n > 0 ? n : 1;
}

cudaError_t launch_sec_trace(const TraceParams& p, int grid, cudaStream_t s) {
  k_sec_trace<<<grid, kTraceThreads, sec_trace_smem(), s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_sec_collect(const TraceParams& p, int grid, cudaStream_t s) {
  k_sec_collect<<<grid, kTraceThreads, sec_collect_smem(), s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_sec_primary(const TraceParams& in, int grid, cudaStream_t s) {
  const TraceParams p = with_parts(in, grid);
  k_sec_primary<<<grid, kTraceThreads, smem_bytes_for<kCfgPackets16>(), s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_sec_resolve(const TraceParams& p, cudaStream_t s) {
  const long long cap = p.sec.level == 0 ? (long long)p.views[0].H * p.views[0].W : p.sec.cap[p.sec.level];
  const int grid = (int)std::min<long long>((cap + 255) / 256, 4096);
  if (grid == 0) return cudaSuccess;
  k_sec_resolve<<<grid, 256, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_sec_sort_keys(const TraceParams& p, uint32_t* keys, uint32_t* vals, cudaStream_t s) {
  const int cap = p.sec.cap[p.sec.level];
  const int grid = std::min((cap + 255) / 256, 148 * 8);
  if (grid == 0) return cudaSuccess;
  k_sec_sort_keys<<<grid, 256, 0, s>>>(p, keys, vals);
  return cudaGetLastError();
}

cudaError_t launch_sec_backward(const TraceParams& p, int grid, cudaStream_t s) {
  k_sec_backward<<<grid, kTraceThreads, smem_bytes_for<kCfgLanes32>(), s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_hit_stream(const HitStreamParams& p, cudaStream_t s) {
  const int grid = (p.R + kTraceThreads - 1) / kTraceThreads;
  if (grid == 0) return cudaSuccess;
  k_hit_stream<<<grid, kTraceThreads, smem_bytes_for<kCfgLanes32>(), s>>>(p);
  return cudaGetLastError();
}

}  // namespace tt
