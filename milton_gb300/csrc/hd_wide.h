// hd_wide.h -- 8-wide bounding-volume hierarchy traversal of the render and ray-query kernels.
//
// The hierarchy is built on the device when a scene is created (bvh.cu) and answers the same
// queries as the kd-tree (hd_trace.h) with the same triangle test: a closest hit is the smallest
// accepted t over the scene's triangles, whatever visits them, so both give the same primitive, t
// and barycentrics, bit for bit.  Where the kd-tree's answer depends on more than that -- near ties, rays in
// its split planes, triangles outside its root box -- it is asked (kWideTie, wide_beside, kWideOutside).  Not
// covered is a triangle edge-on to the ray, whose hit is rounding (one of 11.2 M rays aimed at such places).
//
// Why a wide hierarchy: on the mid scene (1 M triangles) the kd-tree takes 50 dependent node steps
// and 33 triangle tests per ray.  The node here holds eight child boxes as 16-bit floats around the
// node's centre in 128 bytes, one cache line (8-bit grid coordinates in 96 bytes, as the paper has
// them: more conversions per box, and flat boxes grow by a grid step, so that a ray met the wall it
// starts on and the light it ends at; 24-triangle room: 4.5 -> 2.7 triangles per occlusion query, frame
// 0.94 -> 0.87 ms; mid frame 111.4 -> 105.5 ms); the masks, the child order and the single stack entry per
// level are those of Ylitie, Karras and Laine, "Efficient Incoherent Ray Traversal on GPUs Through
// Compressed Wide BVHs", HPG 2017.
//
// Node (32 words, four 256-bit loads):
//   0..2   centre of the node's box, relative to the scene's centre
//   3      index of the first inner child (the inner children of a node are consecutive, in slot
//          order)
//   4      index of the node's first triangle record (the leaf children's triangles are
//          consecutive, in slot order)
//   5      mask of the slots that hold inner nodes
//   6      triangles of the leaf children: bits 3 s .. 3 s + 2 hold slot s's count in unary
//   7      unused
//   8 + 3 s + k   slot s's planes along axis k, relative to the centre: the upper halves of two floats, low
//          plane in bits 0..15, high plane in bits 16..31
// Triangle record: 3 x float4 as a kd leaf's (v0 + primitive id, v1 + flags, v2); flags: 1 = culled, kWideOutside.
//
// A slot's number says where its child lies: bit k set = the upper side along axis k.  A ray visits
// the children it meets in the order of slot XOR octant (its negative directions), which is front to
// back along the octant, so the stack holds one entry (the siblings still to visit) per level.
#pragma once

#include "hd_trace.h"

namespace mgpu {

constexpr int kWideWords = 32;       // 32-bit words per node
constexpr int kWideLeafTris = 3;     // triangles per leaf child
constexpr int kWideMaxDepth = 30;    // levels of node below the root that the traversal stack holds
constexpr uint32_t kWideOutside = 2u;  // flag of a triangle record: it reaches out of the kd-tree's root box (bvh.cu)
constexpr uint32_t kWideRootBits = 0x101u;  // pending slots and inner mask of the root's pseudo parent
// Threads per block: one block per SM at 64 registers a thread.  The rays of one SM are then
// neighbours in the (sorted) queue and share its L1: mid frame, traversal 117 ms in blocks of 128,
// 114 / 108 / 102 ms in blocks of 256 / 512 / 1024.
constexpr int kWideBlock = 1024;
// Rays that a block takes at a time; its warps take them 32 by 32 as they finish (against fixed grid-stride
// rounds the mid frame's traversal went from 102 to 96 ms; now, whole frame: 103.7, 104.0, 104.3 ms at 128, 256,
// 512, and 1 M ray queries 0.215, 0.211, 0.229).
constexpr uint32_t kWideChunk = 256u;
// Triangle tests waiting after a node step that are worth a round of their own: a full queue (32) keeps
// every lane busy but lets the rays go on with a stale closest t (mid closest hits: 49.9 / 46.9 /
// 46.5 ms at 32 / 16 / 8; now flat from 4 to 16, and 2 % slower at 24 in the textured scene).
constexpr uint32_t kWideFlush = 8u;

// Box tests are conservative.  The planes are rounded outward when they are stored.  What rounds relative
// to M, the largest coordinate of the scene box or the ray's origin from the scene's centre -- the
// plane distances (6 x 2^-24 M) and the triangle test's sheared coordinates (6 x 2^-24 of at most
// 2 M) -- is covered by moving every plane outward by 1.5 x 2^-20 M, folded into the ray's constants.
constexpr float kWideEps = 1.5f / 1048576.0f;

// A direction component below 2^-40 of the ray's largest is taken as that in the box tests: the reciprocal of a
// smaller one, multiplied by the origin, overflows, and boxes that the ray passes were missed (components
// of 1e-38; and where the reciprocal itself is infinite every box was met: 200,000 rays 0.3 -> 611 ms).  It is
// still conservative: through the scene such a ray moves at most 2^-38 M along that axis, and the planes
// are 2^-19 M farther out.  (All of it in reciprocals: least is that of the largest component.)
constexpr float kWideMost = 1099511627776.0f;
// ... and from this part of it on the ray is one with a zero component to the kd-tree's rounding (wide_beside)
constexpr float kWideZero = 1.0e30f;
// What the box tests multiply and add lies between 2^-20 and 2^41 times M x least; where that is beyond these,
// products overflow or lose bits below the normal numbers, and the kd-tree answers the ray.  (A scene without
// the hierarchy has an infinite extent, which takes its rays there where it shares a wave with scenes that
// have one.)
constexpr float kWideScaleMin = 1.0e-25f, kWideScaleMax = 1.0e25f;

#if defined(__CUDACC__)

// one half of w (which: the permute's selector) as the upper half of a float
__device__ __forceinline__ float wide_half(uint32_t w, uint32_t which) {
  return __uint_as_float(__byte_perm(w, 0u, which));
}

// Tables in shared memory, per block: first[oct][m] = the slot to visit first among those in m for a ray
// of octant oct (slot XOR oct least), spread[m] = bit s of m moved to bits 3 s .. 3 s + 2.
struct WideTables {
  uint32_t spread[256];
  uint8_t first[8][256];
};

__device__ __forceinline__ void wide_tables(WideTables &t) {
  for (uint32_t k = threadIdx.x; k < 2048u; k += blockDim.x) {
    const uint32_t oct = k >> 8, m = k & 255u;
    uint32_t best = 8u;
    for (uint32_t s = 0; s < 8u; ++s)
      if ((m >> s) & 1u) best = min(best, s ^ oct);
    t.first[oct][m] = (uint8_t)(best ^ oct);
    if (oct == 0u) {
      uint32_t w = 0u;
      for (uint32_t s = 0; s < 8u; ++s) w |= ((m >> s) & 1u) ? 7u << (3u * s) : 0u;
      t.spread[m] = w;
    }
  }
}

struct WideRow {
  uint32_t w[8];
};

__device__ __forceinline__ WideRow wide_load(const uint32_t *p) {
  WideRow r;
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7])
      : "l"(p));
  return r;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

struct WideGroup {
  uint32_t base;  // nodes: first inner child of the parent; triangles: the node's first record
  uint32_t bits;  // nodes: pending slots (bits 0..7) | inner mask << 8; triangles: pending
};

// What a lane keeps in registers through the node steps.  The triangle tests' ray constants are in
// shared memory (WideShared).
struct WideRay {
  V3 inv;
  V3 kn, kf;            // -origin x inv moved outward: added to p x inv, near and far plane distances
  float tmin;
  float best;           // t up to which boxes are visited: the ray's tmax, then just past the closest hit
  const uint8_t *first; // the table row of the ray's octant
};

// Tests the eight children of node idx against (tmin, best]: pending inner children and triangles.
__device__ __forceinline__ void wide_node(const uint32_t *__restrict__ nodes, uint32_t idx, const WideRay &w,
                                          float tmin, const WideTables &tab, WideGroup &ng, WideGroup &tg, uint32_t &tvalid) {
  const uint32_t *q = nodes + (size_t)idx * kWideWords;
  const WideRow a = wide_load(q);
  uint32_t box[24];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const WideRow r = wide_load(q + 8 + 8 * k);
#pragma unroll
    for (int i = 0; i < 8; ++i) box[8 * k + i] = r.w[i];
  }
  const float px = __uint_as_float(a.w[0]), py = __uint_as_float(a.w[1]), pz = __uint_as_float(a.w[2]);
  const float nx = fmaf(px, w.inv.x, w.kn.x), ny = fmaf(py, w.inv.y, w.kn.y), nz = fmaf(pz, w.inv.z, w.kn.z);
  const float fx = fmaf(px, w.inv.x, w.kf.x), fy = fmaf(py, w.inv.y, w.kf.y), fz = fmaf(pz, w.inv.z, w.kf.z);
  // permutes that leave the near and the far half of a pair of planes on top of zeros
  const uint32_t sx = w.inv.x < 0.0f ? 0x3244u : 0x1044u, sy = w.inv.y < 0.0f ? 0x3244u : 0x1044u,
                 sz = w.inv.z < 0.0f ? 0x3244u : 0x1044u;
  const uint32_t ux = sx ^ 0x2200u, uy = sy ^ 0x2200u, uz = sz ^ 0x2200u;
  uint32_t miss = 0u;
#pragma unroll
  for (int i = 7; i >= 0; --i) {
    const uint32_t bx = box[3 * i], by = box[3 * i + 1], bz = box[3 * i + 2];
    const float t0 = max3(fmaf(wide_half(bx, sx), w.inv.x, nx), fmaf(wide_half(by, sy), w.inv.y, ny),
                          fmaf(wide_half(bz, sz), w.inv.z, nz));
    const float t1 = min3(fmaf(wide_half(bx, ux), w.inv.x, fx), fmaf(wide_half(by, uy), w.inv.y, fy),
                          fmaf(wide_half(bz, uz), w.inv.z, fz));
    // a miss if t1 < t0, best < t0 or t1 < tmin: the signs of the differences (NaN from two infinities has a
    // plus: a hit), shifted in.  Additions instead of a maximum, a minimum and comparisons, because
    // those share a pipe with the permutes (terrain 19.9 -> 19.6 ms a frame).
    miss = __funnelshift_l(__float_as_uint(t1 - t0) | __float_as_uint(w.best - t0) | __float_as_uint(t1 - tmin), miss, 1);
  }
  const uint32_t hits = ~miss & 0xFFu, imask = a.w[5];
  ng.base = a.w[3];
  ng.bits = (hits & imask) | (imask << 8);
  tg.base = a.w[4];
  tvalid = a.w[6];
  tg.bits = tab.spread[hits & ~imask] & tvalid;
}

// Per-warp shared memory: every lane's ray for the triangle tests, its best hit so far, and the queue
// of (lane, triangle) tests waiting for a full round.
struct WideShared {
  float4 a[32], b[32];       // (o, tmin), (sx, sy, sz, tmax)
  unsigned long long key[32];  // closest hit: ordered t << 32 | triangle record; ~0 record: none
  uint32_t k[32];            // axis permutation
  uint32_t rec[64];          // queue (ring of 64): triangle record
  uint8_t own[64];           // ... and the lane it is for
  int32_t sphere[32];        // analytic sphere hit before the traversal, -1: none
  const F4 *tris[32];        // the lanes' scenes' triangle records (waves of several scenes)
  uint8_t zero[32];          // axes of zero direction components
  uint32_t tie[32];          // ordered t of the nearest hit that the kd-tree has to decide (kWideTie, wide_beside);
                             // any hit: the record of a hit that it may have to (kWideOutside), with
                             // the upper bit set if it has to (wide_beside); ~0: none
};

__device__ __forceinline__ uint32_t wide_order(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float wide_unorder(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Two hits of a ray closer than this (relative) are decided by the kd-tree: which of two equal or
// nearly equal t a ray reports depends on the order of the tests (leaf order, and the early exit
// once the best hit lies inside the current cell, widened by 2^-18), so such a ray is traced again
// there.  It is a ray through an exact edge, or a surface laid on another: one in some 10^8 on scenes
// without coincident surfaces.
constexpr float kWideTie = 1.0f / 131072.0f;

// So is a ray with a zero direction component, or as good as zero, if its hit touches the plane through its
// origin normal to that axis from one side: if that is a split plane the ray sees only the cells on one side
// of it in the kd-tree, and the triangle may be listed on the other.  Split planes are triangle bounds and
// triangles are listed by their bounds, so a triangle with vertices on both sides is in both cells.
// axes: the mask of those components; within a t of 1e-29 of the plane counts, as the kd-tree takes
// 1e30 for the reciprocal of a zero.
// (Tracing all of them in the kd-tree, lane by lane: 1 M vertical rays from random points among 300 k triangles
// 673 us, now 251; random rays of which 5 % have a zero component 358 us, now 178.)
// Not inlined, and reads the triangle again, so that the tests' code keeps neither the mask nor the vertices.
inline __device__ __noinline__ bool wide_beside(uint32_t axes, V3 o, float t, const F4 *tri) {
  const F4 a = load_f4(tri, 0), b = load_f4(tri, 1), c = load_f4(tri, 2);
  const float e = 1.0e-29f * fabsf(t);
  const V3 lo = v3(fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z)));
  const V3 hi = v3(fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z)));
  return ((axes & 1u) && (o.x - e <= lo.x || o.x + e >= hi.x)) || ((axes & 2u) && (o.y - e <= lo.y || o.y + e >= hi.y)) ||
         ((axes & 4u) && (o.z - e <= lo.z || o.z + e >= hi.z));
}

// Whether the kd-tree finds the hit of a ray on a triangle that reaches out of its root box (kWideOutside): without
// traversing it, so false where that is not certain.  In the root box it does, as it finds any triangle
// there.  Beyond, it does if a leaf that the ray passes lists the triangle: the leaf where the ray leaves
// the box (enters it, for a hit before) does if along every axis the triangle's bounds hold that point
// or, along the one of the face, reach that face, since triangles are listed by their bounds on either
// side of split planes.  No nearer hit ends the kd-tree's search before that leaf: one farther than this hit
// by less than its cells are widened is a near tie.
// (A unit floor under 20,000 triangles, 1 M rays straight down, all of whose hits on it went to the kd-tree:
// closest 1,065 -> 398 us, any 900 -> 86; 256 x 256 x 4 frame 548 -> 304.)
// h: that hit
inline __device__ bool wide_listed(const SceneView &s, const Ray &r, const F4 *tri, Hit &h) {
  const F4 a = load_f4(tri, 0), b = load_f4(tri, 1), c = load_f4(tri, 2);
  float t0, t1;
  const bool hit = intersect_tri(precompute(r), v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z),
                                 (f_bits(b.w) & 1u) != 0u, r.tmin, r.tmax, h.t, h.b1, h.b2);
  const float t = h.t;
  h.prim = (int32_t)f_bits(a.w);
  if (!hit || !clip_root(s, r, v3(1.0f / r.d.x, 1.0f / r.d.y, 1.0f / r.d.z), t0, t1) || !(r.tmin >= 0.0f))
    return false;
  if (t >= t0 && t <= t1) return true;
  const bool exit = t > t1;
  const float at = exit ? t1 : t0;
  const float o[3] = {r.o.x, r.o.y, r.o.z}, d[3] = {r.d.x, r.d.y, r.d.z};
  const float lo[3] = {fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z))};
  const float hi[3] = {fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z))};
  bool all = true;
  for (int k = 0; k < 3; ++k) {
    const float step = at * d[k], p = o[k] + step, m = (fabsf(o[k]) + fabsf(step)) * (1.0f / 65536.0f);
    const bool upper = (d[k] > 0.0f) == exit;  // the face of axis k that the ray leaves (enters) through
    const bool face = ((upper ? s.bmax[k] : s.bmin[k]) - o[k]) * (1.0f / d[k]) == at &&
                      (upper ? hi[k] >= s.bmax[k] : lo[k] <= s.bmin[k]);
    all = all && (face || (p - m >= lo[k] && p + m <= hi[k]));
  }
  return all;
}

// The kd-tree's answer for one ray: closest hit, or any (h.prim >= 0).  seq: a leaf's triangles one after
// another, each against the t before it (ray queries, scenes with analytic spheres); otherwise the
// smallest (t, leaf order) among those accepted against the t before the leaf.  The two differ where
// triangles coincide, so the rule belongs to the scene, not to the launch.
template <bool ANY, bool SPH, bool COUNT>
__device__ __forceinline__ void kd_trace(const SceneView &s, const Ray &r, bool seq, Hit &h, TraceCounts *cnt) {
  TravState st;
  TravEntry stack[kMaxStack];
  if (trav_init<SPH>(s, r, nullptr, 0, st, ANY)) {
    bool done = false;
    while (!done) {
      uint32_t w0, w1;
      float tmax;
      trav_descend<COUNT>(s, st, stack, nullptr, 0, cnt, w0, w1, tmax);
      const float best0 = st.best;
      bool took = false;
      for (uint32_t i = 0; i < (w0 >> 2) && !(ANY && took); ++i) {
        if (COUNT) cnt->tris++;
        const int64_t q = 3 * ((int64_t)w1 + i);
        const F4 a = load_f4(s.ltris, q), b = load_f4(s.ltris, q + 1), c = load_f4(s.ltris, q + 2);
        float t, b1, b2;
        if (intersect_tri(st.pre, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), (f_bits(b.w) & 1u) != 0u,
                          st.ray_tmin, seq ? st.best : best0, t, b1, b2) &&
            (seq || !took || t < st.best)) {
          took = true;
          st.best = t; st.best_prim = (int32_t)f_bits(a.w); st.bb1 = b1; st.bb2 = b2;
        }
      }
      done = (ANY && took) || trav_after_leaf<ANY>(st, stack, tmax);
    }
  }
  h.t = st.best;
  h.prim = st.best_prim;
  h.b1 = st.bb1;
  h.b2 = st.bb2;
}

// outside: the record of the ray's hit, which holds without the kd-tree if that finds it (the upper bit set: none)
template <bool ANY, bool SPH, bool QUERY, bool OUT>
__device__ __noinline__ void kd_ray(const SceneView &s, const Ray &r, Hit &h, uint32_t outside) {
  if (OUT && outside < 0x80000000u && wide_listed(s, r, s.wtris + 3 * (int64_t)outside, h)) return;
  kd_trace<ANY, SPH, false>(s, r, QUERY || (SPH && s.nsphere > 0), h, nullptr);
}

// Rays 0 .. n - 1 through the kd-tree, one per lane, grid-stride: scenes without the hierarchy.
template <bool ANY, bool COUNT, bool SPH, class View, class Load, class Store>
__device__ __forceinline__ void kd_grid(View view, uint32_t n, Load load, Store store, TraceCounts *cnt,
                                        uint32_t &rays_done) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const SceneView &s = view(i);
    Ray r;
    load(i, r);
    ++rays_done;
    Hit h;
    kd_trace<ANY, SPH, COUNT>(s, r, SPH && s.nsphere > 0, h, cnt);
    store(i, h.prim >= 0, h);
  }
}

// The traversal of one warp.  Every lane steps through the nodes of its own ray; the triangles it meets go
// into the warp's queue, and the warp tests them together, each lane one (ray, triangle) pair
// whoever's it is, with the owner's constants from shared memory.  A node step finds a triangle for
// about half the lanes and up to six for one, so testing them lane by lane ran the test with a
// sixth of the lanes (mid frame, closest hits: 78 -> 59 ms).
// What bounds it (ncu, mid scene, second bounce): instruction issue (85 % of the slots), and the pipe that
// takes the byte permutes, minima and comparisons (76 %), with 17 of 32 lanes active; L1 hit rate 81 %,
// L2 below 8 % and DRAM below 3 % of their peaks.  The kd-tree's kernels were bound by the
// latency of 50 dependent node loads per ray.  Mid frame (163 M closest hits, 226 M occlusion
// queries): kd-tree 187.7 ms of traversal, nodes of 80 bytes with per-node slack and child order by mask
// permutation 95.0, nodes of 96 bytes on an 8-bit grid 83.7, as it is now 77.9.
//   ANY     occlusion: the first hit ends the ray; otherwise the closest
//   QUERY   a ray query.  Its near ties are decided in leaf order (seq of kd_trace) whatever the scene, otherwise
//           the scene's rule decides.  Its rays with zero direction components go through the hierarchy
//           (wide_beside): queries along an axis are whole launches of such rays.  A path meets one by
//           chance, the kd-tree answers it, and the render kernels, whose rays all start at t = 0, are spared
//           code that makes them spill.
//   SINGLE  every ray is in the scene view(0), which the kernel passes from its parameter space
//   OUT     records may be flagged kWideOutside.  Occlusion queries without that code are 4 % faster
//           (777,600 rays from terrain 56.8 -> 54.2 us); the render kernels measure the same either way.
// All 32 lanes call round(), the other members are per lane or say so.
template <bool ANY, bool COUNT, bool SPH, bool SINGLE, bool QUERY, bool OUT, class View, class Load, class Store>
struct WideWarp {
  static constexpr unsigned kFull = 0xFFFFFFFFu;
  View view;
  Load load;
  Store store;
  WideShared &sh;
  const WideTables &tab;
  TraceCounts *cnt;
  const uint32_t lane;
  uint2 *stack;
  WideRay w{};
  WideGroup ng{0u, 0u}, tg{0u, 0u};
  uint32_t tvalid = 0u;
  int sp = 0;
  const uint32_t *nodes = nullptr;
  bool active = false;         // the lane's ray has nodes to visit
  bool found = false;          // ANY: it is occluded
  bool kd = false;             // the kd-tree answers it
  uint32_t qh = 0u, qn = 0u;   // queue head and length (uniform over the warp)

  // takes ray i
  __device__ __forceinline__ void start(uint32_t i) {
    const SceneView &s = SINGLE ? view(0u) : view(i);
    if (!SINGLE) nodes = s.wnodes;
    Ray r;
    load(i, r);
    found = false;
    float best = r.tmax;
    int32_t sphere = -1;
    if (SPH) {
      if (s.nsphere > 0) {
        TravState ts;
        ts.best = r.tmax;
        ts.best_prim = -1;
        spheres_hit(s, r, ts, ANY);
        best = ts.best;
        sphere = ts.best_prim;
      }
      sh.sphere[lane] = sphere;
    }
    active = s.ntri > 0 && !(ANY && sphere >= 0);
    const V3 o = r.o - v3(s.wcentre[0], s.wcentre[1], s.wcentre[2]);
    float m = fmaxf(fmaxf(s.wextent, fabsf(o.x)), fmaxf(fabsf(o.y), fabsf(o.z)));
    const V3 inv = v3(1.0f / r.d.x, 1.0f / r.d.y, 1.0f / r.d.z);
    const V3 ai = v3(fabsf(inv.x), fabsf(inv.y), fabsf(inv.z));
    const float least = fminf(ai.x, fminf(ai.y, ai.z)), most = fmaxf(ai.x, fmaxf(ai.y, ai.z));
    const float zero = least * kWideZero, scale = m * least;
    kd = active && ((!QUERY && most >= zero) || !(scale >= kWideScaleMin && scale <= kWideScaleMax));
    active = active && !kd;
    if (active) {
      float t0, t1;
      active = clip_root(s, r, inv, t0, t1) && fmaxf(t0, r.tmin) <= fminf(t1, r.tmax);
    }
    if (active) {
      const RayPre pre = precompute(r);
      const float cap = least * kWideMost;
      w.inv = v3(copysignf(fminf(ai.x, cap), inv.x), copysignf(fminf(ai.y, cap), inv.y), copysignf(fminf(ai.z, cap), inv.z));
      m *= kWideEps;
      const V3 e = v3(m * fabsf(w.inv.x), m * fabsf(w.inv.y), m * fabsf(w.inv.z));
      const V3 k = v3(-(o.x * w.inv.x), -(o.y * w.inv.y), -(o.z * w.inv.z));
      w.kn = k - e;
      w.kf = k + e;
      w.tmin = r.tmin;
      w.best = best;
      w.first = tab.first[(w.inv.x < 0.0f ? 1u : 0u) | (w.inv.y < 0.0f ? 2u : 0u) | (w.inv.z < 0.0f ? 4u : 0u)];
      ng.base = 0u;
      ng.bits = kWideRootBits;
      sp = 0;
      sh.a[lane] = make_float4(r.o.x, r.o.y, r.o.z, r.tmin);
      sh.b[lane] = make_float4(pre.sx, pre.sy, pre.sz, r.tmax);
      if (!SINGLE) sh.tris[lane] = s.wtris;
      sh.k[lane] = (uint32_t)pre.kx | ((uint32_t)pre.ky << 2) | ((uint32_t)pre.kz << 4);
      if (QUERY)
        sh.zero[lane] = most < zero ? (uint8_t)0
                                    : (uint8_t)((ai.x >= zero ? 1u : 0u) | (ai.y >= zero ? 2u : 0u) | (ai.z >= zero ? 4u : 0u));
    }
    if (!ANY) sh.key[lane] = ((unsigned long long)wide_order(best) << 32) | (sphere >= 0 ? 0xFFFFFFFEu : 0xFFFFFFFFu);
    sh.tie[lane] = 0xFFFFFFFFu;
  }

  // one node of the lane's ray: its triangles into tg, its inner children pending
  __device__ __forceinline__ void step() {
    const uint32_t slot = w.first[ng.bits & 0xFFu];
    const uint32_t idx = ng.base + __popc((ng.bits >> 8) & ((1u << slot) - 1u));
    ng.bits &= ~(1u << slot);
    if (ng.bits & 0xFFu) stack[sp++] = make_uint2(ng.base, ng.bits);
    if (COUNT) cnt->nodes++;
    wide_node(SINGLE ? view(0u).wnodes : nodes, idx, w, QUERY ? w.tmin : 0.0f, tab, ng, tg, tvalid);
    if (!(ng.bits & 0xFFu)) {
      if (sp == 0) {
        active = false;
      } else {
        --sp;
        ng.base = stack[sp].x;
        ng.bits = stack[sp].y;
      }
    }
  }

  // the next triangle of the lane into the queue, after those of the lanes of m below it
  __device__ __forceinline__ void push(uint32_t m) {
    const uint32_t k = __ffs(tg.bits) - 1, e = (qh + qn + __popc(m & ((1u << lane) - 1u))) & 63u;
    tg.bits &= tg.bits - 1u;
    sh.rec[e] = tg.base + __popc(tvalid & ((1u << k) - 1u));
    sh.own[e] = (uint8_t)lane;
  }

  // tests the queue's first m <= 32 entries
  __device__ __forceinline__ void round(uint32_t m) {
    __syncwarp(kFull);
    uint32_t hit = 0u;
    if (lane < m) {
      const uint32_t e = (qh + lane) & 63u, rec = sh.rec[e], o = sh.own[e];
      const float4 ra = sh.a[o], rb = sh.b[o];
      const uint32_t kp = sh.k[o];
      RayPre p;
      p.o = v3(ra.x, ra.y, ra.z);
      p.sx = rb.x; p.sy = rb.y; p.sz = rb.z;
      p.kx = (int)(kp & 3u); p.ky = (int)((kp >> 2) & 3u); p.kz = (int)(kp >> 4);
      const F4 *lt = SINGLE ? view(0u).wtris : sh.tris[o];
      const int64_t q = 3 * (int64_t)rec;
      const F4 a = load_f4(lt, q), b = load_f4(lt, q + 1), c = load_f4(lt, q + 2);
      if (COUNT) cnt->tris++;
      float t, b1, b2;
      if (intersect_tri(p, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), (f_bits(b.w) & 1u) != 0u,
                        QUERY ? ra.w : 0.0f, rb.w, t, b1, b2)) {
        const uint32_t axes = QUERY ? sh.zero[o] : 0u;
        const bool beside = axes != 0u && wide_beside(axes, p.o, t, lt + q);
        if (ANY) {
          hit = 1u << o;
          if (beside || (OUT && (f_bits(b.w) & kWideOutside) != 0u)) sh.tie[o] = rec | (beside ? 0x80000000u : 0u);
        } else {
          if (beside) atomicMin(&sh.tie[o], wide_order(t));
          const unsigned long long old = atomicMin(&sh.key[o], ((unsigned long long)wide_order(t) << 32) | rec);
          const float told = wide_unorder((uint32_t)(old >> 32));
          if ((uint32_t)old != 0xFFFFFFFFu && fabsf(t - told) <= kWideTie * fabsf(t))
            atomicMin(&sh.tie[o], wide_order(fminf(t, told)));
        }
      }
    }
    qh = (qh + m) & 63u;
    qn -= m;
    if (ANY) {
      if ((__reduce_or_sync(kFull, hit) >> lane) & 1u) {
        found = true;
        active = false;
        tg.bits = 0u;
      }
    } else {
      __syncwarp(kFull);
      // hits within kWideTie behind the closest are looked at too: they make a near tie
      const float t = wide_unorder((uint32_t)(sh.key[lane] >> 32));
      w.best = fmaf(fabsf(t), 1.0625f * kWideTie, t);
    }
  }

  // the answer of ray i, all of whose triangles have been tested
  __device__ __forceinline__ void finish(uint32_t i) {
    const SceneView &s = SINGLE ? view(0u) : view(i);
    Hit h;
    h.prim = SPH ? sh.sphere[lane] : -1;
    h.b1 = h.b2 = 0.0f;
    uint32_t rec = 0xFFFFFFFFu;
    uint32_t outside = 0xFFFFFFFFu;  // the hit's record, if its triangle reaches out of the root box
    if (ANY) {
      if (found) h.prim = 0;
      kd = kd || sh.tie[lane] != 0xFFFFFFFFu;
    } else {
      const unsigned long long key = sh.key[lane];
      h.t = wide_unorder((uint32_t)(key >> 32));
      rec = (uint32_t)key;
      // (a pair behind the final hit is no tie)
      kd = kd || (sh.tie[lane] != 0xFFFFFFFFu && wide_unorder(sh.tie[lane]) - h.t <= kWideTie * fabsf(h.t));
    }
    const int64_t q = 3 * (int64_t)rec;
    F4 b = {};
    if (!ANY && rec < 0xFFFFFFFEu) {
      b = load_f4(s.wtris, q + 1);
      if (OUT && !kd && (f_bits(b.w) & kWideOutside) != 0u) {
        outside = rec;
        kd = true;
      }
    }
    if (kd || (!ANY && rec < 0xFFFFFFFEu)) {
      Ray r;
      load(i, r);
      if (kd) {
        kd_ray<ANY, SPH, QUERY, OUT>(s, r, h, OUT ? (ANY ? sh.tie[lane] : outside) : 0xFFFFFFFFu);
      } else {
        // the winner again, for its barycentrics: the same inputs, the same result
        const F4 a = load_f4(s.wtris, q), c = load_f4(s.wtris, q + 2);
        float t;
        intersect_tri(precompute(r), v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z),
                      (f_bits(b.w) & 1u) != 0u, r.tmin, r.tmax, t, h.b1, h.b2);
        h.prim = (int32_t)f_bits(a.w);
      }
    }
    store(i, h.prim >= 0, h);
  }
};

// The rays of a block: chunks of rays gridDim apart; as many rounds of at most kWideChunk as the rays need,
// of equal size, so that few rays still spread over all blocks.
struct WideChunks {
  uint32_t chunk;
  __device__ __forceinline__ explicit WideChunks(uint32_t n) {
    const unsigned long long per = (unsigned long long)gridDim.x * kWideChunk;
    const unsigned long long rounds = ((unsigned long long)n + per - 1) / per;
    chunk = rounds ? ((uint32_t)(((unsigned long long)n + gridDim.x * rounds - 1) / (gridDim.x * rounds)) + 31u) & ~31u
                   : 32u;
  }
  // the block's pos-th ray (n or more: none left)
  __device__ __forceinline__ unsigned long long ray(uint32_t pos) const {
    return ((unsigned long long)(pos / chunk) * gridDim.x + blockIdx.x) * chunk + pos % chunk;
  }
};

// All of them, by one block.
struct WideAll {
  __device__ __forceinline__ unsigned long long ray(uint32_t pos) const { return pos; }
};

// Rays 0 .. n - 1 (those that `rays` gives the block), a warp's 32 to completion (next: a counter of the block, zero at the start).  For rays that
// lie in a queue with their neighbours: a lane that ends early waits, which costs less than what the other
// shape (below) adds to the node loop's registers (mid frame 83.7 against 92 ms).
// All 32 lanes of every warp must call this.
template <bool ANY, bool COUNT, bool SPH, bool SINGLE, class Rays, class View, class Load, class Store>
__device__ __forceinline__ void wide_trace(const Rays &rays, View view, uint32_t n, Load load, Store store,
                                           WideShared &sh, const WideTables &tab, uint32_t *next, TraceCounts *cnt,
                                           uint32_t &rays_done) {
  constexpr unsigned kFull = 0xFFFFFFFFu;
  uint2 stack[kWideMaxDepth];
  const uint32_t lane = threadIdx.x & 31u;
  for (;;) {
    uint32_t pos = 0u;
    if (lane == 0u) pos = atomicAdd(next, 32u);
    const unsigned long long first = rays.ray(__shfl_sync(kFull, pos, 0));
    if (first >= n) break;
    const uint32_t i = (uint32_t)first + lane;
    __syncwarp(kFull);  // the previous rays' readers are done with the shared records
    WideWarp<ANY, COUNT, SPH, SINGLE, false, true, View, Load, Store> t{view, load, store, sh, tab, cnt, lane, stack};
    if (i < n) {
      t.start(i);
      ++rays_done;
    }
    while (__any_sync(kFull, t.active)) {
      if (t.active) t.step();
      for (uint32_t m; (m = __ballot_sync(kFull, t.tg.bits != 0u)) != 0u;) {
        if (t.tg.bits) t.push(m);
        t.qn += __popc(m);
        if (t.qn >= 32u) t.round(32u);
      }
      if (t.qn >= kWideFlush) t.round(t.qn);
    }
    if (t.qn) t.round(t.qn);
    if (ANY) __syncwarp(kFull);  // sh.tie (a round of closest hits ends with one)
    if (i < n) t.finish(i);
  }
}

// Rays 0 .. n - 1 in any order of the caller's: lanes whose rays have ended take new ones whenever
// kWideRefill of them wait (1 M random rays, 300 k triangles: closest 0.307 -> 0.224 ms, any
// 0.207 -> 0.125; 12 or 16 measure the same, 8 and 20 less).
// All 32 lanes of every warp must call this.
constexpr uint32_t kWideRefill = 16u;

template <bool ANY, bool SPH, bool OUT, class View, class Load, class Store>
__device__ __forceinline__ void wide_trace_refill(View view, uint32_t n, Load load, Store store, WideShared &sh,
                                                  const WideTables &tab, uint32_t *next) {
  constexpr unsigned kFull = 0xFFFFFFFFu;
  uint2 stack[kWideMaxDepth];
  const WideChunks chunks(n);
  WideWarp<ANY, false, SPH, true, true, OUT, View, Load, Store> t{view, load, store, sh, tab, nullptr, threadIdx.x & 31u, stack};
  uint32_t i = 0u;
  bool have = false;  // the lane holds ray i
  bool more = true;   // the block has rays left (uniform over the warp)
  for (bool swap = true;;) {
    if (swap) {
      if (ANY) __syncwarp(kFull);  // sh.tie
      if (have && !t.active) {
        t.finish(i);
        have = false;
      }
      if (more) {
        const uint32_t want = __ballot_sync(kFull, !have);
        uint32_t pos = 0u;
        if (t.lane == 0u) pos = atomicAdd(next, (uint32_t)__popc(want));
        const unsigned long long r =
            chunks.ray(__shfl_sync(kFull, pos, 0) + __popc(want & ((1u << t.lane) - 1u)));
        more = !__any_sync(kFull, !have && r >= n);
        if (!have && r < n) {
          have = true;
          i = (uint32_t)r;
          t.start(i);
        }
      }
      if (!__any_sync(kFull, have)) break;
    }
    if (t.active) t.step();
    const uint32_t busy = __popc(__ballot_sync(kFull, t.active));
    swap = busy == 0u || (more && busy <= 32u - kWideRefill);
    for (uint32_t m = __ballot_sync(kFull, t.tg.bits != 0u);;) {
      while (m != 0u && t.qn < 32u) {
        if (t.tg.bits) t.push(m);
        t.qn += __popc(m);
        m = __ballot_sync(kFull, t.tg.bits != 0u);
      }
      if (t.qn < (swap ? 1u : kWideFlush)) break;
      t.round(min(t.qn, 32u));
      if (ANY) m = __ballot_sync(kFull, t.tg.bits != 0u);
    }
  }
}

#endif  // __CUDACC__

}  // namespace mgpu
