// hd_wide.h -- 8-wide bounding-volume hierarchy traversal of the render and ray-query kernels.
//
// The hierarchy is built on the device when a scene is created (bvh.cu) and answers the same
// queries as the kd-tree (hd_trace.h) with the same triangle test: a closest hit is the smallest
// accepted t over the scene's triangles, whatever visits them, so both give the same primitive, t
// and barycentrics, bit for bit.
//
// Why a wide hierarchy: on the mid scene (1 M triangles) the kd-tree takes 50 dependent node steps
// and 33 triangle tests per ray.  The node here holds eight child boxes on an 8-bit grid of the
// parent's box in 80 bytes (five 128-bit loads), as in Ylitie, Karras and Laine, "Efficient
// Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs", HPG 2017.
//
// Node (20 words):
//   0..2   origin of the child grid (below the node's box on every axis)
//   3      grid step per axis as the biased exponent of 2^15 x step (8 bits each: x, y, z), then
//          the mask of the slots that hold inner nodes
//   4      index of the first inner child (the inner children of a node are consecutive, in slot
//          order)
//   5      index of the node's first triangle record (the leaf children's triangles are
//          consecutive, in slot order)
//   6      triangles of the leaf children: bits 3 s .. 3 s + 2 hold slot s's count in unary
//   7      unused
//   8..19  child planes: low x, y, z then high x, y, z, 8 bytes each (one per slot)
// Triangle record: 3 x float4 as a kd leaf's (v0 + primitive id, v1 + flags, v2).
//
// A slot's number says where its child lies: bit k set = the upper side along axis k.  A ray visits
// the children it meets in the order of slot XOR (its negative directions), which is front to
// back along its octant, so the stack holds one entry (the siblings still to visit) per level.
#pragma once

#include "hd_trace.h"

namespace mgpu {

constexpr int kWideWords = 20;       // 32-bit words per node
constexpr int kWideLeafTris = 3;     // triangles per leaf child
constexpr int kWideMaxDepth = 30;    // levels of node below the root that the traversal stack holds
constexpr uint32_t kWideRootBits = 0x100u;  // sibling mask of the pseudo parent of the root
// Threads per block: one block per SM at 64 registers a thread.  The rays of one SM are then
// neighbours in the (sorted) queue and share its L1: mid frame, traversal 117 ms in blocks of 128,
// 114 / 108 / 102 ms in blocks of 256 / 512 / 1024.
constexpr int kWideBlock = 1024;
// Rays that a block takes at a time; its warps take them 32 by 32 as they finish (mid frame: 97.0,
// 96.3, 98.2, 101.1 ms at 1024, 512, 2048, 4096 against 102 in fixed grid-stride rounds).
constexpr uint32_t kWideChunk = 512u;
// Triangle tests waiting after a node step that are worth a round of their own: a full queue (32) keeps
// every lane busy but lets the rays go on with a stale closest t (mid closest hits: 49.9 / 46.9 /
// 46.5 ms at 32 / 16 / 8).
constexpr uint32_t kWideFlush = 8u;

// Box tests are conservative.  The builder leaves at least 1/64 step of slack around every child, which
// covers the rounding of the plane distances relative to the node's own size; what is relative to
// the distance |p - o| from the ray's origin (the subtraction, the products, and the triangle
// test's sheared coordinates, together below 6 x 2^-24 |p - o|) is covered by moving every plane
// outward by 2^-20 max |p - o|.
constexpr float kWideEps = 1.0f / 1048576.0f;

#if defined(__CUDACC__)

// the byte `i` of w as the float 1 + byte / 2^15: one byte permute, no integer conversion
__device__ __forceinline__ float wide_byte(uint32_t w, int i) {
  return __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604u | ((uint32_t)i << 4)));
}

// bits of an 8-bit mask moved from s to s XOR x
__device__ __forceinline__ uint32_t wide_permute(uint32_t m, uint32_t x) {
  if (x & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
  if (x & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
  if (x & 4u) m = ((m & 0x0Fu) << 4) | (m >> 4);
  return m;
}

// bit s of an 8-bit mask -> bits 3 s .. 3 s + 2
__device__ __forceinline__ uint32_t wide_spread3(uint32_t m) {
  m = (m | (m << 8)) & 0x00F00Fu;
  m = (m | (m << 4)) & 0x0C30C3u;
  m = (m | (m << 2)) & 0x249249u;
  return m * 7u;
}

struct WideGroup {
  uint32_t base;  // nodes: first inner child of the parent; triangles: the node's first record
  uint32_t bits;  // nodes: pending children (permuted, bits 0..7) | inner mask << 8; triangles: pending
};

// Tests the eight children of node idx against (tmin, best]: pending inner children and triangles.
__device__ __forceinline__ void wide_node(const uint4 *__restrict__ nodes, uint32_t idx, V3 o, V3 inv, float tmin,
                                          float best, uint32_t octx, WideGroup &ng, WideGroup &tg, uint32_t &tvalid) {
  const uint4 *q = nodes + (size_t)idx * (kWideWords / 4);
  const uint4 n0 = __ldg(q), n1 = __ldg(q + 1), n2 = __ldg(q + 2), n3 = __ldg(q + 3), n4 = __ldg(q + 4);
  const float dx = __uint_as_float(n0.x) - o.x, dy = __uint_as_float(n0.y) - o.y, dz = __uint_as_float(n0.z) - o.z;
  const float m = kWideEps * fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz)));
  const float ax = __uint_as_float((n0.w & 0xFFu) << 23) * inv.x;
  const float ay = __uint_as_float(((n0.w >> 8) & 0xFFu) << 23) * inv.y;
  const float az = __uint_as_float(((n0.w >> 16) & 0xFFu) << 23) * inv.z;
  const float cx = fmaf(dx, inv.x, -ax), cy = fmaf(dy, inv.y, -ay), cz = fmaf(dz, inv.z, -az);
  const float ex = m * fabsf(inv.x), ey = m * fabsf(inv.y), ez = m * fabsf(inv.z);
  const float nx = cx - ex, ny = cy - ey, nz = cz - ez, fx = cx + ex, fy = cy + ey, fz = cz + ez;
  const bool sx = inv.x < 0.0f, sy = inv.y < 0.0f, sz = inv.z < 0.0f;
  uint32_t hits = 0u;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t lox = h ? n2.y : n2.x, loy = h ? n2.w : n2.z, loz = h ? n3.y : n3.x;
    const uint32_t hix = h ? n3.w : n3.z, hiy = h ? n4.y : n4.x, hiz = h ? n4.w : n4.z;
    const uint32_t nearx = sx ? hix : lox, neary = sy ? hiy : loy, nearz = sz ? hiz : loz;
    const uint32_t farx = sx ? lox : hix, fary = sy ? loy : hiy, farz = sz ? loz : hiz;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float t0 = fmaxf(fmaxf(fmaf(wide_byte(nearx, i), ax, nx), fmaf(wide_byte(neary, i), ay, ny)),
                             fmaxf(fmaf(wide_byte(nearz, i), az, nz), tmin));
      const float t1 = fminf(fminf(fmaf(wide_byte(farx, i), ax, fx), fmaf(wide_byte(fary, i), ay, fy)),
                             fminf(fmaf(wide_byte(farz, i), az, fz), best));
      if (t0 <= t1) hits |= 1u << (4 * h + i);
    }
  }
  const uint32_t imask = n0.w >> 24;
  ng.base = n1.x;
  ng.bits = wide_permute(hits & imask, octx) | (imask << 8);
  tg.base = n1.y;
  tvalid = n1.z;
  tg.bits = wide_spread3(hits & ~imask) & tvalid;
}

// What a lane keeps in registers through the node steps.  The triangle tests' ray constants are in
// shared memory (WideShared).
struct WideRay {
  V3 o, inv;
  float tmin;
  float best;      // closest t accepted so far (starts at the ray's tmax)
  uint32_t octx;   // 7 XOR the ray's negative directions: pending children are taken from the top bit
};

// Per-warp shared memory: every lane's ray for the triangle tests, its best hit so far, and the queue
// of (lane, triangle) tests waiting for a full round.
struct WideShared {
  float4 a[32], b[32];       // (o, tmin), (sx, sy, sz, tmax)
  unsigned long long key[32];  // closest hit: ordered t << 32 | triangle record; ~0 record: none
  uint32_t k[32];            // axis permutation
  uint32_t rec[64];          // queue (ring of 64): triangle record
  uint8_t own[64];           // ... and the lane it is for
  const F4 *tris[32];        // the lanes' scenes' triangle records (waves of several scenes)
  uint32_t tie[32];          // ordered t of the nearest pair of hits within kWideTie of each other
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
// So is a ray with a zero direction component: one that lies in a split plane sees only the cells on one
// side of it in the kd-tree.
constexpr float kWideTie = 1.0f / 131072.0f;

// The kd-tree's answer for one ray: closest hit, or any (h.prim >= 0).  SEQ: a leaf's triangles one after
// another, each against the t before it; otherwise the smallest (t, leaf order) among those accepted
// against the t before the leaf.
template <bool ANY, bool SPH, bool SEQ>
__device__ __noinline__ void kd_ray(const SceneView &s, const Ray &r, Hit &h) {
  TravState st;
  TravEntry stack[kMaxStack];
  if (trav_init<SPH>(s, r, nullptr, 0, st, ANY)) {
    bool done = false;
    while (!done) {
      uint32_t w0, w1;
      float tmax;
      trav_descend<false>(s, st, stack, nullptr, 0, nullptr, w0, w1, tmax);
      const float best0 = st.best;
      bool took = false;
      for (uint32_t i = 0; i < (w0 >> 2) && !(ANY && took); ++i) {
        const int64_t q = 3 * ((int64_t)w1 + i);
        const F4 a = load_f4(s.ltris, q), b = load_f4(s.ltris, q + 1), c = load_f4(s.ltris, q + 2);
        float t, b1, b2;
        if (intersect_tri(st.pre, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), (f_bits(b.w) & 1u) != 0u,
                          st.ray_tmin, SEQ ? st.best : best0, t, b1, b2) &&
            (SEQ || !took || t < st.best)) {
          took = true;
          st.best = t; st.best_prim = (int32_t)f_bits(a.w); st.bb1 = b1; st.bb2 = b2;
        }
      }
      done = (ANY && took) || trav_after_leaf<false>(st, stack, tmax);
    }
  }
  h.t = st.best;
  h.prim = st.best_prim;
  h.b1 = st.bb1;
  h.b2 = st.bb2;
}

// Traversal of rays 0 .. n - 1, 32 per warp to completion.  Every lane steps through the nodes of its own
// ray; the triangles it meets go into the warp's queue, and the warp tests them together, each lane one
// (ray, triangle) pair whoever's it is, with the owner's constants from shared memory.  A node step
// finds a triangle for about half the lanes and up to six for one, so testing them lane by lane ran
// the test with a sixth of the lanes (mid frame, closest hits: 78 -> 59 ms).
// What bounds it (ncu, mid scene, second bounce): instruction issue, 85 % of the slots and the ALU pipe at
// 76 %, with 17 of 32 lanes active; L1 hit rate 81 %, L2 below 8 % and DRAM below 3 % of their peaks.
// The kd-tree's kernels were bound by the latency of 50 dependent node loads per ray.
// Mid frame (163 M closest hits + 226 M occlusion queries): 187.7 -> 95.8 ms of traversal.
//   ANY     occlusion: the first hit ends the ray; otherwise the closest
//   SEQ     which of the kd-tree's orders decides near ties (kd_ray)
//   SINGLE  every ray is in the scene view(0), which the kernel passes from its parameter space
//   next    a counter of the block, zero at the start
// All 32 lanes of every warp must call this.
template <bool ANY, bool SEQ, bool COUNT, bool SPH, bool SINGLE, class View, class Load, class Store>
__device__ __forceinline__ void wide_trace(View view, uint32_t n, Load load, Store store, WideShared &sh, uint32_t *next,
                                           TraceCounts *cnt, uint32_t &rays_done) {
  constexpr unsigned kFull = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  uint2 stack[kWideMaxDepth];
  // the block takes chunks of rays, gridDim apart; as many rounds of at most kWideChunk as the rays
  // need, of equal size, so that few rays still spread over all blocks
  const unsigned long long rounds = ((unsigned long long)n + gridDim.x * kWideChunk - 1) / (gridDim.x * kWideChunk);
  const uint32_t chunk =
      rounds ? ((uint32_t)(((unsigned long long)n + gridDim.x * rounds - 1) / (gridDim.x * rounds)) + 31u) & ~31u : 32u;
  for (;;) {
    uint32_t pos = 0u;
    if (lane == 0u) pos = atomicAdd(next, 32u);
    pos = __shfl_sync(kFull, pos, 0);
    const unsigned long long r0l =
        ((unsigned long long)(pos / chunk) * gridDim.x + blockIdx.x) * chunk + pos % chunk;
    if (r0l >= n) break;
    const uint32_t r0 = (uint32_t)r0l;
    const uint32_t i = r0 + lane;
    const SceneView &s = view(min(i, n - 1u));
    const uint4 *nodes = s.wnodes;
    WideRay w{};
    WideGroup ng{0u, 0u}, tg{0u, 0u};
    uint32_t tvalid = 0u;
    int sp = 0;
    bool active = false, found = false, kd = false;
    int32_t sphere = -1;
    __syncwarp(kFull);  // the previous rays' readers are done with the shared records
    if (i < n) {
      Ray r;
      load(i, r);
      ++rays_done;
      float best = r.tmax;
      if (SPH && s.nsphere > 0) {
        TravState ts;
        ts.best = r.tmax;
        ts.best_prim = -1;
        spheres_hit(s, r, ts, ANY);
        best = ts.best;
        sphere = ts.best_prim;
      }
      active = s.ntri > 0 && !(ANY && sphere >= 0);
      if (active) {
        float t0, t1;
        active = clip_root(s, r, v3(1.0f / r.d.x, 1.0f / r.d.y, 1.0f / r.d.z), t0, t1) &&
                 fmaxf(t0, r.tmin) <= fminf(t1, r.tmax);
        kd = active && (r.d.x == 0.0f || r.d.y == 0.0f || r.d.z == 0.0f);
        active = active && !kd;
      }
      if (active) {
        const RayPre pre = precompute(r);
        w.o = r.o;
        w.inv = v3(safe_rcp(r.d.x), safe_rcp(r.d.y), safe_rcp(r.d.z));
        w.tmin = r.tmin;
        w.best = best;
        w.octx = 7u ^ ((w.inv.x < 0.0f ? 1u : 0u) | (w.inv.y < 0.0f ? 2u : 0u) | (w.inv.z < 0.0f ? 4u : 0u));
        ng.bits = (1u << w.octx) | kWideRootBits;
        sh.a[lane] = make_float4(r.o.x, r.o.y, r.o.z, r.tmin);
        sh.b[lane] = make_float4(pre.sx, pre.sy, pre.sz, r.tmax);
        if (!SINGLE) sh.tris[lane] = s.wtris;
        sh.k[lane] = (uint32_t)pre.kx | ((uint32_t)pre.ky << 2) | ((uint32_t)pre.kz << 4);
      }
      if (!ANY) {
        sh.key[lane] = ((unsigned long long)wide_order(best) << 32) | (sphere >= 0 ? 0xFFFFFFFEu : 0xFFFFFFFFu);
        sh.tie[lane] = 0xFFFFFFFFu;
      }
    }
    uint32_t qh = 0u, qn = 0u;  // queue head and length (uniform over the warp)
    auto round = [&](uint32_t m) {  // tests the queue's first m <= 32 entries
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
        const F4 *lt = SINGLE ? s.wtris : sh.tris[o];
        const int64_t q = 3 * (int64_t)rec;
        const F4 a = load_f4(lt, q), b = load_f4(lt, q + 1), c = load_f4(lt, q + 2);
        if (COUNT) cnt->tris++;
        float t, b1, b2;
        if (intersect_tri(p, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), (f_bits(b.w) & 1u) != 0u, ra.w,
                          rb.w, t, b1, b2)) {
          if (ANY) {
            hit = 1u << o;
          } else {
            const unsigned long long old =
                atomicMin(&sh.key[o], ((unsigned long long)wide_order(t) << 32) | rec);
            const float told = wide_unorder((uint32_t)(old >> 32));
            if ((uint32_t)old != 0xFFFFFFFFu && fabsf(t - told) <= kWideTie * fabsf(t)) atomicMin(&sh.tie[o], wide_order(fminf(t, told)));
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
        w.best = wide_unorder((uint32_t)(sh.key[lane] >> 32));
      }
    };
    while (__any_sync(kFull, active)) {
      if (active) {
        const uint32_t pos = 31u - __clz(ng.bits & 0xFFu);
        ng.bits &= ~(1u << pos);
        const uint32_t slot = pos ^ w.octx;
        const uint32_t idx = ng.base + __popc((ng.bits >> 8) & ((1u << slot) - 1u));
        if (ng.bits & 0xFFu) stack[sp++] = make_uint2(ng.base, ng.bits);
        if (COUNT) cnt->nodes++;
        wide_node(nodes, idx, w.o, w.inv, w.tmin, w.best, w.octx, ng, tg, tvalid);
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
      for (uint32_t m; (m = __ballot_sync(kFull, tg.bits != 0u)) != 0u;) {
        if (tg.bits) {
          const uint32_t k = __ffs(tg.bits) - 1, e = (qh + qn + __popc(m & below)) & 63u;
          tg.bits &= tg.bits - 1u;
          sh.rec[e] = tg.base + __popc(tvalid & ((1u << k) - 1u));
          sh.own[e] = (uint8_t)lane;
        }
        qn += __popc(m);
        if (qn >= 32u) round(32u);
      }
      if (qn >= kWideFlush) round(qn);
    }
    if (qn) round(qn);
    if (i < n) {
      Hit h;
      h.prim = sphere;
      h.b1 = h.b2 = 0.0f;
      uint32_t rec = 0xFFFFFFFFu;
      if (ANY) {
        if (found) h.prim = 0;
      } else {
        const unsigned long long key = sh.key[lane];
        h.t = wide_unorder((uint32_t)(key >> 32));
        rec = (uint32_t)key;
        // (a pair behind the final hit is no tie)
        kd = kd || (sh.tie[lane] != 0xFFFFFFFFu && wide_unorder(sh.tie[lane]) - h.t <= kWideTie * fabsf(h.t));
      }
      if (kd || (!ANY && rec < 0xFFFFFFFEu)) {
        Ray r;
        load(i, r);
        if (kd) {
          kd_ray<ANY, SPH, SEQ>(s, r, h);
        } else {
          // the winner again, for its barycentrics: the same inputs, the same result
          const int64_t q = 3 * (int64_t)rec;
          const F4 a = load_f4(s.wtris, q), b = load_f4(s.wtris, q + 1), c = load_f4(s.wtris, q + 2);
          float t;
          intersect_tri(precompute(r), v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z),
                        (f_bits(b.w) & 1u) != 0u, r.tmin, r.tmax, t, h.b1, h.b2);
          h.prim = (int32_t)f_bits(a.w);
        }
      }
      store(i, h.prim >= 0, h);
    }
  }
}

#endif  // __CUDACC__

}  // namespace mgpu
