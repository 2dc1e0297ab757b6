// render.cu -- wavefront path tracer: generate -> (extend -> shade -> shadow)* -> accumulate.
//
// Work is organised in waves of paths.  A wave holds one or more job chunks; a chunk is a range
// of pixel slots (8x8 tiles, row-major tile order) x a range of sample passes of one render job
// (one scene, camera, film and set of PathTracer parameters).  A plain render is one job; a batch
// (mgpu_batch_*) packs the chunks of many jobs of uneven size into shared waves, so small scenes
// fill the GPU together.  Per-chunk parameters live in a device array of JobArgs; every path
// records its chunk in path_job[], and every kernel reads its chunk's scene and parameters there.
//
// Per path the state is split in two:
//   path_L[p]     float4  radiance accumulated so far (rgb) + path flags (w) -- path-indexed,
//                          updated by shade (emission, folded direct light), read by accumulate;
//   ray queue     3 x float4 per live path (origin + path index, direction + chunk, throughput +
//                          depth state), compacted every bounce by warp ballot + one atomicAdd per
//                          warp.
// Direct light (DirectIllumination::evaluate over all lights x noDirectSamples,
// DirectIllumination.cpp:46-138) is split in two: shade samples every light, evaluates the BSDF,
// writes each sample's contribution into the path's slot for that sample and queues one shadow
// ray per non-zero contribution; the shadow kernel is a plain any-hit query that zeroes the slot
// of an occluded sample.  The next kernel to see the path (shade at the next bounce, or
// accumulate) folds its slots into the radiance in slot order, so every sum runs in a fixed
// order and the image does not depend on queue order, wave size or batch composition.
#include <string.h>

#include <algorithm>
#include <climits>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"
#include "hd_wide.h"

namespace mgpu {

constexpr int kBlock = 128;
constexpr int kHardCap = 1024;          // vertex cap when max_depth = 0 (Milton has none)
constexpr int kCtrRay = 0;              // counters[kCtrRay + b]  live paths at bounce b
constexpr int kCtrNee = kHardCap + 8;   // counters[kCtrNee + b]  shadow rays at bounce b
constexpr int kCtrTrunc = 2 * (kHardCap + 8);
constexpr int kNumCounters = kCtrTrunc + 8;
constexpr int kBinBits = 14;           // queue binning keys: 2^14 bins
constexpr int kBins = 1 << kBinBits;
constexpr int kBinSmem = kBins * 4;    // dynamic shared memory of a sorting block
constexpr int64_t kBinMinTris = 300000;   // smallest scene whose extension rays are sorted
constexpr double kAutoWaveBytes = 40e9;  // workspace budget of an automatic wave
// Resident 128-thread blocks per SM that the kd-tree kernels are compiled for: 40 registers
constexpr int kTravMinBlocks = 12;

// One job chunk of a wave (device memory).
struct JobArgs {
  SceneView view;
  const float4 *shade;
  const float4 *mats;    // 4 per material
  const float4 *lights;  // 4 per light
  const float2 *uv;      // 3 per triangle (nullptr: every uv is (0, 0))
  const float4 *texrec;  // 2 per texture
  const float4 *texels;
  int32_t bg_tex;          // background environment map (1 + texture index) or 0
  float bg_le[3];          // constant background radiance (bg_tex == 0)
  int32_t nlight, nl_slots;
  float cell_scale[3];     // queue-bin cells: 32 / the scene's extent per axis (0: a flat axis)
  Camera cam;
  Rng rng;
  int32_t W, H, spp, side, s2, nds, nds_side, max_depth, rr_start, efficient, tiles_x;
  int32_t s0, ns;                 // samples [s0, s0 + ns) of this chunk
  int32_t sample_begin, sample_count;
  int64_t slot0, nslots;          // slots [slot0, slot0 + nslots)
  int64_t path_base;              // first wave path of the chunk
  int64_t slot_base;              // first accumulate slot of the chunk in the wave
  float4 *film_sum, *film_c;
  FilmFilter filt;                 // reconstruction filter of the film (kFilterNone: mean only)
  unsigned long long *film_fx;     // its fixed-point splat sums (4 per pixel)
  float4 *path_out;               // optional per-path radiance
};

// One wave (kernel parameter).
struct RenderArgs {
  const JobArgs *jobs;
  int32_t njobs;
  int64_t npaths, nslots;         // paths and accumulate slots in the wave
  int32_t nl_stride;              // light-sample slots per path (max over the wave's chunks)
  uint32_t *path_job;
  float4 *path_L;
  float4 *qo[2], *qd[2], *qt[2];
  float4 *qhit;
  float4 *so, *sd;               // shadow ray queue: origin + slot index, direction + tmax
  float4 *slots;                 // nl_stride per path: direct-light contribution per light sample
  float4 *qo_u, *qd_u, *qt_u;    // unsorted next-ray queue (binning on)
  uint32_t *qkey;                // bin keys of the unsorted queue
  int32_t bin_ext;               // counting-sort the queue by (direction octant, origin cell)
  int32_t dense;                 // every slot of the wave is a pixel
  int32_t sort_hits;             // a scene of the wave has more than one kind of BSDF
  uint32_t *counters;
  unsigned long long *stats;     // [0] extension rays, [1] shadow rays, [2] truncated paths, [3] bounces
  unsigned long long *tcount;    // counted mode: ext nodes, refs, tris, rays; shadow nodes, refs, tris, rays
  int32_t max_b;
  SceneView view0;               // the scene of a wave of one scene (njobs == 1)
};

// A film has fewer than 2^31 pixels and a wave fewer than 2^31 paths (both checked on the host),
// so slot and path indices within a chunk are divided in 32-bit unsigned arithmetic (a 64-bit
// division is several times the instructions, and these run for every path in three kernels).
__device__ __forceinline__ bool slot_pixel(const JobArgs &J, int64_t slot, int &x, int &y) {
  const uint32_t tile = (uint32_t)(slot >> 6), tx = (uint32_t)J.tiles_x;
  const uint32_t ty = tile / tx;
  const int within = (int)(slot & 63);
  x = (int)(tile - ty * tx) * 8 + (within & 7);
  y = (int)ty * 8 + (within >> 3);
  return x < J.W && y < J.H;
}

// global path id (pixel * spp + sample) for wave path p of chunk J
__device__ __forceinline__ uint64_t path_id(const JobArgs &J, int64_t p, int &x, int &y, int &s) {
  const uint32_t lp = (uint32_t)(p - J.path_base), ns = (uint32_t)J.ns;
  const uint32_t q = lp / ns;
  const int64_t slot = J.slot0 + q;
  s = J.s0 + (int)(lp - q * ns);
  slot_pixel(J, slot, x, y);
  return ((uint64_t)y * J.W + x) * (uint64_t)J.spp + (uint64_t)s;
}

// chunk holding wave path p / accumulate slot q (binary search over the sorted bases)
__device__ __forceinline__ int job_of_path(const RenderArgs &a, int64_t p) {
  int lo = 0, hi = a.njobs - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (a.jobs[mid].path_base <= p) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ int job_of_slot(const RenderArgs &a, int64_t q) {
  int lo = 0, hi = a.njobs - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (a.jobs[mid].slot_base <= q) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// warp-aggregated queue append: returns the slot for this lane (valid only if want)
__device__ __forceinline__ uint32_t warp_append(uint32_t *counter, bool want) {
  unsigned active = __activemask();
  unsigned mask = __ballot_sync(active, want);
  if (mask == 0) return 0;
  int lane = threadIdx.x & 31;
  int leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
  base = __shfl_sync(active, base, leader);
  return base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

__device__ __forceinline__ Material load_mat(const JobArgs &J, int i, uint32_t ior_index) {
  float m[16];
  float4 *mm = reinterpret_cast<float4 *>(m);
#pragma unroll
  for (int k = 0; k < 4; ++k) mm[k] = __ldg(J.mats + 4 * i + k);
  return material_from(m, ior_index);
}

// Image maps at a hit of triangle prim with barycentrics (b0, b1, b2): the uv (Shape::_getUV,
// interpolated from the per-vertex uvs), then each textured key of the material and the bump
// map (Material::initSurfacePoint, Material.cpp:157-225).
__device__ __noinline__ void apply_textures(const JobArgs &J, int prim, float b0, float b1, float b2, V3 P,
                                            Material &m, V3 &ns) {
  float u = 0.0f, v = 0.0f;
  if (prim >= J.view.ntri) {
    // Sphere::_getUV (Sphere.cpp:78-85) of the object-space point: the offset from the centre,
    // rotated into the sphere's frame, over its diameter
    const float4 c = __ldg(reinterpret_cast<const float4 *>(J.view.spheres) + 2 * (prim - J.view.ntri));
    const float4 q = __ldg(reinterpret_cast<const float4 *>(J.view.spheres) + 2 * (prim - J.view.ntri) + 1);
    sphere_uv(quat_rotate(q.x, q.y, q.z, q.w, (P - v3(c.x, c.y, c.z)) * (0.5f / c.w)), u, v);
  } else if (J.uv) {
    const float2 a = __ldg(J.uv + 3 * (int64_t)prim), b = __ldg(J.uv + 3 * (int64_t)prim + 1),
                 c = __ldg(J.uv + 3 * (int64_t)prim + 2);
    u = a.x * b0 + b.x * b1 + c.x * b2;
    v = a.y * b0 + b.y * b1 + c.y * b2;
  }
  const int slots[4] = {m.tex_kd, m.tex_ks, m.tex_tr, m.tex_bump};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (slots[k] == 0) continue;
    const float4 r0 = __ldg(J.texrec + 2 * (slots[k] - 1)), r1 = __ldg(J.texrec + 2 * (slots[k] - 1) + 1);
    const int w = __float_as_int(r0.y), h = __float_as_int(r0.z);
    const float4 t = __ldg(J.texels + __float_as_uint(r0.x) + tex_texel(u, v, w, h, r1.x, r1.y));
    if (k < 3) tex_apply(m, k, t.x, t.y, t.z);
    else ns = bump_normal(ns, t.x, t.y, r1.z);
  }
}

// Background radiance of a ray leaving the scene in direction d: EnvironmentMap::getLe(-d)
// (the map's filtered texel at the uv of -d) or the constant of an omni background.
__device__ __noinline__ V3 background(const JobArgs &J, V3 d) {
  if (J.bg_tex == 0) return v3(J.bg_le[0], J.bg_le[1], J.bg_le[2]);
  float u, v;
  env_uv(-d, u, v);
  const float4 r0 = __ldg(J.texrec + 2 * (J.bg_tex - 1)), r1 = __ldg(J.texrec + 2 * (J.bg_tex - 1) + 1);
  const int w = __float_as_int(r0.y), h = __float_as_int(r0.z);
  const float4 t = __ldg(J.texels + __float_as_uint(r0.x) + tex_texel(u, v, w, h, r1.x, r1.y));
  return v3(t.x, t.y, t.z);
}

// light records: 8 float4 each (base record, then the extension)
__device__ __forceinline__ Light load_light(const JobArgs &J, int i) {
  float l[32];
  float4 *ll = reinterpret_cast<float4 *>(l);
#pragma unroll
  for (int k = 0; k < 8; ++k) ll[k] = __ldg(J.lights + 8 * i + k);
  return light_from(l, l + 16);
}

// Binning keys (kBins = 16384).  Ray coherence: rays of one warp should start close together
// and head the same way, so that they visit the same nodes.  Keys combine the direction
// octant with the Morton code of the origin's cell in a 32x32x32 grid over the scene bounds (the
// top bits of it that fit).
__device__ __forceinline__ uint32_t spread4(uint32_t v) {  // 4 bits -> every third bit
  return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6);
}

__device__ __forceinline__ uint32_t spread5(uint32_t v) {  // 5 bits -> every third bit
  return spread4(v & 15u) | ((v & 16u) << 8);
}

// The keys only order the queues (no result depends on them), so the cell is taken with a
// multiplication by the precomputed 32 / extent rather than a division per axis.
__device__ __forceinline__ uint32_t morton15(const JobArgs &J, V3 p) {
  uint32_t c[3];
  const float pp[3] = {p.x, p.y, p.z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int q = (int)((pp[k] - J.view.bmin[k]) * J.cell_scale[k]);
    c[k] = (uint32_t)min(max(q, 0), 31);
  }
  return (spread5(c[0]) << 2) | (spread5(c[1]) << 1) | spread5(c[2]);
}

__device__ __forceinline__ uint32_t ext_key(const JobArgs &J, V3 o, V3 d) {
  uint32_t oct = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
  return (oct << (kBinBits - 3)) | (morton15(J, o) >> (18 - kBinBits));
}

// Most kernels of a small wave are launched so that they may start while the one before it drains (programmatic
// stream serialization): every thread of every kernel calls chain() before it touches memory that another
// kernel writes; it waits there until the kernel before has ended and its writes are visible.  Without
// that launch attribute it returns at once.
__device__ __forceinline__ void chain() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ---------------------------------------------------------------------------------------
// generate: camera rays for every path of the wave (RayTracer::sample, RayTracer.cpp:19-30;
// SuperSampleGenerator strata, SuperSampleGenerator.cpp:60-90)
// A path's entry in the queue is its index in the wave where every slot is a pixel (a.dense: image sides that
// are multiples of 8), else a block reserves its live paths with one atomic (one per warp was 2 M to
// one address on the mid frame).  Throughput and state of a first vertex are constants that shading knows
//.
constexpr int kGenBlock = 256;

__global__ void __launch_bounds__(kGenBlock) k_generate(const __grid_constant__ RenderArgs a) {
  __shared__ uint32_t cnt[kGenBlock / 32], first;
  chain();
  const int64_t n = a.npaths;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if (a.dense && blockIdx.x == 0 && threadIdx.x == 0) a.counters[kCtrRay] = (uint32_t)n;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
    int64_t p = base + threadIdx.x;
    bool valid = p < n;
    bool live = false;
    float4 o4 = make_float4(0, 0, 0, 0), d4 = o4;
    if (valid) {
      const int j = job_of_path(a, p);
      const JobArgs &J = a.jobs[j];
      if (a.njobs > 1) a.path_job[p] = (uint32_t)j;
      int x, y, s;
      uint64_t pid = path_id(J, p, x, y, s);
      live = x < J.W && y < J.H;
      uint32_t flags = 0;
      if (live) {
        uint64_t pix = (uint64_t)y * J.W + x;
        int k = s % J.s2;
        F4u jt = uniforms(J.rng, pix * (uint64_t)J.s2 + (uint64_t)k, kDepthJitter, 0);
        float px = ((float)x + ((float)(k % J.side) + jt.a) / (float)J.side) / (float)J.W;
        float py = ((float)y + ((float)(k / J.side) + jt.b) / (float)J.side) / (float)J.H;
        F4u ui = uniforms(J.rng, pid, kDepthPathInit, 0);
        uint32_t ior = min((uint32_t)(ui.a * 3.0f), 2u);
        flags = ior;
        V3 o, d;
        camera_ray(J.cam, px, py, ui.b, ui.c, o, d);
        o4 = make_float4(o.x, o.y, o.z, __int_as_float((int)p));
        d4 = make_float4(d.x, d.y, d.z, __int_as_float(j));
      }
      a.path_L[p] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(flags));
    }
    uint32_t q = (uint32_t)p;
    if (!a.dense) {
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, live), lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
      if (lane == 0u) cnt[warp] = __popc(m);
      __syncthreads();
      uint32_t at = __popc(m & ((1u << lane) - 1u)), all = 0u;
      for (uint32_t w = 0; w < kGenBlock / 32; ++w) {
        if (w < warp) at += cnt[w];
        all += cnt[w];
      }
      if (threadIdx.x == 0) first = all ? atomicAdd(&a.counters[kCtrRay], all) : 0u;
      __syncthreads();
      q = first + at;
    }
    if (live) {
      a.qo[0][q] = o4;
      a.qd[0][q] = d4;
    }
  }
}

// extend: closest hit for the live queue of bounce b
// Traversal: the 8-wide hierarchy (hd_wide.h), or the kd-tree, one ray per lane, where no scene of a render has
// one and with mgpu_tune_set("wide", 0).
struct WideBlockShared {
  WideShared warp[kWideBlock / 32];
  WideTables tables;
  uint32_t next, next_extend;
};
constexpr int kWideSmem = (int)sizeof(WideBlockShared);

__device__ __forceinline__ WideBlockShared &wide_shared() {
  extern __shared__ __align__(16) unsigned char wide_smem[];
  WideBlockShared &s = *reinterpret_cast<WideBlockShared *>(wide_smem);
  wide_tables(s.tables);
  if (threadIdx.x == 0) s.next = s.next_extend = 0u;
  chain();
  __syncthreads();
  return s;
}

// closest hits of bounce b's rays, by the hierarchy
template <bool COUNT, bool SPH>
__device__ __forceinline__ void wide_extend(const RenderArgs &a, int b, WideBlockShared &ws, TraceCounts *c,
                                            uint32_t &rays) {
  const uint32_t n = a.counters[kCtrRay + b];
  const float4 *qo = a.qo[b & 1], *qd = a.qd[b & 1];
  float4 *qhit = a.qhit;
  auto view_of = [&](uint32_t i) -> const SceneView & { return a.jobs[__float_as_int(qd[i].w)].view; };
  auto view0 = [&](uint32_t) -> const SceneView & { return a.view0; };
  auto load = [&](uint32_t i, Ray &r) {
    float4 o = qo[i], d = qd[i];
    r.o = v3(o.x, o.y, o.z);
    r.tmin = 0.0f;
    r.d = v3(d.x, d.y, d.z);
    r.tmax = INFINITY;
  };
  auto store = [&](uint32_t i, bool hit, const Hit &h) {
    qhit[i] = make_float4(hit ? h.t : INFINITY, __int_as_float(hit ? h.prim : -1), hit ? h.b1 : 0.0f, hit ? h.b2 : 0.0f);
  };
  WideShared &sh = ws.warp[threadIdx.x >> 5];
  uint32_t *next = &ws.next_extend;
  if (a.njobs == 1)
    wide_trace<false, COUNT, SPH, true>(WideChunks(n), view0, n, load, store, sh, ws.tables, next, c, rays);
  else
    wide_trace<false, COUNT, SPH, false>(WideChunks(n), view_of, n, load, store, sh, ws.tables, next, c, rays);
}

// occlusion of bounce b's light samples, by the hierarchy; an occluded sample's slot is zeroed
template <bool COUNT, bool SPH>
__device__ __forceinline__ void wide_shadow(const RenderArgs &a, int b, WideBlockShared &ws, TraceCounts *c,
                                            uint32_t &rays) {
  const uint32_t n = a.counters[kCtrNee + b];
  const float4 *so = a.so, *sd = a.sd;
  float4 *slots = a.slots;
  auto view_of = [&](uint32_t i) -> const SceneView & {
    return a.jobs[a.path_job[__float_as_uint(so[i].w) / (uint32_t)a.nl_stride]].view;
  };
  auto view0 = [&](uint32_t) -> const SceneView & { return a.view0; };
  auto load = [&](uint32_t i, Ray &r) {
    float4 o = so[i], d = sd[i];
    r.o = v3(o.x, o.y, o.z);
    r.tmin = 0.0f;
    r.d = v3(d.x, d.y, d.z);
    r.tmax = d.w;
  };
  auto store = [&](uint32_t i, bool hit, const Hit &) {
    if (hit) slots[__float_as_uint(so[i].w)] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  };
  WideShared &sh = ws.warp[threadIdx.x >> 5];
  uint32_t *next = &ws.next;
  if (a.njobs == 1)
    wide_trace<true, COUNT, SPH, true>(WideChunks(n), view0, n, load, store, sh, ws.tables, next, c, rays);
  else
    wide_trace<true, COUNT, SPH, false>(WideChunks(n), view_of, n, load, store, sh, ws.tables, next, c, rays);
}

// Bounce b + 1's closest hits and bounce b's occlusion queries, which do not depend on each other: one launch,
// and one end at which warps wait for the block's last rays, instead of two of each.
template <bool SPH>
__global__ void __launch_bounds__(kWideBlock, 1) k_traverse(const __grid_constant__ RenderArgs a, int b) {
  TraceCounts c = {0, 0, 0, 0};
  uint32_t rays = 0;
  WideBlockShared &ws = wide_shared();
  wide_extend<false, SPH>(a, b + 1, ws, &c, rays);
  wide_shadow<false, SPH>(a, b, ws, &c, rays);
}

template <bool COUNT, bool WIDE, bool SPH>
__global__ void __launch_bounds__(WIDE ? kWideBlock : kBlock, WIDE ? 1 : kTravMinBlocks)
    k_extend(const __grid_constant__ RenderArgs a, int b) {
  TraceCounts c = {0, 0, 0, 0};
  uint32_t rays = 0;
  if constexpr (WIDE) {
    wide_extend<COUNT, SPH>(a, b, wide_shared(), &c, rays);
  } else {
    chain();
    const float4 *qo = a.qo[b & 1], *qd = a.qd[b & 1];
    float4 *qhit = a.qhit;
    auto view_of = [&](uint32_t i) -> const SceneView & { return a.jobs[__float_as_int(qd[i].w)].view; };
    auto load = [&](uint32_t i, Ray &r) {
      float4 o = qo[i], d = qd[i];
      r.o = v3(o.x, o.y, o.z);
      r.tmin = 0.0f;
      r.d = v3(d.x, d.y, d.z);
      r.tmax = INFINITY;
    };
    auto store = [&](uint32_t i, bool hit, const Hit &h) {
      qhit[i] = make_float4(hit ? h.t : INFINITY, __int_as_float(hit ? h.prim : -1), hit ? h.b1 : 0.0f, hit ? h.b2 : 0.0f);
    };
    kd_grid<false, COUNT, SPH>(view_of, a.counters[kCtrRay + b], load, store, &c, rays);
  }
  if (COUNT && rays + c.nodes + c.tris) {
    atomicAdd(&a.tcount[0], (unsigned long long)c.nodes);
    atomicAdd(&a.tcount[1], (unsigned long long)c.refs);
    atomicAdd(&a.tcount[2], (unsigned long long)c.tris);
    atomicAdd(&a.tcount[3], (unsigned long long)rays);
  }
}

// shade: pending direct light, emission, light sampling, BSDF sample and Russian roulette
// (PathTracer.cpp:36-115, DirectIllumination.cpp:46-138)
__device__ __forceinline__ V3 fold_slots(const RenderArgs &a, int nl, int64_t p, V3 L) {
  const float4 *sl = a.slots + p * a.nl_stride;
  for (int k = 0; k < nl; ++k) {
    float4 c = sl[k];
    L = L + v3(c.x, c.y, c.z);
  }
  return L;
}

// Threads of a shading block, and the rays that it takes at a time.
constexpr int kShadeTile = 256;
// Blocks of the shade kernels per SM: three leave a thread 80 registers and half the spills of 64.  Shading per
// frame at 3 / 4 / 2 blocks: mid scene 21.3 / 21.8 / 24.9 ms, plain box 0.302 / 0.332 / 0.327, terrain
// 3.18 / 3.30 / 3.47, textured 0.99 / 1.00 / 1.12.
constexpr int kShadeMinBlocks = 3;

// Light samples of a wave up to which its launches are chained, and traversals share them
constexpr int64_t kSmallWaveSlots = (int64_t)1 << 22;

// What a shading block keeps in shared memory: per warp the shadow rays that wait for a full 32 (or, while
// the block traces its own rays, the traversal's records), the counts and the order of the tile's
// rays, and the block's own queue counts.
struct ShadeShared {
  union {
    struct {
      float4 so[kShadeTile / 32][64], sd[kShadeTile / 32][64];
    } stage;
    WideShared wide[kShadeTile / 32];
  };
  WideTables tables;
  uint32_t cnt[kShadeTile / 4];
  uint32_t next, rays, shadow;
  uint8_t perm[kShadeTile];
  float held[9][kShadeTile];
};

// Position of the thread among the block's threads ordered by key (0..7).  cnt: 64 words that no thread
// still reads.
__device__ __forceinline__ uint32_t tile_rank(uint32_t *cnt, uint32_t key) {
  constexpr unsigned kFull = 0xFFFFFFFFu;
  static_assert(kShadeTile == 256, "eight warps");
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t mine = 0u, peers = 0u;
#pragma unroll
  for (uint32_t k = 0; k < 8u; ++k) {
    const uint32_t m = __ballot_sync(kFull, key == k);
    if (key == k) peers = m;
    if (lane == k) mine = __popc(m);
  }
  if (lane < 8u) cnt[8u * lane + warp] = mine;
  __syncthreads();
  // exclusive prefix sums of the 64 counts, two per lane, by every warp for itself
  const uint32_t x = cnt[2u * lane], y = cnt[2u * lane + 1u];
  uint32_t inc = x + y;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, inc, d);
    if (lane >= (uint32_t)d) inc += v;
  }
  const uint32_t at = 8u * key + warp;
  const uint32_t ex = __shfl_sync(kFull, inc - x - y, at >> 1), x0 = __shfl_sync(kFull, x, at >> 1);
  return ex + ((at & 1u) ? x0 : 0u) + __popc(peers & ((1u << lane) - 1u));
}

// A warp's shadow rays on their way to the queue: 32 at a time, one atomic and two coalesced stores (one
// atomic per warp and light sample was 20 M to one address on the mid frame).
struct ShadowStage {
  float4 *o, *d;       // ring of 64
  uint32_t *counter;
  float4 *so, *sd;
  uint32_t head, count;  // uniform over the warp
  __device__ __forceinline__ void write(uint32_t m) {
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();
    uint32_t at = 0u;
    if (lane == 0u) at = atomicAdd(counter, m);
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    if (lane < m) {
      so[at + lane] = o[(head + lane) & 63u];
      sd[at + lane] = d[(head + lane) & 63u];
    }
    __syncwarp();
    head = (head + m) & 63u;
    count -= m;
  }
  __device__ __forceinline__ void append(bool want, float4 o4, float4 d4) {
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, want);
    if (want) {
      const uint32_t e = (head + count + __popc(m & ((1u << (threadIdx.x & 31u)) - 1u))) & 63u;
      o[e] = o4;
      d[e] = d4;
    }
    count += __popc(m);
    if (count >= 32u) write(32u);
  }
  __device__ __forceinline__ void flush() {
    if (count) write(count);
  }
};

// One block's closest hits of rays base .. n - 1 of bounce b, and its shadow rays (whole paths, k_shade).
template <bool SPH>
__device__ __noinline__ void block_extend(const RenderArgs &a, ShadeShared &sh, int b, uint32_t base, uint32_t n) {
  const float4 *qo = a.qo[b & 1] + base, *qd = a.qd[b & 1] + base;
  uint32_t done = 0u;
  wide_trace<false, false, SPH, false>(
      WideAll(), [&](uint32_t i) -> const SceneView & { return a.jobs[__float_as_int(qd[i].w)].view; }, n - base,
      [&](uint32_t i, Ray &r) {
        const float4 o = qo[i], d = qd[i];
        r.o = v3(o.x, o.y, o.z);
        r.tmin = 0.0f;
        r.d = v3(d.x, d.y, d.z);
        r.tmax = INFINITY;
      },
      [&](uint32_t i, bool hit, const Hit &h) {
        a.qhit[base + i] = make_float4(hit ? h.t : INFINITY, __int_as_float(hit ? h.prim : -1), hit ? h.b1 : 0.0f,
                                       hit ? h.b2 : 0.0f);
      },
      sh.wide[threadIdx.x >> 5], sh.tables, &sh.next, nullptr, done);
}

template <bool SPH>
__device__ __noinline__ void block_shadow(const RenderArgs &a, ShadeShared &sh, const float4 *so, const float4 *sd,
                                          uint32_t n) {
  uint32_t done = 0u;
  wide_trace<true, false, SPH, false>(
      WideAll(),
      [&](uint32_t i) -> const SceneView & {
        return a.njobs == 1 ? a.jobs[0].view : a.jobs[a.path_job[__float_as_uint(so[i].w) / (uint32_t)a.nl_stride]].view;
      },
      n,
      [&](uint32_t i, Ray &r) {
        const float4 o = so[i], d = sd[i];
        r.o = v3(o.x, o.y, o.z);
        r.tmin = 0.0f;
        r.d = v3(d.x, d.y, d.z);
        r.tmax = d.w;
      },
      [&](uint32_t i, bool hit, const Hit &) {
        if (hit) a.slots[__float_as_uint(so[i].w)] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      },
      sh.wide[threadIdx.x >> 5], sh.tables, &sh.next, nullptr, done);
}

// SURF: the wave has a scene with image maps, a background or analytic spheres.  Scenes without
// them run the variant that has none of those branches, whose register allocation (and spilling)
// is the lighter.
//
// WHOLE: the launch takes whole paths instead of one bounce (waves of few paths).  Every block owns `whole` (at
// most 256) rays of bounce b and runs their bounces to the end: it traces its rays, shades them, traces
// their shadow rays, and keeps the queues in its own part of the arrays.  One launch instead of three per
// bounce, and blocks whose paths have ended do not wait for others.  Both variants come from this one
// text, with the traversal called and not inlined, so that the shading's multiply-adds contract alike in
// them and an image does not depend on the wave size (tests/test_gpu_wide.py compares the bits).
template <bool SURF, bool WHOLE>
__global__ void __launch_bounds__(kShadeTile, kShadeMinBlocks) k_shade(const __grid_constant__ RenderArgs a, int b,
                                                                       uint32_t whole) {
  extern __shared__ __align__(16) unsigned char shade_smem[];
  ShadeShared &sh = *reinterpret_cast<ShadeShared *>(shade_smem);
  if (WHOLE) wide_tables(sh.tables);
  chain();
  uint32_t n = a.counters[kCtrRay + b], base = blockIdx.x * kShadeTile;
  const uint32_t stride = gridDim.x * kShadeTile, total = n;
  const int b0 = b;
  const uint32_t warp = threadIdx.x >> 5;
  uint32_t out = 0u;  // first entry of the queues that the block writes
  uint32_t *next_ctr = &a.counters[kCtrRay + b + 1];
  ShadowStage stage{sh.stage.so[warp], sh.stage.sd[warp], &a.counters[kCtrNee + b], a.so, a.sd, 0u, 0u};
  if (WHOLE) {
    base = blockIdx.x * whole;
    if (base >= total) return;
    out = base;
    n = min(base + whole, total);
    next_ctr = &sh.rays;
    stage.counter = &sh.shadow;
    stage.so = a.so + (size_t)base * a.nl_stride;
    stage.sd = a.sd + (size_t)base * a.nl_stride;
  }
  for (;;) {
    if (base >= n) break;
    const int cur = b & 1, nxt = (b + 1) & 1;
    if (WHOLE) {
      if (threadIdx.x == 0) sh.next = sh.rays = sh.shadow = 0u;
      __syncthreads();
      block_extend<SURF>(a, sh, b, base, n);
      __syncthreads();
    }
    // the tile's rays in the order of what they hit: with the BSDFs of a tile side by side a warp runs one of
    // them, and the barriers keep the block's warps in the same part of a kernel that exceeds the
    // instruction cache (ncu, mid scene, second bounce: lanes per instruction 13.7 -> 24.9, warps waiting
    // for instructions 9.6 -> 0.7 per issue; 30.7 -> 24.5 ms of the mid frame.  Sorted by warps of 128 rays,
    // without barriers: 28.7)
    uint32_t i = base + threadIdx.x;
    if (a.sort_hits) {
      uint32_t cls = 4u;
      if (i < n) {
        const int prim = __float_as_int(a.qhit[i].y);
        cls = 3u;
        if (prim >= 0) {
          const JobArgs &J = a.jobs[__float_as_int(a.qd[cur][i].w)];
          const int mi = __float_as_int(__ldg(J.shade + 3 * (int64_t)prim).w);
          cls = min((uint32_t)__ldg(J.mats + 4 * mi).x, 2u);
        }
      }
      sh.perm[tile_rank(sh.cnt, cls)] = (uint8_t)threadIdx.x;
      __syncthreads();
      i = base + sh.perm[threadIdx.x];
    }
    const bool valid = i < n;
    bool want_next = false, do_nee = false;
    float4 no_o, no_d, no_t;
    int64_t p = 0;
    uint64_t pid = 0;
    int depth = 0, self = -1, j = 0;
    V3 P = v3(0, 0, 0), ns = P, ng = P, d = P, thr = P;
    Material m;
    m.type = 0;
    if (valid) {
      float4 o4 = a.qo[cur][i], d4 = a.qd[cur][i], h4 = a.qhit[i];
      // a first vertex: throughput 1, depth 0 (k_generate writes none)
      const float4 t4 = b == 0 ? make_float4(1.0f, 1.0f, 1.0f, 0.0f) : a.qt[cur][i];
      p = (int64_t)__float_as_int(o4.w);
      j = __float_as_int(d4.w);
      const JobArgs &J = a.jobs[j];
      uint32_t state = __float_as_uint(t4.w);
      depth = (int)(state & 0xFFFFu);
      bool ec = (state >> 16) & 1u;
      thr = v3(t4.x, t4.y, t4.z);
      d = v3(d4.x, d4.y, d4.z);
      int prim = __float_as_int(h4.y);
      float4 L4 = a.path_L[p];
      uint32_t flags = __float_as_uint(L4.w);
      V3 L = v3(L4.x, L4.y, L4.z);
      if (flags & kFlagNeePending) {
        L = fold_slots(a, J.nl_slots, p, L);
        flags &= ~kFlagNeePending;
      }
      if (prim >= 0) {
        int x, y, s;
        pid = path_id(J, p, x, y, s);
        float t = h4.x, b1 = h4.z, b2 = h4.w, b0 = 1.0f - b1 - b2;
        float4 s0 = __ldg(J.shade + 3 * (int64_t)prim), s1 = __ldg(J.shade + 3 * (int64_t)prim + 1);
        if (SURF && prim >= J.view.ntri) {
          // analytic sphere: the hit on the ray, the radial normal (Sphere::_getGeometricNormal)
          const float4 c = __ldg(reinterpret_cast<const float4 *>(J.view.spheres) + 2 * (prim - J.view.ntri));
          P = v3(o4.x, o4.y, o4.z) + d * t;
          ns = normalize(P - v3(c.x, c.y, c.z));
          ng = ns;
        } else {
          float4 va = __ldg(reinterpret_cast<const float4 *>(J.view.tris) + 3 * (int64_t)prim);
          float4 vb = __ldg(reinterpret_cast<const float4 *>(J.view.tris) + 3 * (int64_t)prim + 1);
          float4 vc = __ldg(reinterpret_cast<const float4 *>(J.view.tris) + 3 * (int64_t)prim + 2);
          float4 s2 = __ldg(J.shade + 3 * (int64_t)prim + 2);
          V3 v0 = v3(va.x, va.y, va.z), v1 = v3(vb.x, vb.y, vb.z), v2 = v3(vc.x, vc.y, vc.z);
          P = v0 * b0 + v1 * b1 + v2 * b2;
          ns = normalize(v3(s0.x, s0.y, s0.z) * b0 + v3(s1.x, s1.y, s1.z) * b1 + v3(s2.x, s2.y, s2.z) * b2);
          ng = normalize(cross(v1 - v0, v2 - v0));
        }
        int mi = __float_as_int(s0.w);
        self = __float_as_int(s1.w);
        m = load_mat(J, mi, flags & kFlagIorMask);
        if (SURF && (m.tex_kd | m.tex_ks | m.tex_tr | m.tex_bump) != 0) apply_textures(J, prim, b0, b1, b2, P, m, ns);
        bool spec = is_specular(m);
        if (spec) flags |= kFlagSpecular;
        if (self >= 0) {
          Light lt = load_light(J, self);
          V3 Le = light_le(lt, ns, -d);
          if (!J.efficient || depth == 0) L = L + mul(thr, Le);
          else if (ec) L = L + mul(thr, Le) * (lt.area / (t * t));
        }
        if (J.efficient && !spec && J.nlight > 0) {
          do_nee = true;
          flags |= kFlagNeePending;
        }
        F4u u = uniforms(J.rng, pid, (uint32_t)depth, 0);
        V3 wo, fs;
        int ev = bsdf_sample(m, ns, d, flags & kFlagIorMask, u.a, u.b, u.c, wo, fs);
        if (ev > 0) {
          float pc = depth < J.rr_start ? (nonzero(fs) ? 1.0f : 0.0f) : fminf(0.95f, maxc(fs));
          bool capped = (J.max_depth > 0 && depth + 1 >= J.max_depth);
          if (!capped && u.d < pc) {
            if (depth + 1 >= kHardCap) {
              flags |= kFlagTruncated;
              atomicAdd(&a.counters[kCtrTrunc], 1u);
            } else {
              want_next = true;
              if (depth == 0) flags |= kFlagContinued0;
              V3 nthr = mul(thr, fs) * rcp(pc);
              bool nec = spec && dot(ns, wo) > kEps;
              V3 org = offset_origin(P, dot(ng, wo) > 0.0f ? ng : -ng);
              no_o = make_float4(org.x, org.y, org.z, o4.w);
              no_d = make_float4(wo.x, wo.y, wo.z, d4.w);
              no_t = make_float4(nthr.x, nthr.y, nthr.z, __uint_as_float((uint32_t)(depth + 1) | (nec ? 0x10000u : 0u)));
            }
          }
        }
      } else if (SURF && (J.bg_tex != 0 || J.bg_le[0] != 0.0f || J.bg_le[1] != 0.0f || J.bg_le[2] != 0.0f)) {
        L = L + mul(thr, background(J, d));  // PathTracer.cpp:39-42: a miss adds the background
      }
      a.path_L[p] = make_float4(L.x, L.y, L.z, __uint_as_float(flags));
    }
    const JobArgs &J = a.jobs[j];
    const uint32_t q = out + warp_append(next_ctr, want_next);
    if (want_next) {
      if (a.bin_ext) {
        a.qo_u[q] = no_o;
        a.qd_u[q] = no_d;
        a.qt_u[q] = no_t;
        a.qkey[q] = ext_key(J, v3(no_o.x, no_o.y, no_o.z), v3(no_d.x, no_d.y, no_d.z));
      } else {
        a.qo[nxt][q] = no_o;
        a.qd[nxt][q] = no_d;
        a.qt[nxt][q] = no_t;
      }
    }
    // What the light samples need now and then waits in shared memory, not in registers that spill (textured
    // frame, shading 1.007 -> 0.979 ms; plain box and mid scene within 1 %).  Read back through `held`, which
    // the compiler may not keep in registers.
    volatile float(*held)[kShadeTile] = sh.held;
    held[0][threadIdx.x] = ng.x; held[1][threadIdx.x] = ng.y; held[2][threadIdx.x] = ng.z;
    held[3][threadIdx.x] = thr.x; held[4][threadIdx.x] = thr.y; held[5][threadIdx.x] = thr.z;
    held[6][threadIdx.x] = d.x; held[7][threadIdx.x] = d.y; held[8][threadIdx.x] = d.z;
    auto hold = [&](int k) { return v3(held[k][threadIdx.x], held[k + 1][threadIdx.x], held[k + 2][threadIdx.x]); };
    // light samples: every lane of the warp runs the same k loop (uniform trip count: the
    // wave's stride), so the warp-aggregated append stays converged
    const int s2n = J.nds_side * J.nds_side;
    const float inv_nds = rcp((float)J.nds);
    F4u u = {0.0f, 0.0f, 0.0f, 0.0f};  // light samples 2m and 2m + 1 share counter block 1 + m
    for (int k = 0; k < a.nl_stride; ++k) {
      bool want = false;
      float4 so4, sd4;
      if (do_nee && k < J.nl_slots) {
        int li = k / s2n, within = k - li * s2n;
        int sy = within / J.nds_side, sx = within - sy * J.nds_side;
        V3 c = v3(0.0f, 0.0f, 0.0f);
        Light lt = load_light(J, li);
        if ((k & 1) == 0) u = uniforms(J.rng, pid, (uint32_t)depth, 1u + (uint32_t)(k >> 1));
        // a point light takes one sample (DirectIllumination.cpp:97-99): the first stratum
        if (li != self && (lt.type != kLightPoint || within == 0)) {
          float ux = (float)sx + ((k & 1) ? u.c : u.a), uy = (float)sy + ((k & 1) ? u.d : u.b);
          if (J.nds_side != 1) {  // x / 1 = x: one light sample per light needs no division
            ux = ux / (float)J.nds_side;
            uy = uy / (float)J.nds_side;
          }
          float r1 = 0.0f, r2 = 0.0f;
          if (lt.type == kLightMesh) {
            F4u um = uniforms(J.rng, pid, (uint32_t)depth, kMeshLightBlock + (uint32_t)k);
            r1 = um.a;
            r2 = um.b;
          }
          V3 lp, ln, lg;
          light_point(
              lt, ux, uy, r1, r2,
              [&](uint32_t t, int c) {
                const float4 q = __ldg(reinterpret_cast<const float4 *>(J.view.tris) + 3 * (int64_t)t + c);
                return v3(q.x, q.y, q.z);
              },
              [&](uint32_t t, int c) {
                const float4 q = __ldg(J.shade + 3 * (int64_t)t + c);
                return v3(q.x, q.y, q.z);
              },
              lp, ln, lg);
          V3 wo = lp - P;
          float t = length(wo);
          wo = wo * rcp(t);
          const bool point = lt.type == kLightPoint;
          float cwo = fabsf(dot(ns, wo)), cwi = point ? 1.0f : fabsf(dot(ln, wo));
          V3 fr = bsdf_eval(m, ns, hold(6), wo);
          if (cwo > 0.0f && cwi > 0.0f && nonzero(fr)) {
            V3 Le = light_le(lt, ln, -wo);
            // area / samples for an area light, 1 for a point (DirectIllumination.cpp:127-128)
            c = mul(hold(3), mul(fr, Le)) * (cwo * cwi / (t * t) * (point ? 1.0f : lt.area * inv_nds));
            if (nonzero(c)) {
              want = true;
              const V3 g = hold(0);
              // both ends of the shadow segment are moved off their surfaces toward each other
              // (Wachter and Binder), so that neither the shading point's nor the light's own
              // surface can occlude it, however grazing the direction
              V3 org = offset_origin(P, dot(g, wo) > 0.0f ? g : -g);
              V3 tgt = offset_origin(lp, dot(lg, wo) < 0.0f ? lg : -lg);
              V3 sdir = tgt - org;
              const float sl = length(sdir);
              sdir = sdir * rcp(sl);
              so4 = make_float4(org.x, org.y, org.z, __uint_as_float((uint32_t)(p * a.nl_stride + k)));
              sd4 = make_float4(sdir.x, sdir.y, sdir.z, sl);
            }
          }
        }
        a.slots[p * a.nl_stride + k] = make_float4(c.x, c.y, c.z, 0.0f);
      }
      stage.append(want, so4, sd4);
    }
    if (!WHOLE) {
      base += stride;
      continue;
    }
    stage.flush();
    __syncthreads();
    const uint32_t nshadow = sh.shadow, nrays = sh.rays;
    __syncthreads();
    if (threadIdx.x == 0) sh.next = 0u;
    __syncthreads();
    block_shadow<SURF>(a, sh, stage.so, stage.sd, nshadow);
    __syncthreads();
    if (threadIdx.x == 0) {
      if (b > b0) atomicAdd(&a.counters[kCtrRay + b], n - base);
      atomicAdd(&a.counters[kCtrNee + b], nshadow);
    }
    n = base + nrays;
    ++b;
    if (b >= a.max_b) n = base;
  }
  if (!WHOLE) stage.flush();
}


// shadow: any-hit query per queued light sample; an occluded sample's slot is zeroed
template <bool COUNT, bool WIDE, bool SPH>
__global__ void __launch_bounds__(WIDE ? kWideBlock : kBlock, WIDE ? 1 : kTravMinBlocks)
    k_shadow(const __grid_constant__ RenderArgs a, int b) {
  TraceCounts c = {0, 0, 0, 0};
  uint32_t rays = 0;
  if constexpr (WIDE) {
    wide_shadow<COUNT, SPH>(a, b, wide_shared(), &c, rays);
  } else {
    chain();
    const float4 *so = a.so, *sd = a.sd;
    float4 *slots = a.slots;
    auto view_of = [&](uint32_t i) -> const SceneView & {
      if (a.njobs == 1) return a.jobs[0].view;
      return a.jobs[a.path_job[__float_as_uint(so[i].w) / (uint32_t)a.nl_stride]].view;
    };
    auto load = [&](uint32_t i, Ray &r) {
      float4 o = so[i], d = sd[i];
      r.o = v3(o.x, o.y, o.z);
      r.tmin = 0.0f;
      r.d = v3(d.x, d.y, d.z);
      r.tmax = d.w;
    };
    auto store = [&](uint32_t i, bool hit, const Hit &) {
      if (hit) slots[__float_as_uint(so[i].w)] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    kd_grid<true, COUNT, SPH>(view_of, a.counters[kCtrNee + b], load, store, &c, rays);
  }
  if (COUNT && rays + c.nodes + c.tris) {
    atomicAdd(&a.tcount[4], (unsigned long long)c.nodes);
    atomicAdd(&a.tcount[5], (unsigned long long)c.refs);
    atomicAdd(&a.tcount[6], (unsigned long long)c.tris);
    atomicAdd(&a.tcount[7], (unsigned long long)rays);
  }
}

// ---------------------------------------------------------------------------------------
// counting sort of a queue by key: histogram -> exclusive scan -> scatter with per-block
// range reservations (one global atomic per block chunk and non-empty bin)
__global__ void __launch_bounds__(256) k_bin_hist(const uint32_t *__restrict__ keys, const uint32_t *count,
                                                 uint32_t *__restrict__ hist) {
  extern __shared__ uint32_t h[];  // kBins
  for (int i = threadIdx.x; i < kBins; i += blockDim.x) h[i] = 0;
  __syncthreads();
  const uint32_t n = *count;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    atomicAdd(&h[keys[i] & (kBins - 1)], 1u);
  __syncthreads();
  for (int i = threadIdx.x; i < kBins; i += blockDim.x)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

// single block of 1024 threads: hist -> cursor (exclusive prefix sum)
__global__ void __launch_bounds__(1024) k_bin_scan(const uint32_t *__restrict__ hist, uint32_t *__restrict__ cursor) {
  __shared__ uint32_t part[1024];
  const int per = kBins / 1024;
  uint32_t loc[kBins / 1024];
  uint32_t sum = 0;
  for (int k = 0; k < per; ++k) {
    loc[k] = sum;
    sum += hist[threadIdx.x * per + k];
  }
  part[threadIdx.x] = sum;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    uint32_t v = threadIdx.x >= (unsigned)off ? part[threadIdx.x - off] : 0u;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  uint32_t base = threadIdx.x ? part[threadIdx.x - 1] : 0u;
  for (int k = 0; k < per; ++k) cursor[threadIdx.x * per + k] = base + loc[k];
}

__global__ void __launch_bounds__(256) k_bin_scatter(const uint32_t *__restrict__ keys, const uint32_t *count,
                                                    uint32_t *__restrict__ cursor, const float4 *__restrict__ in0,
                                                    const float4 *__restrict__ in1, const float4 *__restrict__ in2,
                                                    float4 *__restrict__ out0, float4 *__restrict__ out1,
                                                    float4 *__restrict__ out2) {
  constexpr int kPer = 32;                 // entries per thread per chunk
  constexpr int kChunk = 256 * kPer;
  extern __shared__ uint32_t h[];  // kBins
  const uint32_t n = *count;
  for (uint32_t c0 = blockIdx.x * kChunk; c0 < n; c0 += gridDim.x * kChunk) {
    for (int i = threadIdx.x; i < kBins; i += blockDim.x) h[i] = 0;
    __syncthreads();
    uint32_t key[kPer], rank[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      uint32_t i = c0 + k * 256 + threadIdx.x;
      key[k] = i < n ? (keys[i] & (kBins - 1)) : 0u;
      rank[k] = i < n ? atomicAdd(&h[key[k]], 1u) : 0u;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kBins; i += blockDim.x)
      if (h[i]) h[i] = atomicAdd(&cursor[i], h[i]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      uint32_t i = c0 + k * 256 + threadIdx.x;
      if (i < n) {
        uint32_t pos = h[key[k]] + rank[k];
        out0[pos] = in0[i];
        out1[pos] = in1[i];
        out2[pos] = in2[i];
      }
    }
    __syncthreads();
  }
}

// accumulate: per pixel, Kahan-add the wave's samples into the compensated FP32 film
// (ProgressiveFilterValue::addSample, ProgressiveFilterValue.h:33-36, box weight 1)
// Reconstruction splat of one sample (ReconstructionRenderOutput::addSample,
// ReconstructionRenderOutput.cpp:30-83): the sample's film position is regenerated from its
// jitter (as k_generate draws it) and its radiance is added, weighted, to every pixel within the
// filter's half width whose weight is positive.  Fixed point 2^-24 makes the sums independent of
// the order of the atomic additions; non-finite or oversized contributions are dropped.
__device__ void splat(const JobArgs &J, int x, int y, int s, V3 L) {
  const int k = s % J.s2;
  const uint64_t pix = (uint64_t)y * J.W + x;
  const F4u jt = uniforms(J.rng, pix * (uint64_t)J.s2 + (uint64_t)k, kDepthJitter, 0);
  const float px = ((float)x + ((float)(k % J.side) + jt.a) / (float)J.side) / (float)J.W;
  const float py = ((float)y + ((float)(k / J.side) + jt.b) / (float)J.side) / (float)J.H;
  const float cx = px * (float)J.W, cy = py * (float)J.H;
  const int h = J.filt.half;
  const int y0 = max(0, y - h), y1 = min(J.H - 1, y + h), x0 = max(0, x - h), x1 = min(J.W - 1, x + h);
  const float scale = 16777216.0f;  // 2^24
  for (int yy = y0; yy <= y1; ++yy)
    for (int xx = x0; xx <= x1; ++xx) {
      const float w = filter_eval(J.filt, (float)xx - cx, (float)yy - cy);
      if (!(w > 0.0f)) continue;
      const float v[4] = {w * L.x * scale, w * L.y * scale, w * L.z * scale, w * scale};
      if (!(v[0] < 1e18f && v[1] < 1e18f && v[2] < 1e18f && v[3] < 1e18f)) continue;
      unsigned long long *dst = J.film_fx + 4 * ((int64_t)yy * J.W + xx);
#pragma unroll
      for (int c = 0; c < 4; ++c) atomicAdd(dst + c, (unsigned long long)llrintf(v[c]));
    }
}

__global__ void __launch_bounds__(kBlock) k_accumulate(const __grid_constant__ RenderArgs a) {
  chain();
  // the wave's counts, by one warp (one thread took 43 us over the 1,024 bounces of a wave without a depth cap:
  // analytic spheres, 1.08 M paths, 65 -> 22 us)
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    unsigned long long ext = 0, bounces = 0, sh = 0;
    for (int b = threadIdx.x; b < a.max_b; b += 32) {
      uint32_t c = a.counters[kCtrRay + b];
      ext += c;
      bounces += c ? 1ull : 0ull;
      sh += a.counters[kCtrNee + b];
    }
    for (int d = 16; d > 0; d >>= 1) {
      ext += __shfl_xor_sync(0xFFFFFFFFu, ext, d);
      sh += __shfl_xor_sync(0xFFFFFFFFu, sh, d);
      bounces += __shfl_xor_sync(0xFFFFFFFFu, bounces, d);
    }
    if (threadIdx.x == 0) {
      a.stats[0] += ext;
      a.stats[1] += sh;
      a.stats[2] += a.counters[kCtrTrunc];
      a.stats[3] += bounces;
    }
  }
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < a.nslots; q += stride) {
    const JobArgs &J = a.jobs[job_of_slot(a, q)];
    const int64_t lq = q - J.slot_base;
    int x, y;
    if (!slot_pixel(J, J.slot0 + lq, x, y)) continue;
    int64_t pix = (int64_t)y * J.W + x;
    float4 S = J.film_sum[pix], C = J.film_c[pix];
    for (int si = 0; si < J.ns; ++si) {
      const int64_t p = J.path_base + lq * J.ns + si;
      float4 L4 = a.path_L[p];
      V3 L = v3(L4.x, L4.y, L4.z);
      if (__float_as_uint(L4.w) & kFlagNeePending) L = fold_slots(a, J.nl_slots, p, L);
      L = apply_mask(L, __float_as_uint(L4.w));
      if (J.path_out) {
        int s = J.s0 + si - J.sample_begin;
        J.path_out[pix * J.sample_count + s] = make_float4(L.x, L.y, L.z, L4.w);
      }
      float yx = L.x - C.x, tx = S.x + yx; C.x = (tx - S.x) - yx; S.x = tx;
      float yy = L.y - C.y, ty = S.y + yy; C.y = (ty - S.y) - yy; S.y = ty;
      float yz = L.z - C.z, tz = S.z + yz; C.z = (tz - S.z) - yz; S.z = tz;
      // second moment of the per-sample luminance (variance / error estimates), unfused
      const float lum = __fmul_rn(__fadd_rn(__fadd_rn(L.x, L.y), L.z), 1.0f / 3.0f);
      C.w = __fadd_rn(C.w, __fmul_rn(lum, lum));
      if (J.film_fx) splat(J, x, y, J.s0 + si, L);
    }
    S.w += (float)J.ns;
    J.film_sum[pix] = S;
    J.film_c[pix] = C;
  }
}

// ---------------------------------------------------------------------------------------
// host driver

struct Workspace {
  int device = -1;
  int64_t cap = 0;       // paths
  int64_t slot_cap = 0;  // light-sample slots
  int64_t job_cap = 0;   // JobArgs entries
  void *block = nullptr;
  float4 *path_L = nullptr, *qo[2] = {}, *qd[2] = {}, *qt[2] = {}, *qhit = nullptr;
  float4 *so = nullptr, *sd = nullptr, *slots = nullptr;
  float4 *qo_u = nullptr, *qd_u = nullptr, *qt_u = nullptr;
  uint32_t *qkey = nullptr, *hist = nullptr, *cursor = nullptr;  // hist/cursor: kBins each
  uint32_t *path_job = nullptr;
  JobArgs *jobs = nullptr;
  uint32_t *counters = nullptr;
  unsigned long long *stats = nullptr;   // 4
  unsigned long long *tcount = nullptr;  // 8
  uint32_t *h_counters = nullptr;  // pinned (owned) or a static host word (allocation-free path)
  bool owned = true;
  ~Workspace() {
    if (!owned) return;
    if (block) cudaFree(block);
    if (h_counters) cudaFreeHost(h_counters);
  }
};

constexpr int kCarveoutAuto = -2;

// process-wide tuning knobs (mgpu_tune_set)
struct Tuning {
  // the 8-wide hierarchy where every scene of a render has one; 0: the kd-tree
  std::atomic<int> wide{1};
  // waves of at most this many paths run whole paths in one launch (0: none do; -1: what is resident at once)
  std::atomic<int64_t> whole_paths{-1};
  // shapes of kd-tree kernels that are no more: kept for callers that set and read them back
  std::atomic<int> persistent{0}, coop_leaf{3}, trav_block{256};
  std::atomic<int> bin_extension{1};  // counting-sort extension rays by (octant, origin cell)
  // waves of fewer paths, and scenes of fewer than kBinMinTris triangles, skip the sort: it pays where
  // tree and triangles are well beyond the L1s (64 M paths, sorted against not: 2 M triangles 318.5 / 326.5 ms,
  // 1 M 103.8 / 107.4, 300 k 70.3 / 71.2; with 8-bit nodes 150 k 60.2 / 60.1, 50 k 31.8 / 30.8, 36 triangles
  // 68.9 / 57.3; 16 M paths of 2 M 82.0 / 83.6, 1 M 27.7 / 27.9, 300 k 18.8 / 18.6).  0: sort every wave.
  std::atomic<int64_t> bin_min_paths{(int64_t)1 << 25};
  // a sort of the shadow rays cost more than it saved and is no more (1 M triangles, 64 M paths: 6.1 ms of sorting
  // and key writes for 3.5 of traversal); kept for callers that set and read it back
  std::atomic<int> bin_shadow{1};
  // shared-memory carveout (%) of the traversal / shade kernels: -2 = per kernel, the least that
  // keeps its resident blocks (the rest of the SM's 256 KB is L1); -1 = the driver's choice
  std::atomic<int> carveout{kCarveoutAuto};
};
static Tuning g_tune;

static thread_local Workspace *t_ws = nullptr;
static thread_local mgpu_render_stats t_stats{};
static thread_local cudaStream_t t_stats_stream = nullptr;
static thread_local bool t_stats_pending = false;
static thread_local unsigned long long *t_stats_dev = nullptr;  // device stats of the last render
static thread_local uint32_t *t_counters_dev = nullptr;          // queue counters of its last wave

// Per-kernel timing with CUDA events recorded on the launching stream around every launch.
enum { kProfGenerate = 0, kProfExtend, kProfShade, kProfShadow, kProfAccumulate, kProfBin, kProfClasses };
struct Profiler {
  bool enabled = false;
  std::vector<cudaEvent_t> pool;
  size_t used = 0;
  std::vector<std::pair<int, size_t>> marks;  // (class, index of begin event); end = begin + 1
  cudaStream_t stream = nullptr;
  double ms[kProfClasses] = {0, 0, 0, 0, 0, 0};
  uint64_t launches[kProfClasses] = {0, 0, 0, 0, 0, 0};
  cudaEvent_t next() {
    if (used == pool.size()) {
      cudaEvent_t e;
      cudaEventCreate(&e);
      pool.push_back(e);
    }
    return pool[used++];
  }
  int begin(int cls, cudaStream_t st) {
    if (!enabled) return -1;
    stream = st;
    size_t i = used;
    cudaEventRecord(next(), st);
    next();
    marks.push_back({cls, i});
    return (int)marks.size() - 1;
  }
  void end(int mark, cudaStream_t st) {
    if (mark < 0) return;
    cudaEventRecord(pool[marks[(size_t)mark].second + 1], st);
  }
  int flush() {
    if (marks.empty()) return MGPU_OK;
    MGPU_CUDA(cudaStreamSynchronize(stream));
    for (auto &m : marks) {
      float t = 0;
      MGPU_CUDA(cudaEventElapsedTime(&t, pool[m.second], pool[m.second + 1]));
      ms[m.first] += t;
      launches[m.first] += 1;
    }
    marks.clear();
    used = 0;
    return MGPU_OK;
  }
};
static thread_local Profiler t_prof;

// float4 arrays: path_L, 2 x (qo, qd, qt), qhit, unsorted (qo, qd, qt) = 11 per path;
// so, sd, slots = 3 per light sample; a uint32 key and path_job per path; JobArgs entries
static size_t workspace_bytes(int64_t paths, int64_t slots, int64_t jobs) {
  size_t f4 = (size_t)paths * 11 + (size_t)slots * 3;
  size_t u32 = (size_t)paths * 2 + 2 * kBins + kNumCounters;
  return f4 * sizeof(float4) + (size_t)jobs * sizeof(JobArgs) + 12 * sizeof(unsigned long long) +
         u32 * sizeof(uint32_t) + 1024;
}

static void workspace_layout(Workspace *w, void *block, int64_t paths, int64_t slots, int64_t jobs) {
  w->cap = paths;
  w->slot_cap = slots;
  w->job_cap = jobs;
  w->block = block;
  float4 *f = (float4 *)block;
  w->path_L = f; f += paths;
  for (int k = 0; k < 2; ++k) { w->qo[k] = f; f += paths; w->qd[k] = f; f += paths; w->qt[k] = f; f += paths; }
  w->qhit = f; f += paths;
  w->qo_u = f; f += paths; w->qd_u = f; f += paths; w->qt_u = f; f += paths;
  w->so = f; f += slots; w->sd = f; f += slots; w->slots = f; f += slots;
  w->jobs = (JobArgs *)f;  // JobArgs is a multiple of 8 bytes; float4 alignment holds
  w->stats = (unsigned long long *)(w->jobs + jobs);
  w->tcount = w->stats + 4;
  uint32_t *u = (uint32_t *)(w->tcount + 8);
  w->qkey = u; u += paths;
  w->path_job = u; u += paths;
  w->hist = u; u += kBins;
  w->cursor = u; u += kBins;
  w->counters = u;
}

static int ensure_workspace(int64_t paths, int64_t slots, int64_t jobs) {
  int dev = 0;
  MGPU_CUDA(cudaGetDevice(&dev));
  if (t_ws && t_ws->device == dev && t_ws->cap >= paths && t_ws->slot_cap >= slots && t_ws->job_cap >= jobs)
    return MGPU_OK;
  if (t_ws) {
    paths = std::max(paths, t_ws->cap);
    slots = std::max(slots, t_ws->slot_cap);
    jobs = std::max(jobs, t_ws->job_cap);
    cudaDeviceSynchronize();
    delete t_ws;
    t_ws = nullptr;
  }
  Workspace *w = new Workspace();
  w->device = dev;
  void *block = nullptr;
  cudaError_t e = cudaMalloc(&block, workspace_bytes(paths, slots, jobs));
  if (e != cudaSuccess) {
    delete w;
    return cuda_fail(e, "render workspace cudaMalloc");
  }
  workspace_layout(w, block, paths, slots, jobs);
  e = cudaMallocHost(&w->h_counters, 64);
  if (e != cudaSuccess) {
    delete w;
    return cuda_fail(e, "render workspace cudaMallocHost");
  }
  t_ws = w;
  return MGPU_OK;
}

// ---------------------------------------------------------------------------------------
// Fixed scratch for mgpu_render_noalloc: one static device array per process and device,
// resident from module load until exit.  Host code only holds a stand-in for the array's
// name; the device address comes from cudaGetSymbolAddress, once per device.
constexpr size_t kNoAllocBytes = (size_t)32 << 20;  // 32 MiB
constexpr int64_t kNoAllocJobs = 256;              // chunk descriptors kept in the scratch
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];
constexpr int kNoAllocMaxDevices = 64;
static std::mutex g_noalloc_mu;
static void *g_noalloc_ptr[kNoAllocMaxDevices];
static uint32_t g_noalloc_host_counter[16];  // pageable host word for live-path counts

static int noalloc_scratch(void **out) {
  int dev = 0;
  MGPU_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(MGPU_E_INVALID, "mgpu_render_noalloc: device ordinal too large");
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "mgpu_render_noalloc: cudaGetSymbolAddress of the fixed scratch");
    if (!p) return fail(MGPU_E_CUDA, "mgpu_render_noalloc: fixed scratch has no device address");
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return MGPU_OK;
}

// paths per wave that fit the fixed scratch for nl_slots light samples per path; asked: the limit of an
// explicit wave_paths, which stays what it was when a light sample took 84 bytes (now 48)
static int64_t noalloc_paths(int64_t nl_slots, bool asked) {
  const size_t fixed = workspace_bytes(0, 0, kNoAllocJobs);
  const size_t per = 11 * sizeof(float4) + 2 * sizeof(uint32_t) + (size_t)nl_slots * (asked ? 84 : 3 * sizeof(float4));
  if (kNoAllocBytes <= fixed) return 0;
  int64_t p = (int64_t)((kNoAllocBytes - fixed) / per);
  return p / 64 * 64;
}

// Function attributes belong to a device's context: they are set on the current device before
// its first render and again after the carveout knob changes.
//   the sorting blocks: kBins counters of dynamic shared memory, above the 48 KB default;
//   the wide traversal kernels: their warps' records, above the 48 KB default too;
//   the traversal and shade kernels: the L1 / shared-memory split ("carveout").  These kernels
//   chase pointers through L1 and need little shared memory, so the automatic carveout asks for
//   the least shared memory that keeps the kernel's register-limited number of resident blocks and
//   leaves the rest of the SM's 256 KB to L1.
struct CarveoutKernel {
  const void *f;
  int block;
  int dyn;  // dynamic shared memory of a block
};

static std::vector<CarveoutKernel> carveout_kernels() {
  return {{(const void *)k_extend<false, true, false>, kWideBlock, kWideSmem},
          {(const void *)k_extend<false, true, true>, kWideBlock, kWideSmem},
          {(const void *)k_extend<true, true, false>, kWideBlock, kWideSmem},
          {(const void *)k_extend<true, true, true>, kWideBlock, kWideSmem},
          {(const void *)k_shadow<false, true, false>, kWideBlock, kWideSmem},
          {(const void *)k_shadow<false, true, true>, kWideBlock, kWideSmem},
          {(const void *)k_shadow<true, true, false>, kWideBlock, kWideSmem},
          {(const void *)k_shadow<true, true, true>, kWideBlock, kWideSmem},
          {(const void *)k_traverse<false>, kWideBlock, kWideSmem},
          {(const void *)k_traverse<true>, kWideBlock, kWideSmem},
          {(const void *)k_extend<false, false, true>, kBlock, 0},
          {(const void *)k_extend<true, false, true>, kBlock, 0},
          {(const void *)k_shadow<false, false, true>, kBlock, 0},
          {(const void *)k_shadow<true, false, true>, kBlock, 0},
          {(const void *)k_shade<false, false>, kShadeTile, (int)sizeof(ShadeShared)},
          {(const void *)k_shade<true, false>, kShadeTile, (int)sizeof(ShadeShared)},
          {(const void *)k_shade<false, true>, kShadeTile, (int)sizeof(ShadeShared)},
          {(const void *)k_shade<true, true>, kShadeTile, (int)sizeof(ShadeShared)}};
}

// percent of the SM's shared memory that holds the kernel's resident blocks (registers and
// threads permitting) with their static shared memory and the per-block reservation
static cudaError_t auto_carveout(const CarveoutKernel &k, int smem_sm, int reserved, int &pct) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, k.f);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k.f, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e != cudaSuccess) return e;
  int blocks = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k.f, k.block, (size_t)k.dyn);
  if (e != cudaSuccess) return e;
  const int64_t need = (int64_t)blocks * (int64_t)(fa.sharedSizeBytes + (size_t)k.dyn + (size_t)reserved);
  pct = (int)std::min<int64_t>(100, (need * 100 + smem_sm - 1) / smem_sm);
  return cudaSuccess;
}

static cudaError_t kernel_attributes() {
  static std::mutex mu;
  static std::vector<int> applied;  // per device: the carveout knob last applied, INT_MIN = none
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int want = g_tune.carveout.load();
  std::lock_guard<std::mutex> lock(mu);
  if ((int)applied.size() <= dev) applied.resize((size_t)dev + 1, INT_MIN);
  if (applied[(size_t)dev] == want) return cudaSuccess;
  if (applied[(size_t)dev] == INT_MIN) {
    const void *bins[] = {(const void *)k_bin_hist, (const void *)k_bin_scatter};
    for (const void *kf : bins)
      if ((e = cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, kBinSmem)) != cudaSuccess) return e;
    for (const CarveoutKernel &k : carveout_kernels())
      if (k.dyn && (e = cudaFuncSetAttribute(k.f, cudaFuncAttributeMaxDynamicSharedMemorySize, k.dyn)) != cudaSuccess)
        return e;
  }
  int smem_sm = 0, reserved = 0;
  if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) != cudaSuccess) return e;
  for (const CarveoutKernel &k : carveout_kernels()) {
    int pct = want;
    if (want == kCarveoutAuto && (e = auto_carveout(k, smem_sm, reserved, pct)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k.f, cudaFuncAttributePreferredSharedMemoryCarveout, pct)) != cudaSuccess) return e;
  }
  applied[(size_t)dev] = want;
  return cudaSuccess;
}

static int grid_for(const void *kern, size_t smem, int block = kBlock) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, smem);
  if (per_sm < 1) per_sm = 1;
  return device_sm_count() * per_sm;
}

// A launch that, if chained, may overlap the end of the kernel before it on the stream (chain()).
template <class... P, class... A>
static void launch(bool chained, void (*kern)(P...), unsigned grid, int block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&c, kern, static_cast<P>(args)...);
}

static Camera make_camera(const float *c) {
  // ThinLensCamera::setOrientation (ThinLensCamera.cpp:241-259) and _computeMatrix (:204-210)
  double eye[3] = {c[0], c[1], c[2]}, look[3] = {c[3], c[4], c[5]}, up[3] = {c[6], c[7], c[8]};
  double n[3] = {-look[0], -look[1], -look[2]};
  double u[3] = {up[1] * n[2] - up[2] * n[1], up[2] * n[0] - up[0] * n[2], up[0] * n[1] - up[1] * n[0]};
  double ln = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]), lu = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
  for (int k = 0; k < 3; ++k) { n[k] /= ln; u[k] /= lu; }
  double v[3] = {n[1] * u[2] - n[2] * u[1], n[2] * u[0] - n[0] * u[2], n[0] * u[1] - n[1] * u[0]};
  double va = c[9] * (3.14159265358979323846 / 180.0);
  double th = tan(va / 2), tw = c[10] * th;
  Camera k;
  k.eye = v3((float)eye[0], (float)eye[1], (float)eye[2]);
  k.u = v3((float)u[0], (float)u[1], (float)u[2]);
  k.v = v3((float)v[0], (float)v[1], (float)v[2]);
  k.n = v3((float)n[0], (float)n[1], (float)n[2]);
  k.tan_w = (float)tw;
  k.tan_h = (float)th;
  k.aperture = c[11];
  k.focal_len = c[12];
  k.focal_dist = c[13];
  return k;
}

// A render request: one scene, parameters, film, optional per-path output.
struct Job {
  const mgpu_scene *scene;
  mgpu_render_params p;
  mgpu_film *film;
  float *path_out;
};

static int validate(const Job &j) {
  const mgpu_render_params *rp = &j.p;
  if (!j.scene || !j.film) return fail(MGPU_E_INVALID, "mgpu_render: null argument");
  if (rp->width != j.film->width || rp->height != j.film->height)
    return fail(MGPU_E_INVALID, "mgpu_render: film size differs from the render size");
  if (rp->width <= 0 || rp->height <= 0 || rp->spp <= 0 || rp->sample_count < 0 || rp->sample_begin < 0 ||
      rp->no_direct_samples <= 0 || rp->max_depth < 0 || rp->rr_start_depth < 0)
    return fail(MGPU_E_INVALID, "mgpu_render: bad parameters");
  if ((int64_t)rp->sample_begin + rp->sample_count > (int64_t)1 << 30)
    return fail(MGPU_E_INVALID, "mgpu_render: sample range too large");
  if (!(rp->camera[11] >= 0.0f) ||
      (rp->camera[11] > 0.0f && !(rp->camera[12] > 0.0f && rp->camera[13] > 0.0f)))
    return fail(MGPU_E_INVALID, "mgpu_render: a thin lens needs focal length and focal distance > 0 "
                                "(resolve autofocus before rendering)");
  int nds_side = std::max(1, (int)sqrt((double)rp->no_direct_samples));
  if ((int64_t)j.scene->nlight * nds_side * nds_side > 4096)
    return fail(MGPU_E_INVALID, "mgpu_render: too many light samples per vertex");
  return MGPU_OK;
}

// the job-level part of JobArgs
static JobArgs job_args(const Job &j) {
  const mgpu_scene *sc = j.scene;
  const mgpu_render_params *rp = &j.p;
  JobArgs J;
  memset(&J, 0, sizeof(J));
  J.view = sc->view;
  J.shade = sc->d_shade;
  J.mats = (const float4 *)sc->d_mats;
  J.lights = (const float4 *)sc->d_lights;
  J.uv = sc->d_uv;
  J.texrec = sc->d_texrec;
  J.texels = sc->d_texels;
  J.bg_tex = sc->bg_tex;
  for (int k = 0; k < 3; ++k) J.bg_le[k] = sc->bg_le[k];
  J.nlight = sc->nlight;
  J.cam = make_camera(rp->camera);
  J.rng.k0 = (uint32_t)rp->seed;
  J.rng.k1 = (uint32_t)(rp->seed >> 32);
  J.rng.stream = rp->stream_id;
  J.W = rp->width;
  J.H = rp->height;
  J.spp = rp->spp;
  J.side = std::max(1, (int)sqrt((double)rp->spp));
  J.s2 = J.side * J.side;
  J.nds = rp->no_direct_samples;
  J.nds_side = std::max(1, (int)sqrt((double)rp->no_direct_samples));
  J.nl_slots = sc->nlight * J.nds_side * J.nds_side;
  J.max_depth = rp->max_depth;
  J.rr_start = rp->rr_start_depth;
  J.efficient = rp->efficient_direct;
  J.tiles_x = (J.W + 7) / 8;
  J.sample_begin = rp->sample_begin;
  J.sample_count = rp->sample_count;
  J.film_sum = j.film->d_sum;
  J.film_c = j.film->d_c;
  J.filt = j.film->filter;
  J.film_fx = j.film->d_fx;
  J.path_out = (float4 *)j.path_out;
  for (int k = 0; k < 3; ++k) {
    const float ext = J.view.bmax[k] - J.view.bmin[k];
    J.cell_scale[k] = ext > 0.0f ? 32.0f / ext : 0.0f;
  }
  return J;
}

struct Wave {
  std::vector<JobArgs> chunks;
  int64_t npaths = 0, nslots = 0;
  int32_t nl_stride = 1;
  int32_t max_b = 1;
  bool unlimited = false;  // a chunk has no depth cap: drain by reading the live count
};

// Splits every job into chunks (sample passes outer, slot ranges inner, as many passes of the
// whole image as fit a wave) and packs them into waves of at most `cap` paths.  Two chunks of
// one job that share pixels never go into the same wave (their accumulate threads would race
// on the film); chunks of one job keep their sample order across waves.
static void pack_waves(const std::vector<Job> &jobs, int64_t cap, std::vector<Wave> &waves) {
  waves.clear();
  Wave cur;
  std::vector<int> last_job_wave(jobs.size(), -1);
  auto flush = [&]() {
    if (!cur.chunks.empty()) waves.push_back(cur);
    cur = Wave();
  };
  for (size_t ji = 0; ji < jobs.size(); ++ji) {
    const Job &job = jobs[ji];
    if (job.p.sample_count == 0) continue;
    JobArgs base = job_args(job);
    const int64_t total_slots = (int64_t)base.tiles_x * ((base.H + 7) / 8) * 64;
    const int ns = (int)std::max<int64_t>(1, std::min<int64_t>(job.p.sample_count, cap / total_slots));
    const int64_t spw = std::min<int64_t>(total_slots, std::max<int64_t>(64, cap / ns) / 64 * 64);
    bool job_in_cur = false;
    for (int s0 = job.p.sample_begin; s0 < job.p.sample_begin + job.p.sample_count; s0 += ns) {
      const int nsc = std::min(ns, job.p.sample_begin + job.p.sample_count - s0);
      for (int64_t slot0 = 0; slot0 < total_slots; slot0 += spw) {
        const int64_t nsl = std::min(spw, total_slots - slot0);
        const int64_t np = nsl * nsc;
        // a new sample range of a job already in this wave would revisit its pixels
        const bool conflict = job_in_cur && slot0 == 0;
        if (cur.npaths + np > cap || conflict) {
          flush();
          job_in_cur = false;
        }
        JobArgs J = base;
        J.s0 = s0;
        J.ns = nsc;
        J.slot0 = slot0;
        J.nslots = nsl;
        J.path_base = cur.npaths;
        J.slot_base = cur.nslots;
        cur.chunks.push_back(J);
        cur.npaths += np;
        cur.nslots += nsl;
        cur.nl_stride = std::max(cur.nl_stride, std::max(1, J.nl_slots));
        if (job.p.max_depth > 0) cur.max_b = std::max(cur.max_b, std::min(job.p.max_depth, kHardCap));
        else cur.unlimited = true;
        job_in_cur = true;
      }
    }
  }
  flush();
  for (auto &w : waves)
    if (w.unlimited) w.max_b = kHardCap;
}

// Renders a list of jobs.  noalloc: use the fixed scratch instead of the cached workspace.
template <bool COUNT>
static int render_jobs(const std::vector<Job> &jobs, void *stream, bool noalloc, int64_t wave_req,
                       uint64_t *graph_launches = nullptr, bool capture = false) {
  for (const Job &j : jobs) {
    int rc = validate(j);
    if (rc != MGPU_OK) return rc;
  }
  cudaStream_t caller = as_stream(stream);
  cudaStream_t st = caller;
  int32_t nl_max = 1;
  for (const Job &j : jobs)
    nl_max = std::max(nl_max, std::max(1, job_args(j).nl_slots));
  // automatic wave: the largest power of two up to 2^26 paths whose workspace fits 40 GB (larger
  // waves mean fewer bounce tails: mid frame 606 / 634 / 647 Mpaths/s at 2^24 / 2^25 / 2^26)
  int64_t wave = wave_req;
  if (wave <= 0) {
    const double per_path = (double)workspace_bytes((int64_t)1 << 20, ((int64_t)1 << 20) * nl_max, 1) / (1 << 20);
    wave = (int64_t)1 << 26;
    while (wave > ((int64_t)1 << 20) && (double)wave * per_path > kAutoWaveBytes) wave >>= 1;
  }
  if (noalloc) {
    const int64_t pmax = noalloc_paths(nl_max, true);
    if (pmax < 64)
      return fail(MGPU_E_INVALID, "mgpu_render_noalloc: " + std::to_string(nl_max) +
                                      " light samples per vertex do not fit the 32 MiB fixed scratch");
    if (wave_req > pmax)
      return fail(MGPU_E_INVALID, "mgpu_render_noalloc: wave_paths " + std::to_string(wave_req) +
                                      " exceeds the fixed scratch (32 MiB holds " + std::to_string(pmax) +
                                      " paths at " + std::to_string(nl_max) + " light samples per vertex)");
    wave = wave_req > 0 ? wave_req : noalloc_paths(nl_max, false);
  }
  std::vector<Wave> waves;
  bool use_graph = false;
  int64_t cap = 0, ncap = 0, nmax = 0, job_slots = 0;
  Workspace fixed_ws;
  Workspace *w = nullptr;
  for (;;) {
    pack_waves(jobs, wave, waves);
    if (waves.empty()) return MGPU_OK;
    bool any_unlimited = false;
    for (auto &wv : waves) any_unlimited |= wv.unlimited;
    use_graph = capture && !any_unlimited && !noalloc;
    // chunk descriptors: all of them up front when the launches are captured in a graph (no
    // host copies inside a capture), else each wave's own before its launches
    cap = ncap = nmax = 0;
    for (auto &wv : waves) {
      cap = std::max(cap, wv.npaths);
      ncap += (int64_t)wv.chunks.size();
      nmax = std::max(nmax, (int64_t)wv.chunks.size());
    }
    job_slots = use_graph ? ncap : nmax;
    if (noalloc) {
      if (job_slots > kNoAllocJobs)
        return fail(MGPU_E_INVALID, "mgpu_render_noalloc: more than " + std::to_string(kNoAllocJobs) +
                                        " chunks in one wave");
      void *base = nullptr;
      int rc = noalloc_scratch(&base);
      if (rc != MGPU_OK) return rc;
      fixed_ws.owned = false;
      MGPU_CUDA(cudaGetDevice(&fixed_ws.device));
      workspace_layout(&fixed_ws, base, cap, std::max<int64_t>(1, cap * nl_max), kNoAllocJobs);
      fixed_ws.h_counters = g_noalloc_host_counter;
      w = &fixed_ws;
      break;
    }
    int rc = ensure_workspace(cap, std::max<int64_t>(1, cap * nl_max), job_slots);
    if (rc == MGPU_E_NOMEM && wave_req <= 0 && wave > ((int64_t)1 << 20)) {
      cudaGetLastError();  // clear the failed allocation
      wave >>= 1;          // an automatic wave that does not fit the free memory: halve it
      continue;
    }
    if (rc != MGPU_OK) return rc;
    w = t_ws;
    break;
  }
  // (a copy from pageable memory returns once the runtime has staged the source)
  if (use_graph) {
    std::vector<JobArgs> all;
    all.reserve((size_t)ncap);
    for (auto &wv : waves) all.insert(all.end(), wv.chunks.begin(), wv.chunks.end());
    MGPU_CUDA(cudaMemcpyAsync(w->jobs, all.data(), all.size() * sizeof(JobArgs), cudaMemcpyHostToDevice, st));
  }

  bool sort_hits = false;
  for (const Job &j : jobs) sort_hits = sort_hits || j.scene->mixed;
  MGPU_CUDA(kernel_attributes());
  const int g_gen = grid_for((const void *)k_generate, 0, kGenBlock);
  const int g_sha = grid_for((const void *)k_shade<true, false>, sizeof(ShadeShared), kShadeTile);
  const int g_acc = grid_for((const void *)k_accumulate, 0);
  const int g_bin = device_sm_count() * 4;
  const int bin_ext = g_tune.bin_extension.load();
  const int64_t bin_min = g_tune.bin_min_paths.load();

  // The launches are captured on a private stream (the caller's may be the legacy default
  // stream, which cannot capture) and the graph is launched on the caller's stream.
  cudaGraph_t graph = nullptr;
  if (use_graph) {
    static thread_local cudaStream_t t_capture = nullptr;
    if (!t_capture) MGPU_CUDA(cudaStreamCreateWithFlags(&t_capture, cudaStreamNonBlocking));
    st = t_capture;
    MGPU_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  }

  mgpu_render_stats stats{};
  uint64_t launches = 0;
  Profiler off;  // the allocation-free and graph paths record no events
  Profiler &pf = (noalloc || use_graph) ? off : t_prof;
  cudaError_t err = cudaMemsetAsync(w->stats, 0, 12 * sizeof(unsigned long long), st);
  size_t job_off = 0;
  for (size_t wi = 0; wi < waves.size() && err == cudaSuccess; ++wi) {
    const Wave &wv = waves[wi];
    RenderArgs a;
    memset(&a, 0, sizeof(a));
    if (use_graph) {
      a.jobs = w->jobs + job_off;
      job_off += wv.chunks.size();
    } else {
      a.jobs = w->jobs;
      err = cudaMemcpyAsync(w->jobs, wv.chunks.data(), wv.chunks.size() * sizeof(JobArgs), cudaMemcpyHostToDevice, st);
      if (err != cudaSuccess) break;
    }
    a.njobs = (int32_t)wv.chunks.size();
    a.view0 = wv.chunks[0].view;
    a.npaths = wv.npaths;
    a.nslots = wv.nslots;
    a.nl_stride = wv.nl_stride;
    a.path_job = w->path_job;
    a.path_L = w->path_L;
    for (int k = 0; k < 2; ++k) { a.qo[k] = w->qo[k]; a.qd[k] = w->qd[k]; a.qt[k] = w->qt[k]; }
    a.qhit = w->qhit;
    a.so = w->so; a.sd = w->sd; a.slots = w->slots;
    a.qo_u = w->qo_u; a.qd_u = w->qd_u; a.qt_u = w->qt_u;
    a.qkey = w->qkey;
    int64_t wave_tris = 0;
    for (const JobArgs &c : wv.chunks) wave_tris = std::max(wave_tris, c.view.ntri);
    a.bin_ext = wv.npaths >= bin_min && (wave_tris >= kBinMinTris || bin_min == 0) ? bin_ext : 0;
    a.sort_hits = sort_hits;
    a.dense = 1;
    for (const JobArgs &c : wv.chunks) a.dense = a.dense && c.W % 8 == 0 && c.H % 8 == 0;
    a.counters = w->counters;
    a.stats = w->stats;
    a.tcount = w->tcount;
    a.max_b = wv.max_b;
    const int max_b = wv.max_b;
    bool sph = false;   // a chunk's scene has analytic spheres: the traversal kernels that test them
    bool wide = false;  // ... has the hierarchy, or no triangles; the rays of one that has not take the kd-tree
    for (const JobArgs &c : wv.chunks) {
      sph = sph || c.view.nsphere > 0;
      wide = wide || c.view.wnodes != nullptr || c.view.ntri == 0;
    }
    wide = wide && g_tune.wide.load() != 0;
    auto kext = !wide ? k_extend<COUNT, false, true> : sph ? k_extend<COUNT, true, true> : k_extend<COUNT, true, false>;
    auto kshw = !wide ? k_shadow<COUNT, false, true> : sph ? k_shadow<COUNT, true, true> : k_shadow<COUNT, true, false>;
    auto ktrv = sph ? k_traverse<true> : k_traverse<false>;
    const int tb = wide ? kWideBlock : kBlock;
    const size_t tsm = wide ? (size_t)kWideSmem : 0;
    const int g_ext = grid_for((const void *)kext, tsm, tb);
    const int g_shw = grid_for((const void *)kshw, tsm, tb);
    bool splats = false;  // a chunk's film has a reconstruction filter
    for (const JobArgs &c : wv.chunks) splats = splats || c.film_fx != nullptr;
    bool surf = false;  // a chunk's scene has image maps, a background or analytic spheres
    for (const JobArgs &c : wv.chunks)
      surf = surf || c.texrec != nullptr || c.bg_tex != 0 || c.bg_le[0] != 0.0f || c.bg_le[1] != 0.0f ||
             c.bg_le[2] != 0.0f || c.view.nsphere > 0;
    err = cudaMemsetAsync(w->counters, 0, kNumCounters * sizeof(uint32_t), st);
    int m = pf.begin(kProfGenerate, st);
    k_generate<<<g_gen, kGenBlock, 0, st>>>(a);
    pf.end(m, st);
    ++launches;
    // In waves of few light samples the starts and ends of launches count (851 paths 118 -> 111 us, 30,400 without
    // allocation 419 -> 386, two passes of 0.97 M paths 2.65 -> 2.585 ms); in larger ones kernels that overlap
    // gain nothing (ten scenes, 10 M paths: 4.69 / 4.68) or lose (textured, 5.3 M: 2.925 / 2.95).  Blocks that come
    // early fill the first SMs that come free instead of spreading over all, so a kernel whose work is in its
    // first few blocks is not chained: shading (plain box 838 / 827 us chained / not, spheres 1.561 / 1.541 ms) and
    // accumulation through a reconstruction filter (141 x 37 pixels of 64 samples 1.29 / 0.49 ms).
    const bool chained = wv.npaths * wv.nl_stride <= kSmallWaveSlots;
    auto kshd = surf ? k_shade<true, false> : k_shade<false, false>;
    auto kshp = surf ? k_shade<true, true> : k_shade<false, true>;
    int b = 0;
    // Whole paths in one launch where the rays fit the blocks that are resident at once: with more, the queues'
    // compaction over the whole wave is worth its launches (waves against whole paths: 3,404 paths of a 2 k-triangle
    // scene 144 / 75 us, 49,152 212 / 94; in the plain box 115,600 379 / 269, 155,236 404 / 398; textured
    // 115,600 561 / 521, 155,236 591 / 737; 105,800 without a depth cap 1,006 / 461).
    const bool can_whole = wide && !COUNT && g_tune.whole_paths.load() != 0;
    const int64_t whole_max = g_tune.whole_paths.load() > 0
                                  ? g_tune.whole_paths.load()
                                  : (int64_t)device_sm_count() * kShadeMinBlocks * kShadeTile;
    auto run_whole = [&](int64_t rays, int from) {
      // a block per SM at least, then full tiles (textured, 49,152 paths: 398 us in tiles of 256, 557 of 96)
      const int64_t sms = device_sm_count();
      const uint32_t per = (uint32_t)std::min<int64_t>(kShadeTile, ((rays + sms - 1) / sms + 31) / 32 * 32);
      RenderArgs w1 = a;
      w1.bin_ext = 0;  // a block's next rays stay with the block
      const int mk = pf.begin(kProfShade, st);
      launch(chained, kshp, (unsigned)((rays + per - 1) / per), kShadeTile, sizeof(ShadeShared), st, w1, from, per);
      pf.end(mk, st);
      ++launches;
    };
    if (can_whole && wv.npaths <= whole_max) {
      run_whole(wv.npaths, 0);
      b = max_b;
    }
    // From the second bounce on, a bounce's occlusion queries and the next one's closest hits in one launch, where
    // they are few enough that the ends of the launches count (per frame, apart against together, by the
    // wave's light samples: 2.9 M, 300,000 triangles to depth 8, 2 passes 2.93 / 2.66 ms; 1.0 M in the
    // plain box 0.866 / 0.840; 2.2 M, spheres without a depth cap 1.62 / 1.58; but 5.3 M textured 2.93 / 2.97 and
    // 64 M paths of the mid scene 109.2 / 112.0: two traversals in one kernel leave each fewer
    // registers, and the first bounce is the largest).  Per-kernel timing keeps them apart.
    const bool merge = chained && wide && !COUNT && !pf.enabled;
    while (b < max_b && err == cudaSuccess) {
      // with a fixed depth cap every bounce is launched blind; without one, check the live
      // count every 4 bounces and stop when the wave has drained
      int chunk = wv.unlimited ? std::min(4, max_b - b) : max_b;
      for (int k = 0; k < chunk; ++k, ++b) {
        if (k == 0 || b < 2 || !merge) {
          m = pf.begin(kProfExtend, st);
          launch(chained, kext, g_ext, tb, tsm, st, a, b);
          pf.end(m, st);
          ++launches;
        }
        m = pf.begin(kProfShade, st);
        kshd<<<g_sha, kShadeTile, sizeof(ShadeShared), st>>>(a, b, 0);
        pf.end(m, st);
        if (a.bin_ext && b + 1 < max_b) {
          const int nx = (b + 1) & 1;
          m = pf.begin(kProfBin, st);
          cudaMemsetAsync(w->hist, 0, kBins * sizeof(uint32_t), st);
          k_bin_hist<<<g_bin, 256, kBinSmem, st>>>(w->qkey, a.counters + kCtrRay + b + 1, w->hist);
          k_bin_scan<<<1, 1024, 0, st>>>(w->hist, w->cursor);
          k_bin_scatter<<<g_bin, 256, kBinSmem, st>>>(w->qkey, a.counters + kCtrRay + b + 1, w->cursor, w->qo_u, w->qd_u,
                                                      w->qt_u, w->qo[nx], w->qd[nx], w->qt[nx]);
          pf.end(m, st);
          launches += 3;
        }
        m = pf.begin(kProfShadow, st);
        if (merge && b > 0 && k + 1 < chunk) launch(chained, ktrv, g_ext, tb, tsm, st, a, b);
        else launch(chained, kshw, g_shw, tb, tsm, st, a, b);
        pf.end(m, st);
        launches += 2;
      }
      if (!wv.unlimited) break;
      err = cudaMemcpyAsync(w->h_counters, w->counters + kCtrRay + b, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
      if (err == cudaSuccess) err = cudaStreamSynchronize(st);
      if (err != cudaSuccess || w->h_counters[0] == 0) break;
      if (can_whole && (int64_t)w->h_counters[0] <= whole_max && b < max_b) {  // the long tail of few paths
        run_whole(w->h_counters[0], b);
        break;
      }
    }
    m = pf.begin(kProfAccumulate, st);
    launch(chained && !splats, k_accumulate, g_acc, kBlock, 0, st, a);
    pf.end(m, st);
    ++launches;
    if (err == cudaSuccess) err = cudaGetLastError();
  }
  if (use_graph) {
    cudaError_t ec = cudaStreamEndCapture(st, &graph);
    if (err == cudaSuccess) err = ec;
    if (err == cudaSuccess) {
      cudaGraphExec_t exec = nullptr;
      err = cudaGraphInstantiate(&exec, graph, 0);
      if (err == cudaSuccess) err = cudaGraphLaunch(exec, caller);
      if (exec) cudaGraphExecDestroy(exec);
    }
    if (graph) cudaGraphDestroy(graph);
    if (graph_launches) *graph_launches += 1;
  }
  if (err != cudaSuccess) return cuda_fail(err, "render");
  g_launches.fetch_add(launches);
  stats.paths = 0;
  for (const Job &j : jobs) stats.paths += (uint64_t)j.p.width * j.p.height * (uint64_t)j.p.sample_count;
  stats.kernel_launches = launches;
  t_stats = stats;
  t_stats_stream = caller;
  t_stats_dev = w->stats;
  t_counters_dev = w->counters;
  t_stats_pending = true;
  return MGPU_OK;
}

template <bool COUNT>
static int render_one(const mgpu_scene *sc, const mgpu_render_params *rp, mgpu_film *film, float *d_path_out,
                      void *stream, bool noalloc = false) {
  if (!sc || !rp || !film) return fail(MGPU_E_INVALID, "mgpu_render: null argument");
  std::vector<Job> jobs(1);
  jobs[0].scene = sc;
  jobs[0].p = *rp;
  jobs[0].film = film;
  jobs[0].path_out = d_path_out;
  if (rp->sample_count == 0) return validate(jobs[0]);
  return render_jobs<COUNT>(jobs, stream, noalloc, rp->wave_paths);
}

}  // namespace mgpu

// A batch: render requests that share waves (mgpu_batch_*).
struct mgpu_batch {
  std::vector<mgpu::Job> jobs;
  int64_t wave_paths = 0;
  int use_graph = 1;
  uint64_t graph_launches = 0;
};

using namespace mgpu;

extern "C" {

int mgpu_render(const mgpu_scene *scene, const mgpu_render_params *params, mgpu_film *film, void *stream) {
  return render_one<false>(scene, params, film, nullptr, stream);
}

int mgpu_render_paths(const mgpu_scene *scene, const mgpu_render_params *params, mgpu_film *film, float *d_path_L,
                      void *stream) {
  if (!d_path_L) return fail(MGPU_E_INVALID, "mgpu_render_paths: null path buffer");
  return render_one<false>(scene, params, film, d_path_L, stream);
}

// Allocation-free render: the same estimator and film as mgpu_render, over the fixed 32 MiB
// scratch instead of a cudaMalloc'd workspace.  See include/mgpu.h for the contract.
int mgpu_render_noalloc(const mgpu_scene *scene, const mgpu_render_params *params, mgpu_film *film, void *stream) {
  return render_one<false>(scene, params, film, nullptr, stream, true);
}

int mgpu_render_counted(const mgpu_scene *scene, const mgpu_render_params *params, mgpu_film *film,
                        uint64_t *counts8, void *stream) {
  if (!counts8) return fail(MGPU_E_INVALID, "mgpu_render_counted: null output");
  int rc = render_one<true>(scene, params, film, nullptr, stream);
  if (rc != MGPU_OK) return rc;
  MGPU_CUDA(cudaStreamSynchronize(as_stream(stream)));
  MGPU_CUDA(cudaMemcpy(counts8, t_ws->tcount, 8 * sizeof(uint64_t), cudaMemcpyDeviceToHost));
  return MGPU_OK;
}

int mgpu_batch_create(mgpu_batch **out) {
  if (!out) return fail(MGPU_E_INVALID, "mgpu_batch_create: null argument");
  *out = new (std::nothrow) mgpu_batch();
  if (!*out) return fail(MGPU_E_NOMEM, "mgpu_batch_create: out of host memory");
  return MGPU_OK;
}

int mgpu_batch_add(mgpu_batch *b, const mgpu_scene *scene, const mgpu_render_params *params, mgpu_film *film) {
  if (!b || !scene || !params || !film) return fail(MGPU_E_INVALID, "mgpu_batch_add: null argument");
  Job j;
  j.scene = scene;
  j.p = *params;
  j.film = film;
  j.path_out = nullptr;
  int rc = validate(j);
  if (rc != MGPU_OK) return rc;
  b->jobs.push_back(j);
  return MGPU_OK;
}

int mgpu_batch_set(mgpu_batch *b, int64_t wave_paths, int32_t use_graph) {
  if (!b || wave_paths < 0 || wave_paths > INT32_MAX) return fail(MGPU_E_INVALID, "mgpu_batch_set: bad argument");
  b->wave_paths = wave_paths;
  b->use_graph = use_graph;
  return MGPU_OK;
}

int mgpu_batch_render(mgpu_batch *b, void *stream) {
  if (!b) return fail(MGPU_E_INVALID, "mgpu_batch_render: null batch");
  if (b->jobs.empty()) return MGPU_OK;
  return render_jobs<false>(b->jobs, stream, false, b->wave_paths, &b->graph_launches, b->use_graph != 0);
}

int mgpu_batch_clear(mgpu_batch *b) {
  if (!b) return fail(MGPU_E_INVALID, "mgpu_batch_clear: null batch");
  b->jobs.clear();
  return MGPU_OK;
}

int mgpu_batch_destroy(mgpu_batch *b) {
  delete b;
  return MGPU_OK;
}

int mgpu_render_wave_queues(uint32_t *ext, uint32_t *shadow, int32_t max_bounces) {
  if (!ext || !shadow || max_bounces <= 0) return fail(MGPU_E_INVALID, "mgpu_render_wave_queues: bad argument");
  if (!t_counters_dev) return fail(MGPU_E_STATE, "mgpu_render_wave_queues: nothing rendered on this thread");
  MGPU_CUDA(cudaStreamSynchronize(t_stats_stream));
  const uint32_t *ctr = t_counters_dev;
  int n = std::min(max_bounces, kHardCap);
  MGPU_CUDA(cudaMemcpy(ext, ctr + kCtrRay, n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
  MGPU_CUDA(cudaMemcpy(shadow, ctr + kCtrNee, n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
  return MGPU_OK;
}

int mgpu_render_stats_get(mgpu_render_stats *out) {
  if (!out) return fail(MGPU_E_INVALID, "mgpu_render_stats_get: null argument");
  if (t_stats_pending && t_stats_dev) {
    unsigned long long h[4];
    MGPU_CUDA(cudaStreamSynchronize(t_stats_stream));
    MGPU_CUDA(cudaMemcpy(h, t_stats_dev, sizeof(h), cudaMemcpyDeviceToHost));
    t_stats.extension_rays = h[0];
    t_stats.shadow_rays = h[1];
    t_stats.truncated_paths = h[2];
    t_stats.bounces = h[3];
    t_stats_pending = false;
  }
  *out = t_stats;
  return MGPU_OK;
}

int mgpu_profile_enable(int enable) {
  Profiler &p = t_prof;
  int rc = p.flush();
  if (rc != MGPU_OK) return rc;
  p.enabled = enable != 0;
  for (int k = 0; k < kProfClasses; ++k) { p.ms[k] = 0; p.launches[k] = 0; }
  return MGPU_OK;
}

int mgpu_profile_read(double *ms6, uint64_t *launches6) {
  if (!ms6 || !launches6) return fail(MGPU_E_INVALID, "mgpu_profile_read: null argument");
  Profiler &p = t_prof;
  int rc = p.flush();
  if (rc != MGPU_OK) return rc;
  for (int k = 0; k < kProfClasses; ++k) { ms6[k] = p.ms[k]; launches6[k] = p.launches[k]; }
  return MGPU_OK;
}

int mgpu_tune_set(const char *key, int64_t value) {
  if (!key) return fail(MGPU_E_INVALID, "mgpu_tune_set: null key");
  std::string k(key);
  if (k == "persistent") g_tune.persistent.store(value != 0);
  else if (k == "coop_leaf" && value >= 0 && value <= 3) g_tune.coop_leaf.store((int)value);
  else if (k == "trav_block" && (value == 64 || value == 128 || value == 256)) g_tune.trav_block.store((int)value);
  else if (k == "wide") g_tune.wide.store(value != 0);
  else if (k == "whole_paths" && value >= -1) g_tune.whole_paths.store(value);
  else if (k == "bin_shadow") g_tune.bin_shadow.store(value != 0);
  else if (k == "bin_extension") g_tune.bin_extension.store(value != 0);
  else if (k == "bin_min_paths" && value >= 0) g_tune.bin_min_paths.store(value);
  else if (k == "carveout" && value >= kCarveoutAuto && value <= 100) {
    // applied per device before its next render (kernel_attributes)
    g_tune.carveout.store((int)value);
  } else return fail(MGPU_E_INVALID, "mgpu_tune_set: unknown key or bad value " + k);
  return MGPU_OK;
}

int mgpu_tune_get(const char *key, int64_t *value) {
  if (!key || !value) return fail(MGPU_E_INVALID, "mgpu_tune_get: null argument");
  std::string k(key);
  if (k == "persistent") *value = g_tune.persistent.load();
  else if (k == "coop_leaf") *value = g_tune.coop_leaf.load();
  else if (k == "trav_block") *value = g_tune.trav_block.load();
  else if (k == "wide") *value = g_tune.wide.load();
  else if (k == "whole_paths") *value = g_tune.whole_paths.load();
  else if (k == "bin_shadow") *value = g_tune.bin_shadow.load();
  else if (k == "bin_extension") *value = g_tune.bin_extension.load();
  else if (k == "bin_min_paths") *value = g_tune.bin_min_paths.load();
  else if (k == "carveout") *value = g_tune.carveout.load();
  else return fail(MGPU_E_INVALID, "mgpu_tune_get: unknown key " + k);
  return MGPU_OK;
}

}  // extern "C"
