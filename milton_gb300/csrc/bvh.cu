// bvh.cu -- device build of the 8-wide hierarchy that the traversal kernels use (hd_wide.h).
//
// Runs inside mgpu_scene_create on the triangles just uploaded, so a scene's preparation stays one
// host kd-tree (the object that Milton's callers inspect) and one upload:
//   1. Morton order of the triangle boxes' centres (16 bits per axis, one radix sort);
//   2. a binary hierarchy by parallel locally-ordered clustering (Meister and Bittner, TVCG 2018):
//      every cluster looks for the neighbour within kRadius places whose union with it has the
//      least surface area; mutual pairs merge; repeat on the compacted array;
//   3. the cheapest 8-wide cut of every subtree by the surface-area dynamic program of Ylitie,
//      Karras and Laine (HPG 2017), bottom-up;
//   4. top-down, level by level: eight lanes per wide node list its children, give them slots by
//      octant, quantise their boxes outward and write node and triangles (one thread per node took
//      93 us a level of dependent steps; 1 M triangles: scene creation 7.7 -> 6.5 ms, of which the
//      build is 2.6).
// Every kernel is bounded: sizes are read from device counters that only earlier launches write,
// and a build that does not fit its arrays reports so and the scene keeps the kd-tree traversal.
#include <string.h>

#include <algorithm>

#include "common.cuh"
#include "hd_wide.h"

namespace mgpu {

namespace {

// neighbours looked at on each side (mid frame, traversal: 94.8 ms at 8, 95.8 at 16, 97.2 at 32)
constexpr int kRadius = 8;
constexpr int kPlocBlock = 256;
constexpr int kTailMax = 2048;       // clusters that one block finishes in shared memory
constexpr int kSmall = kTailMax;     // triangles of a scene that one block builds
constexpr int kRadixItems = 16;      // keys per thread of a radix-sort block
constexpr int kRadixTile = 256 * kRadixItems;
constexpr int kMortonBits = 48;
constexpr int kMaxLevels = kWideMaxDepth;
// costs of the surface-area dynamic program: one wide node step against one triangle test (0.1 to 0.333
// measure the same; above 1/3 the bound of wide_node_cap would not hold)
constexpr float kCostNode = 1.0f, kCostTri = 0.3f;

struct Box {
  float lo[3], hi[3];
};

__device__ __forceinline__ float half_area(const Box &b) {
  const float x = b.hi[0] - b.lo[0], y = b.hi[1] - b.lo[1], z = b.hi[2] - b.lo[2];
  return x * y + y * z + z * x;
}

__device__ __forceinline__ Box join(const Box &a, const Box &b) {
  Box r;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r.lo[k] = fminf(a.lo[k], b.lo[k]);
    r.hi[k] = fmaxf(a.hi[k], b.hi[k]);
  }
  return r;
}

// A binary node: leaves 0 .. n - 1 in Morton order, inner nodes n .. 2 n - 2.
struct BNode {
  Box box;
  int32_t left, right;  // inner: children; leaf: primitive id, -1
};

// The dynamic program's answer for an inner node: c[i - 1] the least cost of covering its subtree with
// at most i children; pick[i]: how many of the i go to the left child (0: the i - 1 answer is as
// good); pick[0] = 1: the subtree as one leaf child; pick[8]: the split of a wide node here.
struct Cut {
  float c[7];
  uint8_t pick[9];
  uint8_t prims;  // triangles of the subtree, 255 = more than a leaf holds
  uint16_t pad;
};

struct Build {
  int32_t n;
  const F4 *tris;
  uint32_t *bounds;       // 6 ordered words: centre minima, maxima
  uint64_t *key[2];
  int32_t *val[2];
  uint32_t *hist;         // radix histograms
  BNode *node;            // 2 n - 1
  int32_t *parent;        // 2 n - 1
  uint32_t *arrived;      // n - 1: children whose cut is done
  Cut *cut;               // n - 1
  int32_t *cl[2];         // clusters
  int32_t *nn;
  uint2 *bsum;            // per block: survivors, merges
  uint32_t *ctr;          // counters (kC*)
  int32_t *wroot;         // binary root of every wide node
  uint32_t *wnodes;
  F4 *wtris;
  uint32_t cap_nodes;
  float centre[3];        // node coordinates are relative to it
  float bmin[3], bmax[3];  // the kd-tree's root box
};

// counters
constexpr int kCCount = 0;    // clusters left
constexpr int kCNext = 1;     // next inner binary node
constexpr int kCForce = 2;    // the next round pairs neighbours
constexpr int kCParity = 3;   // which cluster array is current
constexpr int kCNodes = 4;    // wide nodes
constexpr int kCTris = 5;     // triangle records
constexpr int kCFail = 6;
constexpr int kCOut = 7;      // a triangle sticks out
constexpr int kCLevel = 8;    // first wide node of each level (kMaxLevels + 2)
constexpr int kNumC = kCLevel + kMaxLevels + 8;
static_assert(kNumC <= kWideCounters, "the caller's counters");

__device__ __forceinline__ uint32_t order_bits(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unorder_bits(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Whether a triangle reaches out of the kd-tree's root box.  The root box leaves out triangles whose bounds compare
// equal under Milton's fuzzy comparison (flat ones from -1 to 1, kdbuild.cpp); rays find such a triangle only
// where a leaf on their way through the root box lists it, wherever they hit it.  Its records carry
// kWideOutside, and the kd-tree decides a ray that hits one before anything else, unless it is certain
// to find that hit (wide_listed).
__device__ __forceinline__ bool sticks_out(const Build &B, const Box &b) {
  bool out = false;
  for (int k = 0; k < 3; ++k) out = out || b.lo[k] < B.bmin[k] || b.hi[k] > B.bmax[k];
  return out;
}

__device__ __forceinline__ Box tri_box(const Build &B, int64_t t) {
  const F4 a = load_f4(B.tris, 3 * t), b = load_f4(B.tris, 3 * t + 1), c = load_f4(B.tris, 3 * t + 2);
  Box r;
  r.lo[0] = fminf(a.x, fminf(b.x, c.x)); r.hi[0] = fmaxf(a.x, fmaxf(b.x, c.x));
  r.lo[1] = fminf(a.y, fminf(b.y, c.y)); r.hi[1] = fmaxf(a.y, fmaxf(b.y, c.y));
  r.lo[2] = fminf(a.z, fminf(b.z, c.z)); r.hi[2] = fmaxf(a.z, fmaxf(b.z, c.z));
  // nothing hits a point, and the kd-tree's bounds leave it out: it must not widen the hierarchy's.  (Bounds of
  // nothing, where the kd-tree leaves out every triangle, would make it infinite and its areas NaN, which
  // no order of neighbours survives.)
  if (r.lo[0] == r.hi[0] && r.lo[1] == r.hi[1] && r.lo[2] == r.hi[2])
    for (int k = 0; k < 3; ++k)
      r.lo[k] = r.hi[k] = B.bmin[k] <= B.bmax[k] ? fminf(fmaxf(r.lo[k], B.bmin[k]), B.bmax[k]) : 0.0f;
  return r;
}

__global__ void k_bvh_init(Build B) {
  if (threadIdx.x < kNumC) B.ctr[threadIdx.x] = 0u;
  __syncthreads();
  if (threadIdx.x == 0) {
    B.ctr[kCCount] = (uint32_t)B.n;
    B.ctr[kCNext] = (uint32_t)B.n;
    B.ctr[kCNodes] = 1u;  // the root
    B.ctr[kCLevel + 1] = 1u;
  }
  if (threadIdx.x < 6) B.bounds[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
}

// bounds of the triangle boxes' centres over triangles first, first + stride, ... into six ordered words
__device__ void centre_bounds(const Build &B, int64_t first, int64_t stride, uint32_t *g) {
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t t = first; t < B.n; t += stride) {
    const Box b = tri_box(B, t);
    for (int k = 0; k < 3; ++k) {
      const float c = 0.5f * b.lo[k] + 0.5f * b.hi[k];
      lo[k] = fminf(lo[k], c);
      hi[k] = fmaxf(hi[k], c);
    }
  }
  for (int k = 0; k < 3; ++k) {
    const uint32_t l = __reduce_min_sync(0xFFFFFFFFu, order_bits(lo[k]));
    const uint32_t h = __reduce_max_sync(0xFFFFFFFFu, order_bits(hi[k]));
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&g[k], l);
      atomicMax(&g[3 + k], h);
    }
  }
}

__global__ void __launch_bounds__(256) k_bvh_bounds(Build B) {
  centre_bounds(B, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x, B.bounds);
}

// 16 bits -> every third bit
__device__ __forceinline__ uint64_t spread16(uint32_t v) {
  uint64_t x = v & 0xFFFFu;
  x = (x | (x << 16)) & 0x0000FF0000FFull;
  x = (x | (x << 8)) & 0x00F00F00F00Full;
  x = (x | (x << 4)) & 0x0C30C30C30C3ull;
  x = (x | (x << 2)) & 0x249249249249ull;
  return x;
}

// One cell size for the three axes, so that a flat scene spends its bits where its extent is.
__device__ __forceinline__ uint64_t morton_key(const Build &B, const uint32_t *g, int64_t t) {
  float lo[3], ext = 0.0f;
  for (int k = 0; k < 3; ++k) {
    lo[k] = unorder_bits(g[k]);
    ext = fmaxf(ext, unorder_bits(g[3 + k]) - lo[k]);
  }
  const float scale = ext > 0.0f ? 65535.0f / ext : 0.0f;
  const Box b = tri_box(B, t);
  uint32_t c[3];
  for (int k = 0; k < 3; ++k)
    c[k] = (uint32_t)fminf(fmaxf((0.5f * b.lo[k] + 0.5f * b.hi[k] - lo[k]) * scale, 0.0f), 65535.0f);
  return (spread16(c[0]) << 2) | (spread16(c[1]) << 1) | spread16(c[2]);
}

__global__ void __launch_bounds__(256) k_bvh_morton(Build B) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < B.n; t += (int64_t)gridDim.x * blockDim.x) {
    B.key[0][t] = morton_key(B, B.bounds, t);
    B.val[0][t] = (int32_t)t;
  }
}

// radix sort pass, 8 bits: per-block digit counts (digit-major), scan, stable scatter
__global__ void __launch_bounds__(256) k_bvh_radix_count(const uint64_t *__restrict__ key, int32_t n, int shift,
                                                         uint32_t *__restrict__ hist) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0u;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kRadixTile;
#pragma unroll 4
  for (int j = 0; j < kRadixItems; ++j) {
    const int64_t i = base + j * 256 + threadIdx.x;
    if (i < n) atomicAdd(&h[(uint32_t)(key[i] >> shift) & 255u], 1u);
  }
  __syncthreads();
  hist[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// exclusive scan of m words by one block of 1024 threads
__device__ __forceinline__ void block_scan(uint32_t *a, uint32_t m, uint32_t *part) {
  uint32_t carry = 0u;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t base = 0; base < m; base += 4096) {
    const uint32_t i = base + 4 * threadIdx.x;
    uint32_t x[4], sum = 0u;
    for (int k = 0; k < 4; ++k) {
      x[k] = i + k < m ? a[i + k] : 0u;
      sum += x[k];
    }
    uint32_t inc = sum;
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
      if (lane >= (uint32_t)d) inc += y;
    }
    if (lane == 31u) part[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = part[lane], wi = w;
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, d);
        if (lane >= (uint32_t)d) wi += y;
      }
      part[lane] = wi - w;
      if (lane == 31u) part[32] = wi;
    }
    __syncthreads();
    uint32_t e = carry + part[warp] + inc - sum;
    for (int k = 0; k < 4; ++k) {
      if (i + k < m) a[i + k] = e;
      e += x[k];
    }
    carry += part[32];
    __syncthreads();
  }
}

__global__ void __launch_bounds__(1024) k_bvh_radix_scan(uint32_t *hist, uint32_t m) {
  __shared__ uint32_t part[33];
  block_scan(hist, m, part);
}

__global__ void __launch_bounds__(256) k_bvh_radix_scatter(const uint64_t *__restrict__ key,
                                                           const int32_t *__restrict__ val, int32_t n, int shift,
                                                           const uint32_t *__restrict__ hist,
                                                           uint64_t *__restrict__ key_out,
                                                           int32_t *__restrict__ val_out) {
  // keys in blocked order per warp: warp w takes keys [w 512, w 512 + 512) of the tile, 32 at a time,
  // so the ranks of equal digits follow the key order (stable)
  __shared__ uint32_t cnt[8][256];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < 8 * 256; i += 256) (&cnt[0][0])[i] = 0u;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kRadixTile + warp * (kRadixTile / 8);
  uint32_t rank[kRadixItems], digit[kRadixItems];
#pragma unroll
  for (int j = 0; j < kRadixItems; ++j) {
    const int64_t i = base + j * 32 + lane;
    const bool ok = i < n;
    const uint32_t d = ok ? (uint32_t)(key[i] >> shift) & 255u : 256u;
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
    uint32_t before = 0u;
    const int leader = __ffs(peers) - 1;
    if (ok && (int)lane == leader) {
      before = cnt[warp][d];
      cnt[warp][d] = before + __popc(peers);
    }
    before = __shfl_sync(0xFFFFFFFFu, before, leader);
    digit[j] = d;
    rank[j] = before + __popc(peers & ((1u << lane) - 1u));
    __syncwarp();
  }
  __syncthreads();
  {
    uint32_t s = hist[(size_t)threadIdx.x * gridDim.x + blockIdx.x];
    for (int w = 0; w < 8; ++w) {
      const uint32_t c = cnt[w][threadIdx.x];
      cnt[w][threadIdx.x] = s;
      s += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRadixItems; ++j) {
    const int64_t i = base + j * 32 + lane;
    if (i < n) {
      const uint32_t p = cnt[warp][digit[j]] + rank[j];
      key_out[p] = key[i];
      val_out[p] = val[i];
    }
  }
}

__device__ __forceinline__ Box make_leaf(const Build &B, int64_t i, int32_t t) {
  BNode nd;
  nd.box = tri_box(B, t);
  nd.left = t;
  nd.right = -1;
  B.node[i] = nd;
  if (i < B.n - 1) B.arrived[i] = 0u;
  return nd.box;
}

__global__ void __launch_bounds__(256) k_bvh_leaves(Build B, const int32_t *__restrict__ order) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < B.n; i += (int64_t)gridDim.x * blockDim.x) {
    make_leaf(B, i, order[i]);
    B.cl[0][i] = (int32_t)i;
  }
}

// ---- clustering ---------------------------------------------------------------------------

// Whether cluster i prefers neighbour j, union area a, to bj, union area best (bj < 0: none yet): the least
// area; the order (area, smaller index, larger index) is the same from both sides, so the least pair
// overall is mutual and every round merges.
__device__ __forceinline__ bool nearer(int i, float a, int j, float best, int bj) {
  const int mn = min(i, j), mx = max(i, j), bn = min(i, bj), bx = max(i, bj);
  return bj < 0 || a < best || (a == best && (mn < bn || (mn == bn && mx < bx)));
}

// The neighbour of cluster i (at sb[at]): of its 2 x kRadius candidates number q, q + lanes, ...
__device__ __forceinline__ int nearest(const Box *sb, int at, int i, int count, int q, int lanes, float &best) {
  int bj = -1;
  best = INFINITY;
  for (int o = q; o < 2 * kRadius; o += lanes) {
    const int d = (o & 1) ? 1 + (o >> 1) : -1 - (o >> 1), j = i + d;
    if (j < 0 || j >= count) continue;
    const float a = half_area(join(sb[at], sb[at + d]));
    if (nearer(i, a, j, best, bj)) {
      best = a;
      bj = j;
    }
  }
  return bj;
}

__global__ void __launch_bounds__(kPlocBlock) k_bvh_nearest(Build B) {
  __shared__ Box sb[kPlocBlock + 2 * kRadius];
  const int count = (int)B.ctr[kCCount];
  if (count <= kTailMax) return;
  const bool force = B.ctr[kCForce] != 0u;
  const int32_t *cl = B.cl[B.ctr[kCParity]];
  for (int base = blockIdx.x * kPlocBlock; base < count; base += gridDim.x * kPlocBlock) {
    for (int k = threadIdx.x; k < kPlocBlock + 2 * kRadius; k += kPlocBlock) {
      const int j = base - kRadius + k;
      if (j >= 0 && j < count) sb[k] = B.node[cl[j]].box;
    }
    __syncthreads();
    const int i = base + (int)threadIdx.x;
    float best;
    if (i < count)
      B.nn[i] = force ? ((i ^ 1) < count ? (i ^ 1) : -1) : nearest(sb, (int)threadIdx.x + kRadius, i, count, 0, 1, best);
    __syncthreads();
  }
}

// what becomes of cluster i: merged into a new node (i the smaller of a mutual pair), gone (the larger),
// kept
__device__ __forceinline__ int fate(const int32_t *nn, int i) {
  const int j = nn[i];
  if (j < 0 || nn[j] != i) return 0;
  return i < j ? 1 : 2;
}

__global__ void __launch_bounds__(1024) k_bvh_merge_count(Build B) {
  const int count = (int)B.ctr[kCCount];
  if (count <= kTailMax) return;
  __shared__ uint32_t sk, sm;
  for (int blk = blockIdx.x; blk * 1024 < count; blk += gridDim.x) {
    if (threadIdx.x == 0) sk = sm = 0u;
    __syncthreads();
    const int i = blk * 1024 + (int)threadIdx.x;
    const int f = i < count ? fate(B.nn, i) : 2;
    const uint32_t keep = __popc(__ballot_sync(0xFFFFFFFFu, f != 2)), merge = __popc(__ballot_sync(0xFFFFFFFFu, f == 1));
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&sk, keep);
      atomicAdd(&sm, merge);
    }
    __syncthreads();
    if (threadIdx.x == 0) B.bsum[blk] = make_uint2(sk, sm);
    __syncthreads();
  }
}

// one block: exclusive scan of the per-block counts; leaves the totals in the entry after the last
__global__ void __launch_bounds__(1024) k_bvh_merge_scan(Build B) {
  const int count = (int)B.ctr[kCCount];
  if (count <= kTailMax) return;
  const int nb = (count + 1023) / 1024;
  __shared__ uint32_t wk[32], wm[32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t ck = 0u, cm = 0u;
  for (int base = 0; base < nb; base += 1024) {
    const int i = base + (int)threadIdx.x;
    const uint2 x = i < nb ? B.bsum[i] : make_uint2(0u, 0u);
    uint32_t ik = x.x, im = x.y;
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, ik, d), b = __shfl_up_sync(0xFFFFFFFFu, im, d);
      if (lane >= (uint32_t)d) { ik += a; im += b; }
    }
    if (lane == 31u) { wk[warp] = ik; wm[warp] = im; }
    __syncthreads();
    uint32_t pk = ck, pm = cm, tk = 0u, tm = 0u;
    for (uint32_t w = 0; w < 32; ++w) {
      if (w < warp) { pk += wk[w]; pm += wm[w]; }
      tk += wk[w];
      tm += wm[w];
    }
    if (i < nb) B.bsum[i] = make_uint2(pk + ik - x.x, pm + im - x.y);
    ck += tk;
    cm += tm;
    __syncthreads();
  }
  if (threadIdx.x == 0) B.bsum[nb] = make_uint2(ck, cm);
}

__device__ __forceinline__ void make_inner(const Build &B, int32_t id, int32_t l, int32_t r) {
  BNode nd;
  nd.box = join(B.node[l].box, B.node[r].box);
  nd.left = l;
  nd.right = r;
  B.node[id] = nd;
  B.parent[l] = id;
  B.parent[r] = id;
}

__global__ void __launch_bounds__(1024) k_bvh_merge(Build B) {
  const int count = (int)B.ctr[kCCount];
  if (count <= kTailMax) return;
  const uint32_t par = B.ctr[kCParity], next = B.ctr[kCNext];
  const int32_t *cl = B.cl[par];
  int32_t *out = B.cl[par ^ 1u];
  __shared__ uint32_t wk[32], wm[32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (int blk = blockIdx.x; blk * 1024 < count; blk += gridDim.x) {
    const int i = blk * 1024 + (int)threadIdx.x;
    const int f = i < count ? fate(B.nn, i) : 2;
    const uint32_t mk = __ballot_sync(0xFFFFFFFFu, f != 2), mm = __ballot_sync(0xFFFFFFFFu, f == 1);
    if (lane == 0u) { wk[warp] = __popc(mk); wm[warp] = __popc(mm); }
    __syncthreads();
    const uint2 b = B.bsum[blk];
    uint32_t k = b.x + __popc(mk & ((1u << lane) - 1u)), m = b.y + __popc(mm & ((1u << lane) - 1u));
    for (uint32_t w = 0; w < warp; ++w) { k += wk[w]; m += wm[w]; }
    if (f != 2) {
      int32_t id = cl[i];
      if (f == 1) {
        const int32_t l = id, r = cl[B.nn[i]];
        id = (int32_t)(next + m);
        make_inner(B, id, l, r);
      }
      out[k] = id;
    }
    __syncthreads();
  }
}

// closes a round: the new count, the next inner node; a round that merged less than a tenth of the
// clusters (chains of clusters each nearest to the one before) makes the next pair neighbours,
// which bounds the number of rounds by the logarithm of the triangle count
__global__ void k_bvh_round(Build B) {
  const uint32_t count = B.ctr[kCCount];
  if (count <= (uint32_t)kTailMax) return;
  const uint2 t = B.bsum[(count + 1023u) / 1024u];
  B.ctr[kCForce] = t.y < count / 10u ? 1u : 0u;
  B.ctr[kCCount] = t.x;
  B.ctr[kCNext] += t.y;
  B.ctr[kCParity] ^= 1u;
}

// All remaining rounds of at most kTailMax clusters by one block of 1024 threads: id, sb hold the clusters
// and their boxes, nn is scratch; the next inner node is next0.
struct TailShared {
  Box sb[kTailMax];
  int32_t id[kTailMax], nn[kTailMax];
  uint32_t wk[32], wm[32], next;
  int force;
};

__device__ void cluster_tail(const Build &B, TailShared &S, int count, uint32_t next0) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) { S.next = next0; S.force = 0; }
  __syncthreads();
  while (count > 1) {
    const bool force = S.force != 0;
    // up to 16 lanes share a cluster's candidates: the rounds of few clusters are many, and each waited for
    // the 16 candidates one after another (36 clusters: 43 -> 24 us; 2,048: 148 -> 109)
    int lanes = 1;
    while (lanes < 2 * kRadius && 2 * lanes * count <= 1024) lanes *= 2;
    for (int base = 0; base < count; base += 1024 / lanes) {
      const int i = base + (int)threadIdx.x / lanes, q = (int)threadIdx.x & (lanes - 1);
      float best = INFINITY;
      int j = -1;
      if (i < count) j = force ? ((i ^ 1) < count ? (i ^ 1) : -1) : nearest(S.sb, i, i, count, q, lanes, best);
      for (int d = 1; d < lanes; d <<= 1) {
        const float oa = __shfl_xor_sync(0xFFFFFFFFu, best, d);
        const int oj = __shfl_xor_sync(0xFFFFFFFFu, j, d);
        if (!force && oj >= 0 && nearer(i, oa, oj, best, j)) {
          best = oa;
          j = oj;
        }
      }
      if (q == 0 && i < count) S.nn[i] = j;
    }
    __syncthreads();
    // two clusters per thread, in order; the warps beyond them only wait
    const uint32_t warps = ((uint32_t)count + 63u) / 64u;
    const bool busy = warp < warps;
    const int i0 = 2 * (int)threadIdx.x, i1 = i0 + 1;
    const int f0 = i0 < count ? fate(S.nn, i0) : 2, f1 = i1 < count ? fate(S.nn, i1) : 2;
    uint32_t k = 0u, m = 0u;
    if (busy) {
      const uint32_t k2 = (f0 != 2) + (f1 != 2), m2 = (f0 == 1) + (f1 == 1);
      uint32_t ik = k2, im = m2;
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, ik, d), b = __shfl_up_sync(0xFFFFFFFFu, im, d);
        if (lane >= (uint32_t)d) { ik += a; im += b; }
      }
      if (lane == 31u) { S.wk[warp] = ik; S.wm[warp] = im; }
      k = ik - k2;
      m = im - m2;
    }
    __syncthreads();
    uint32_t tk = 0u, tm = 0u;
    for (uint32_t w = 0; w < warps; ++w) {
      if (w < warp) { k += S.wk[w]; m += S.wm[w]; }
      tk += S.wk[w];
      tm += S.wm[w];
    }
    Box nb[2];
    int32_t ni[2];
    const uint32_t next = S.next;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = i0 + h, f = h ? f1 : f0;
      if (f == 2) continue;
      ni[h] = S.id[i];
      nb[h] = S.sb[i];
      if (f == 1) {
        const int j = S.nn[i];
        const int32_t nid = (int32_t)(next + m);
        ++m;
        BNode nd;
        nd.box = join(S.sb[i], S.sb[j]);
        nd.left = S.id[i];
        nd.right = S.id[j];
        B.node[nid] = nd;
        B.parent[S.id[i]] = nid;
        B.parent[S.id[j]] = nid;
        ni[h] = nid;
        nb[h] = nd.box;
      }
    }
    __syncthreads();
    if (f0 != 2) { S.id[k] = ni[0]; S.sb[k] = nb[0]; ++k; }
    if (f1 != 2) { S.id[k] = ni[1]; S.sb[k] = nb[1]; }
    if (threadIdx.x == 0) {
      S.next = next + tm;
      S.force = tm == 0u || tm < (uint32_t)count / 10u ? 1 : 0;  // the next round merges, whatever the areas
    }
    count = (int)tk;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    B.parent[S.id[0]] = -1;
    B.wroot[0] = S.id[0];
  }
  __syncthreads();
}

// the last kTailMax clusters
__global__ void __launch_bounds__(1024) k_bvh_tail(Build B) {
  extern __shared__ __align__(16) unsigned char smem[];
  TailShared &S = *reinterpret_cast<TailShared *>(smem);
  const int count = (int)B.ctr[kCCount];
  if (count > kTailMax) return;
  const int32_t *cl = B.cl[B.ctr[kCParity]];
  for (int i = threadIdx.x; i < count; i += 1024) {
    S.id[i] = cl[i];
    S.sb[i] = B.node[cl[i]].box;
  }
  cluster_tail(B, S, count, B.ctr[kCNext]);
}

// ---- the dynamic program ------------------------------------------------------------------

struct Costs {
  float c[7];
  int prims;
};

template <bool BLOCK>
__device__ __forceinline__ Costs costs_of(const Build &B, int32_t id) {
  Costs r;
  if (id < B.n) {
    const float a = half_area(B.node[id].box) * kCostTri;
    for (int k = 0; k < 7; ++k) r.c[k] = a;
    r.prims = 1;
  } else {
    const Cut *q = B.cut + (id - B.n);
    for (int k = 0; k < 7; ++k) r.c[k] = BLOCK ? q->c[k] : __ldcg(&q->c[k]);
    r.prims = BLOCK ? q->prims : __ldcg(&q->prims);
  }
  return r;
}

// Leaf i climbs; the second child to arrive at a node computes its cut.  Nothing waits.  arrived: children of
// inner node n + k whose cut is done.  BLOCK: all leaves climb in one block, which needs neither fences
// nor loads beyond its SM.
template <bool BLOCK>
__device__ void climb(const Build &B, int64_t i, uint32_t *arrived) {
  int32_t at = B.n > 1 ? B.parent[i] : -1;
  while (at >= 0) {
    if (BLOCK) __threadfence_block(); else __threadfence();
    if (atomicAdd(&arrived[at - B.n], 1u) == 0u) break;
    if (BLOCK) __threadfence_block(); else __threadfence();
    const BNode nd = B.node[at];
    const Costs l = costs_of<BLOCK>(B, nd.left), r = costs_of<BLOCK>(B, nd.right);
    const float area = half_area(nd.box);
    Cut c;
    c.pad = 0;
    float dist[9];
    c.pick[1] = 0;
    for (int j = 2; j <= 8; ++j) {
      float best = INFINITY;
      int bk = 1;
      for (int k = 1; k < j; ++k) {
        if (k > 7 || j - k > 7) continue;
        const float v = l.c[k - 1] + r.c[j - k - 1];
        if (v < best) { best = v; bk = k; }
      }
      dist[j] = best;
      c.pick[j] = (uint8_t)bk;
    }
    const int prims = l.prims + r.prims;
    const float inner = dist[8] + area * kCostNode;
    const float leaf = prims <= kWideLeafTris ? area * (float)prims * kCostTri : INFINITY;
    c.pick[0] = (prims <= kWideLeafTris && leaf <= inner) ? 1 : 0;
    c.c[0] = c.pick[0] ? leaf : inner;
    for (int j = 2; j <= 7; ++j) {
      if (dist[j] <= c.c[j - 2]) {
        c.c[j - 1] = dist[j];
      } else {
        c.c[j - 1] = c.c[j - 2];
        c.pick[j] = 0;
      }
    }
    c.prims = (uint8_t)min(prims, 255);
    B.cut[at - B.n] = c;
    at = B.parent[at];
  }
}

__global__ void __launch_bounds__(128) k_bvh_cut(Build B) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < B.n; i += (int64_t)gridDim.x * blockDim.x)
    climb<false>(B, i, B.arrived);
}

// ---- wide nodes ---------------------------------------------------------------------------

// first wide node of the next level = the nodes there are now
__global__ void k_bvh_level(Build B, int level) { B.ctr[kCLevel + level] = B.ctr[kCNodes]; }

// The upper half of the smallest float no less than v whose lower half is zero.
__device__ __forceinline__ uint32_t plane_above(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u + ((u & 0x80000000u) ? 0u : 0xFFFFu)) >> 16;
}

// Eight lanes per wide node, one per child (called by whole warps; valid is uniform over the eight).
// xn, xj: eight words of shared memory each per group.
__device__ void emit_node(const Build &B, uint32_t w, bool valid, int32_t *xn, int32_t *xj) {
  const uint32_t lane = threadIdx.x & 7u, shift = threadIdx.x & 24u, group = 0xFFu << shift;
  if (!valid) return;
  const int32_t root = B.wroot[w];
  // the children that the dynamic program picked: every lane holds (node, budget), and those that it
  // splits hand their right half to the next free lane
  int32_t x = -1;
  int j = 0, nk = 1;
  if (root < B.n) {
    if (lane == 0u) { x = root; j = 1; }
  } else {
    const int k8 = B.cut[root - B.n].pick[8];
    nk = 2;
    if (lane < 2u) {
      x = lane == 0u ? B.node[root].left : B.node[root].right;
      j = lane == 0u ? k8 : 8 - k8;
    }
  }
  bool leaf = false;
  for (;;) {
    int k = 0;
    if (x >= B.n) {
      const Cut *c = B.cut + (x - B.n);
      while (j > 1 && c->pick[j] == 0) --j;
      if (j > 1) k = c->pick[j];
      else leaf = c->pick[0] != 0;
    } else {
      leaf = x >= 0;
    }
    const uint32_t split = (__ballot_sync(group, k > 0) >> shift) & 0xFFu;
    if (split == 0u) break;
    if (k > 0) {
      const int at = nk + __popc(split & ((1u << lane) - 1u));
      xn[at] = B.node[x].right;
      xj[at] = j - k;
      x = B.node[x].left;
      j = k;
    }
    __syncwarp(group);
    const int nk2 = nk + __popc(split);
    if ((int)lane >= nk && (int)lane < nk2) {
      x = xn[lane];
      j = xj[lane];
    }
    nk = nk2;
    __syncwarp(group);
  }
  const Box box = B.node[root].box;
  Box kb = box;
  if (x >= 0) kb = B.node[x].box;
  // slots: repeatedly the (child, slot) with the child farthest along the slot's diagonal
  float off[3];
  for (int k = 0; k < 3; ++k) off[k] = 0.5f * (kb.lo[k] + kb.hi[k]) - 0.5f * (box.lo[k] + box.hi[k]);
  uint32_t free_slots = 0xFFu;
  int slot = -1;
  for (int r = 0; r < nk; ++r) {
    float best = -INFINITY;
    uint32_t at = lane << 4;  // (lane, slot)
    if (x >= 0 && slot < 0) {
      at |= (uint32_t)__ffs(free_slots) - 1u;
      for (int q = 0; q < 8; ++q) {
        const float v = ((q & 1) ? off[0] : -off[0]) + ((q & 2) ? off[1] : -off[1]) + ((q & 4) ? off[2] : -off[2]);
        if (((free_slots >> q) & 1u) && v > best) { best = v; at = (lane << 4) | (uint32_t)q; }
      }
    } else {
      at |= 0x100u;  // not a candidate
    }
    for (int d = 1; d < 8; d <<= 1) {
      const float ob = __shfl_xor_sync(group, best, d);
      const uint32_t oa = __shfl_xor_sync(group, at, d);
      const bool me = !(at & 0x100u), other = !(oa & 0x100u);
      if (other && (!me || ob > best || (ob == best && oa < at))) { best = ob; at = oa; }
    }
    if ((at >> 4) == lane) slot = (int)(at & 7u);
    free_slots &= ~(1u << (at & 7u));
  }
  // the node's centre, relative to the scene's
  float mid[3];
  bool fits = true;
  for (int k = 0; k < 3; ++k) {
    const float lo = box.lo[k] - B.centre[k], hi = box.hi[k] - B.centre[k];
    mid[k] = 0.5f * lo + 0.5f * hi;
    fits = fits && fmaxf(fabsf(lo), fabsf(hi)) <= 1.0e37f;  // the stored planes are finite
  }
  const int cnt = x < 0 || !leaf ? 0 : (x < B.n ? 1 : (int)B.cut[x - B.n].prims);
  const uint32_t imask = __reduce_or_sync(group, x >= 0 && !leaf ? 1u << slot : 0u);
  const uint32_t tvalid = __reduce_or_sync(group, cnt ? ((1u << cnt) - 1u) << (3 * slot) : 0u);
  const uint32_t ninner = __popc(imask), ntris = __popc(tvalid);
  uint32_t cb = 0u, tb = 0u;
  if (lane == 0u) {
    if (ninner) cb = atomicAdd(&B.ctr[kCNodes], ninner);
    if (ntris) tb = atomicAdd(&B.ctr[kCTris], ntris);
  }
  cb = __shfl_sync(group, cb, (int)shift);
  tb = __shfl_sync(group, tb, (int)shift);
  if (cb + ninner > B.cap_nodes || tb + ntris > (uint32_t)B.n || !fits) {
    if (lane == 0u) B.ctr[kCFail] = 1u;
    return;
  }
  uint32_t *o = B.wnodes + (size_t)w * kWideWords;
  if (x < 0) {  // an empty slot: neither mask names it
    int skip = (int)lane - nk;
    uint32_t f = free_slots;
    while (skip-- > 0) f &= f - 1u;
    const int e = __ffs(f) - 1;
    for (int k = 0; k < 3; ++k) o[8 + 3 * e + k] = 0u;
  } else {
    for (int k = 0; k < 3; ++k) {
      const float lo = __double2float_rd((double)kb.lo[k] - B.centre[k] - mid[k]);
      const float hi = __double2float_ru((double)kb.hi[k] - B.centre[k] - mid[k]);
      o[8 + 3 * slot + k] = (plane_above(-lo) ^ 0x8000u) | (plane_above(hi) << 16);
    }
    if (leaf) {
      uint32_t at = tb + __popc(tvalid & ((1u << (3 * slot)) - 1u));
      int32_t st[4];
      int sp = 0;
      st[sp++] = x;
      while (sp > 0) {
        const int32_t y = st[--sp];
        if (y >= B.n) {
          st[sp++] = B.node[y].right;
          st[sp++] = B.node[y].left;
          continue;
        }
        const int64_t t = B.node[y].left;
        F4 a = load_f4(B.tris, 3 * t), bb = load_f4(B.tris, 3 * t + 1);
        const F4 c = load_f4(B.tris, 3 * t + 2);
        const bool out = sticks_out(B, B.node[y].box);
        if (out) B.ctr[kCOut] = 1u;
        bb.w = __uint_as_float((__float_as_uint(a.w) & 1u) | (out ? kWideOutside : 0u));
        a.w = __int_as_float((int)t);
        B.wtris[3 * (size_t)at] = a;
        B.wtris[3 * (size_t)at + 1] = bb;
        B.wtris[3 * (size_t)at + 2] = c;
        ++at;
      }
    } else {
      B.wroot[cb + __popc(imask & ((1u << slot) - 1u))] = x;
    }
  }
  if (lane == 0u) {
    for (int k = 0; k < 3; ++k) o[k] = __float_as_uint(mid[k]);
    o[3] = cb;
    o[4] = tb;
    o[5] = imask;
    o[6] = tvalid;
    o[7] = 0u;
  }
}

__global__ void __launch_bounds__(128) k_bvh_emit(Build B, int level) {
  __shared__ int32_t xn[128], xj[128];
  if (B.ctr[kCFail] != 0u) return;  // an earlier level did not fit
  const uint32_t w0 = B.ctr[kCLevel + level], w1 = B.ctr[kCLevel + level + 1];
  const uint32_t g = threadIdx.x & ~7u;
  for (uint32_t base = w0 + blockIdx.x * 16u; base < w1; base += gridDim.x * 16u) {
    const uint32_t w = base + threadIdx.x / 8u;
    emit_node(B, w, w < w1, xn + g, xj + g);
    __syncwarp();
  }
}

// ---- small scenes -------------------------------------------------------------------------

// Up to kSmall triangles: the whole build in one block, so that preparing a small scene costs one
// launch (36 triangles: scene creation 0.33 -> 0.25 ms with the kernels above, warm 155 -> 118 us since
// lanes share a cluster's candidates and the climb stays in the block).  It is a chain of short dependent
// steps, bound by their latency: 36 triangles 55 us, 200 83, 2,048 239.  Same order, same clusters as
// the kernels above.
struct SmallShared {
  TailShared tail;
  uint64_t key[kSmall];
  uint16_t val[kSmall];
  uint32_t bounds[6];
  uint32_t more;
};

__global__ void __launch_bounds__(1024) k_bvh_small(Build B) {
  extern __shared__ __align__(16) unsigned char smem[];
  SmallShared &S = *reinterpret_cast<SmallShared *>(smem);
  const uint32_t n = (uint32_t)B.n;
  if (threadIdx.x < kNumC) B.ctr[threadIdx.x] = threadIdx.x == kCNodes ? 1u : 0u;
  if (threadIdx.x < 6) S.bounds[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
  __syncthreads();
  centre_bounds(B, threadIdx.x, 1024, S.bounds);
  __syncthreads();
  uint32_t m = 2;
  while (m < n) m <<= 1;
  for (uint32_t i = threadIdx.x; i < m; i += 1024) {
    S.key[i] = i < n ? morton_key(B, S.bounds, i) : ~0ull;
    S.val[i] = (uint16_t)i;
  }
  __syncthreads();
  // bitonic sort, ties by index: the order of the radix sort
  for (uint32_t size = 2; size <= m; size <<= 1)
    for (uint32_t step = size >> 1; step > 0; step >>= 1) {
      for (uint32_t p = threadIdx.x; p < m / 2; p += 1024) {
        const uint32_t i = 2 * p - (p & (step - 1)), j = i + step;
        const bool up = (i & size) == 0;
        const bool gt = S.key[i] > S.key[j] || (S.key[i] == S.key[j] && S.val[i] > S.val[j]);
        if (gt == up) {
          const uint64_t tk = S.key[i]; S.key[i] = S.key[j]; S.key[j] = tk;
          const uint16_t tv = S.val[i]; S.val[i] = S.val[j]; S.val[j] = tv;
        }
      }
      __syncthreads();
    }
  uint32_t *arrived = reinterpret_cast<uint32_t *>(S.key);  // the keys have been used
  for (uint32_t i = threadIdx.x; i < n; i += 1024) {
    arrived[i] = 0u;
    S.tail.sb[i] = make_leaf(B, i, S.val[i]);
    S.tail.id[i] = (int32_t)i;
  }
  __syncthreads();
  cluster_tail(B, S.tail, (int)n, n);
  for (uint32_t i = threadIdx.x; i < n; i += 1024) climb<true>(B, i, arrived);
  __syncthreads();
  uint32_t w0 = 0u, w1 = 1u;
  int level = 0;
  for (; level < kMaxLevels && w0 < w1; ++level) {
    for (uint32_t base = w0; base < w1; base += 128u) {
      const uint32_t w = base + threadIdx.x / 8u;
      emit_node(B, w, w < w1, S.tail.id + (threadIdx.x & ~7u), S.tail.nn + (threadIdx.x & ~7u));
      __syncwarp();
    }
    __threadfence_block();
    __syncthreads();
    if (threadIdx.x == 0) S.more = __ldcg(&B.ctr[kCFail]) ? w1 : __ldcg(&B.ctr[kCNodes]);
    __syncthreads();
    w0 = w1;
    w1 = S.more;
  }
  if (threadIdx.x == 0 && w0 < w1) B.ctr[kCFail] = 1u;  // deeper than the traversal's stack
}

size_t up256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace

// Wide nodes at most.  A node with an inner child X has five children or more: with four slots free, the half of X
// that has the fewer children in X's own cut (four at most) would take their places and the other half, Y,
// that of X, at no more cost since Y's area is at most X's.  A node without one holds at least four
// triangles (three fit a leaf child, and three tests cost less than a node).  4 I + 3 L < n and 4 L <= n bound
// I + L by 5 n / 16.  Where areas are equal (a scene without any, overflown ones) the program may leave X
// closed and a build may exceed this; it then reports so and the scene keeps the kd-tree.
// (Measured: 0.07 to 0.13 nodes per triangle from 500 triangles on.)
int64_t wide_node_cap(int64_t ntri) { return ntri <= 0 ? 0 : 5 * ntri / 16 + 8; }

namespace {
size_t place_scratch(Build &B, int64_t n, char *base) {
  const size_t N = (size_t)n;
  const size_t radix_blocks = (N + kRadixTile - 1) / kRadixTile;
  size_t off = 0;
  auto take = [&](size_t bytes) { char *p = base + off; off += up256(bytes); return p; };
  B.node = (BNode *)take(2 * N * sizeof(BNode));
  B.parent = (int32_t *)take(2 * N * 4);
  B.arrived = (uint32_t *)take(N * 4);
  B.cut = (Cut *)take(N * sizeof(Cut));
  B.wroot = (int32_t *)take((size_t)wide_node_cap(n) * 4 + 64);
  if (n <= kSmall) return off;
  B.bounds = (uint32_t *)take(64);
  for (int k = 0; k < 2; ++k) {
    B.key[k] = (uint64_t *)take(N * 8);
    B.val[k] = (int32_t *)take(N * 4);
    B.cl[k] = (int32_t *)take(N * 4);
  }
  B.hist = (uint32_t *)take(radix_blocks * 256 * 4);
  B.nn = (int32_t *)take(N * 4);
  B.bsum = (uint2 *)take((N / 1024 + 8) * 8);
  return off;
}
}  // namespace

// Bytes of scratch that the build of n triangles takes.
size_t wide_scratch(int64_t n) {
  Build B;
  return n > 0 ? place_scratch(B, n, nullptr) : 0;
}

void wide_result(const uint32_t *h, int64_t n, uint32_t *nodes, bool *ok, bool *outside) {
  *ok = h[kCFail] == 0u && h[kCTris] == (uint32_t)n;  // (a tree deeper than the traversal's stack lacks triangles)
  *nodes = *ok ? h[kCNodes] : 0u;
  *outside = *ok && h[kCOut] != 0u;
}

int wide_build(const F4 *tris, int64_t n, const SceneView &view, void *wnodes, F4 *wtris, void *scratch, uint32_t *ctr,
               cudaStream_t st) {
  if (n <= 0) return MGPU_OK;
  Build B;
  memset(&B, 0, sizeof(B));
  B.ctr = ctr;
  B.n = (int32_t)n;
  B.tris = tris;
  B.wnodes = (uint32_t *)wnodes;
  B.wtris = wtris;
  for (int k = 0; k < 3; ++k) {
    B.centre[k] = view.wcentre[k];
    B.bmin[k] = view.bmin[k];
    B.bmax[k] = view.bmax[k];
  }
  B.cap_nodes = (uint32_t)wide_node_cap(n);
  const int radix_blocks = (int)((n + kRadixTile - 1) / kRadixTile);
  cudaError_t e = cudaSuccess;
  place_scratch(B, n, (char *)scratch);
  const int sms = device_sm_count();
  uint64_t launches = 0;
  auto grid = [&](int64_t items, int block) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((items + block - 1) / block, (int64_t)sms * 16));
  };
  uint32_t h[kNumC];
  auto counters = [&]() {
    cudaError_t r = cudaGetLastError();
    if (r == cudaSuccess) r = cudaMemcpyAsync(h, B.ctr, sizeof(h), cudaMemcpyDeviceToHost, st);
    return r == cudaSuccess ? cudaStreamSynchronize(st) : r;
  };
  if (n <= kSmall) {
    e = cudaFuncSetAttribute((const void *)k_bvh_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(SmallShared));
    if (e == cudaSuccess) {
      k_bvh_small<<<1, 1024, sizeof(SmallShared), st>>>(B);
      ++launches;
      e = cudaGetLastError();
    }
  } else {
    k_bvh_init<<<1, 128, 0, st>>>(B);
    k_bvh_bounds<<<grid(n, 256), 256, 0, st>>>(B);
    k_bvh_morton<<<grid(n, 256), 256, 0, st>>>(B);
    launches += 3;
    int cur = 0;
    for (int shift = 0; shift < kMortonBits; shift += 8, cur ^= 1) {
      k_bvh_radix_count<<<radix_blocks, 256, 0, st>>>(B.key[cur], B.n, shift, B.hist);
      k_bvh_radix_scan<<<1, 1024, 0, st>>>(B.hist, (uint32_t)radix_blocks * 256u);
      k_bvh_radix_scatter<<<radix_blocks, 256, 0, st>>>(B.key[cur], B.val[cur], B.n, shift, B.hist, B.key[cur ^ 1],
                                                        B.val[cur ^ 1]);
      launches += 3;
    }
    k_bvh_leaves<<<grid(n, 256), 256, 0, st>>>(B, B.val[cur]);
    ++launches;
    // rounds of clustering until one block can finish; the count is read every four rounds
    int64_t count = n;
    while (count > kTailMax && e == cudaSuccess) {
      for (int r = 0; r < 4; ++r) {
        k_bvh_nearest<<<grid(count, kPlocBlock), kPlocBlock, 0, st>>>(B);
        k_bvh_merge_count<<<grid(count, 1024), 1024, 0, st>>>(B);
        k_bvh_merge_scan<<<1, 1024, 0, st>>>(B);
        k_bvh_merge<<<grid(count, 1024), 1024, 0, st>>>(B);
        k_bvh_round<<<1, 1, 0, st>>>(B);
        launches += 5;
      }
      e = counters();
      if (e == cudaSuccess && (int64_t)h[kCCount] >= count) break;  // every round merges, so this does not happen
      if (e == cudaSuccess) count = h[kCCount];
    }
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute((const void *)k_bvh_tail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(TailShared));
    if (e == cudaSuccess && count <= kTailMax) {
      k_bvh_tail<<<1, 1024, sizeof(TailShared), st>>>(B);
      k_bvh_cut<<<grid(n, 128), 128, 0, st>>>(B);
      launches += 2;
      // wide levels until one is empty; the counters are read every eight levels
      int level = 0;
      for (bool more = true; more && level < kMaxLevels && e == cudaSuccess;) {
        for (int k = 0; k < 8 && level < kMaxLevels; ++k, ++level) {
          k_bvh_emit<<<grid((int64_t)B.cap_nodes * 8, 128), 128, 0, st>>>(B, level);
          k_bvh_level<<<1, 1, 0, st>>>(B, level + 2);
          launches += 2;
        }
        e = counters();
        if (e == cudaSuccess) more = h[kCLevel + level] != h[kCLevel + level + 1] && h[kCFail] == 0u;
      }
    }
  }
  g_launches.fetch_add(launches);
  if (e != cudaSuccess) return cuda_fail(e, "wide hierarchy build");
  return MGPU_OK;
}

}  // namespace mgpu
