// api.cu -- error reporting, host kd-tree objects, scene upload and film objects of libmgpu.
#include <string.h>
#include <sys/mman.h>
#include <unistd.h>

#include <cmath>
#include <map>
#include <mutex>
#include <new>
#include <vector>

#include "common.cuh"
#include "hd_wide.h"

namespace mgpu {

static thread_local std::string t_last_error;
std::atomic<uint64_t> g_launches{0};

void set_error(const std::string &msg) { t_last_error = msg; }
int fail(int code, const std::string &msg) {
  t_last_error = msg;
  return code;
}
int cuda_fail(cudaError_t e, const char *what) {
  t_last_error = std::string(what) + ": " + cudaGetErrorString(e);
  cudaGetLastError();  // reported here: the next call's check of its launches does not find it again
  return e == cudaErrorMemoryAllocation ? MGPU_E_NOMEM : MGPU_E_CUDA;
}

int device_sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 1;
  return n > 0 ? n : 1;
}

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Device-ready copies of the scene's triangles: tree layout with leaf-ordered records,
// triangles by id (3 x float4, v0.w = flags) and shading records (3 x float4: (n0, material),
// (n1, light), (n2, 0)).
static void stage_device_arrays(const mgpu_scene_desc *desc, mgpu_accel *a) {
  const int64_t T = desc->ntri;
  kd_device_layout(a->tree, desc->tri_v, desc->tri_flags, a->dpairs, a->ltris);
  a->tris.resize((size_t)T * 3);
  a->shade.resize((size_t)T * 3);
  for (int64_t t = 0; t < T; ++t) {
    const float *v = desc->tri_v + t * 9;
    uint32_t fl = desc->tri_flags ? desc->tri_flags[t] : 0u;
    for (int k = 0; k < 3; ++k) {
      F4 q; q.x = v[3 * k]; q.y = v[3 * k + 1]; q.z = v[3 * k + 2]; q.w = 0.0f;
      if (k == 0) memcpy(&q.w, &fl, 4);
      a->tris[3 * t + k] = q;
    }
    V3 e1 = v3(v[3] - v[0], v[4] - v[1], v[5] - v[2]);
    V3 e2 = v3(v[6] - v[0], v[7] - v[1], v[8] - v[2]);
    V3 fn = normalize(cross(e1, e2));
    int32_t mat = desc->tri_mat[t];
    int32_t li = desc->tri_light ? desc->tri_light[t] : -1;
    for (int k = 0; k < 3; ++k) {
      float4 q;
      if (desc->tri_n) {
        const float *n = desc->tri_n + t * 9 + 3 * k;
        q = make_float4(n[0], n[1], n[2], 0.0f);
      } else {
        q = make_float4(fn.x, fn.y, fn.z, 0.0f);
      }
      if (k == 0) memcpy(&q.w, &mat, 4);
      if (k == 1) memcpy(&q.w, &li, 4);
      a->shade[3 * t + k] = q;
    }
  }
}

static void register_staging(mgpu_accel *a) {
  // page-locked staging makes every later upload a direct DMA; failure just leaves it pageable
  if (a->registered) return;
  a->registered = true;
  auto reg = [](void *p, size_t n) {
    if (n) cudaHostRegister(p, n, cudaHostRegisterDefault);
  };
  reg(a->dpairs.data(), a->dpairs.size() * sizeof(Pair));
  reg(a->ltris.data(), a->ltris.size() * sizeof(F4));
  reg(a->tris.data(), a->tris.size() * sizeof(F4));
  reg(a->shade.data(), a->shade.size() * sizeof(float4));
  cudaGetLastError();  // clear a failed registration
}

// Offsets of the arrays in a scene's one device allocation (256-byte aligned each).
struct SceneLayout {
  size_t off_pairs, off_refs, off_tris, off_shade, off_mats, off_lights, off_uv, off_texrec, off_texels, off_sph,
      off_wnodes, off_wtris, off_err, total;
};
// uv_tris: triangles with uploaded uvs (0 or all); ntex textures holding texels texels in all;
// nsph analytic spheres (2 float4 each, and 3 shading records after the triangles'); wide: with the 8-wide
// hierarchy, whose build takes its scratch where the kd-tree and the shading records (off_pairs to off_mats)
// are uploaded afterwards: nothing is allocated for it, and freed, which would wait for the whole device
static SceneLayout scene_layout(const mgpu_accel *a, int32_t nmat, int32_t nlight, int64_t uv_tris = 0,
                                int32_t ntex = 0, uint64_t texels = 0, int32_t nsph = 0, bool wide = true) {
  SceneLayout L;
  L.off_tris = 0;
  L.off_pairs = align_up(L.off_tris + std::max<size_t>(a->tris.size(), 1) * sizeof(F4), 256);
  L.off_refs = align_up(L.off_pairs + a->dpairs.size() * sizeof(Pair), 256);
  L.off_shade = align_up(L.off_refs + std::max<size_t>(a->ltris.size(), 1) * sizeof(F4), 256);
  L.off_mats = align_up(L.off_shade + std::max<size_t>(a->shade.size() + 3 * (size_t)std::max(nsph, 0), 1) *
                                          sizeof(float4), 256);
  if (wide) L.off_mats = std::max(L.off_mats, align_up(L.off_pairs + wide_scratch(a->ntri), 256));
  L.off_lights = align_up(L.off_mats + (size_t)std::max(nmat, 0) * 16 * sizeof(float), 256);
  L.off_uv = align_up(L.off_lights + std::max<size_t>((size_t)std::max(nlight, 0), 1) * 32 * sizeof(float), 256);
  L.off_texrec = align_up(L.off_uv + (size_t)std::max<int64_t>(uv_tris, 0) * 3 * sizeof(float2), 256);
  L.off_texels = align_up(L.off_texrec + (size_t)std::max(ntex, 0) * 2 * sizeof(float4), 256);
  L.off_sph = align_up(L.off_texels + (size_t)texels * sizeof(float4), 256);
  L.off_wnodes = align_up(L.off_sph + (size_t)std::max(nsph, 0) * 2 * sizeof(float4), 256);
  L.off_wtris = align_up(L.off_wnodes + (wide ? (size_t)wide_node_cap(a->ntri) * kWideWords * sizeof(uint32_t) : 0), 256);
  L.off_err = align_up(L.off_wtris + (wide ? (size_t)a->ntri * 3 * sizeof(F4) : 0), 256);
  L.total = L.off_err + 256;
  return L;
}

// Film error estimate.  Per pixel with n > 1 samples: the sample variance of the per-sample
// luminance (r+g+b)/3 from the film's sum and sum of squares, divided by n, is the variance
// of the pixel's mean; the film's estimate is the square root of its average over those
// pixels (the expected RMSE of the image against the converged one).  Each film is reduced by
// kErrBlocks blocks in a fixed order, so the value is deterministic.
struct FilmRef {
  const float4 *sum;
  const float4 *c;
  int64_t npix;
  int64_t first = 0;  // its first block among those of all films
};
constexpr int kErrBlocks = 64, kErrThreads = 256;

// Blocks that reduce one film: one per 2,048 pixels within [64, 1024] (by the film alone, so that its value does
// not depend on the films beside it; each film has its own number, or one large film would make a
// thousand idle blocks and 16 KB of partial sums of every small one).  64 for every film left the GPU idle on large ones (483,003
// pixels: 212 -> 87 us a call, with two divisions a pixel instead of five).
constexpr int kErrMaxBlocks = 1024;
__host__ __device__ inline int err_blocks(int64_t npix) {
  const int64_t b = (npix + 2047) / 2048;
  return b < kErrBlocks ? kErrBlocks : (b > kErrMaxBlocks ? kErrMaxBlocks : (int)b);
}

// sum over the block in a fixed tree
__device__ __forceinline__ void err_reduce(double &a, double &c) {
  __shared__ double sa[kErrThreads], sc[kErrThreads];
  sa[threadIdx.x] = a;
  sc[threadIdx.x] = c;
  __syncthreads();
  for (int w = kErrThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      sa[threadIdx.x] += sa[threadIdx.x + w];
      sc[threadIdx.x] += sc[threadIdx.x + w];
    }
    __syncthreads();
  }
  a = sa[0];
  c = sc[0];
}

__global__ void __launch_bounds__(kErrThreads) k_film_error_partial(const FilmRef *films, int n, double2 *partial) {
  int at = 0;  // the film of this block: the last that begins no later
  for (int hi = n - 1; at < hi;) {
    const int mid = (at + hi + 1) >> 1;
    if (films[mid].first <= (int64_t)blockIdx.x) at = mid; else hi = mid - 1;
  }
  const FilmRef f = films[at];
  const int nb = err_blocks(f.npix);
  double acc = 0.0, cnt = 0.0;
  for (int64_t i = ((int64_t)blockIdx.x - f.first) * kErrThreads + threadIdx.x; i < f.npix; i += (int64_t)nb * kErrThreads) {
    const float4 S = f.sum[i], C = f.c[i];
    const double n = S.w;
    if (n > 1.0) {
      // two divisions (FP64 runs at two a clock and SM): 1 / n, and the variance of the mean,
      // (m2 - mean^2) n / (n - 1) / n
      const double inv = 1.0 / n;
      const double mean = ((((double)S.x - C.x) + ((double)S.y - C.y)) + ((double)S.z - C.z)) * (inv * (1.0 / 3.0));
      acc += fmax((double)C.w * inv - mean * mean, 0.0) / (n - 1.0);
      cnt += 1.0;
    }
  }
  err_reduce(acc, cnt);
  if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(acc, cnt);
}

__global__ void __launch_bounds__(kErrThreads) k_film_error_final(const FilmRef *films, const double2 *partial,
                                                                  double *out) {
  const FilmRef f = films[blockIdx.x];
  const int nb = err_blocks(f.npix);
  double a = 0.0, c = 0.0;
  for (int b = threadIdx.x; b < nb; b += kErrThreads) {
    const double2 p = partial[f.first + b];
    a += p.x;
    c += p.y;
  }
  err_reduce(a, c);
  if (threadIdx.x == 0) out[blockIdx.x] = c > 0.0 ? sqrt(a / c) : INFINITY;
}

// Reinhard tone map (ReinhardToneMap::map, M/renderers/tonemaps/ReinhardToneMap.cpp:25-94) of the
// film's per-pixel means, in FP64: key = exp(mean log(1e-7 + Y)), white = 1 / max(Y)^2 (the
// unscaled maximum, as the reference has it), Y' = L (1 + L white) / (1 + L) with L = 0.18 Y /
// key, chromaticity kept, gamma 2.22, clamp to [0, 255] and truncate (a NaN, as from an
// all-black pixel, becomes 0).  sRGB <-> XYZ matrices as ColorUtils.cpp:115-133 (the standard
// D65 pair).
__device__ const double kRgbToXyz[9] = {0.41245322014416, 0.35757958129350, 0.18042258997054,
                                        0.21267112134122, 0.71515920531078, 0.07216877677613,
                                        0.01933381646199, 0.11919354020663, 0.95022692228971};
__device__ const double kXyzToRgb[9] = {3.240479, -1.537150, -0.498535, -0.969256, 1.875992,
                                        0.041556, 0.055648, -0.204043, 1.057311};

struct ToneSrc {
  FilmRef f;
  const unsigned long long *fx;  // filtered sums, or null for the per-pixel mean
};

__device__ __forceinline__ void film_xyz(const ToneSrc &t, int64_t i, double &X, double &Y, double &Z) {
  double r = 0.0, g = 0.0, b = 0.0;
  if (t.fx) {
    const double w = (double)t.fx[4 * i + 3];
    if (w > 0.0) {
      r = (double)t.fx[4 * i] / w;
      g = (double)t.fx[4 * i + 1] / w;
      b = (double)t.fx[4 * i + 2] / w;
    }
  } else {
    const float4 S = t.f.sum[i], C = t.f.c[i];
    const double n = S.w;
    if (n > 0.0) {
      r = ((double)S.x - C.x) / n;
      g = ((double)S.y - C.y) / n;
      b = ((double)S.z - C.z) / n;
    }
  }
  X = kRgbToXyz[0] * r + kRgbToXyz[1] * g + kRgbToXyz[2] * b;
  Y = kRgbToXyz[3] * r + kRgbToXyz[4] * g + kRgbToXyz[5] * b;
  Z = kRgbToXyz[6] * r + kRgbToXyz[7] * g + kRgbToXyz[8] * b;
}

__global__ void __launch_bounds__(kErrThreads) k_tonemap_reduce(ToneSrc t, double2 *partial) {
  double lsum = 0.0, ymax = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kErrThreads + threadIdx.x; i < t.f.npix;
       i += (int64_t)kErrBlocks * kErrThreads) {
    double X, Y, Z;
    film_xyz(t, i, X, Y, Z);
    lsum += log(1e-7 + Y);
    ymax = fmax(ymax, Y);
  }
  __shared__ double sa[kErrThreads], sm[kErrThreads];
  sa[threadIdx.x] = lsum;
  sm[threadIdx.x] = ymax;
  __syncthreads();
  for (int w = kErrThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      sa[threadIdx.x] += sa[threadIdx.x + w];
      sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + w]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(sa[0], sm[0]);
}

__global__ void k_tonemap_map(ToneSrc t, const double2 *partial, uchar4 *out) {
  const FilmRef &f = t.f;
  __shared__ double s_scale, s_white;
  if (threadIdx.x == 0) {
    double a = 0.0, m = 0.0;
    for (int b = 0; b < kErrBlocks; ++b) {
      a += partial[b].x;
      m = fmax(m, partial[b].y);
    }
    const double key = exp(a / (double)f.npix);
    s_scale = key <= 0.0 ? 0.0 : 0.18 / key;
    s_white = m <= 0.0 ? 0.0 : 1.0 / (m * m);
  }
  __syncthreads();
  const double scale = s_scale, white = s_white, corr = 1.0 / 2.22;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < f.npix; i += (int64_t)gridDim.x * blockDim.x) {
    double X, Y, Z;
    film_xyz(t, i, X, Y, Z);
    const double s = X + Y + Z;
    const double cx = X / s, cy = Y / s;  // xyY chromaticity (NaN for a black pixel)
    const double lum = scale * Y;
    const double Yd = lum * (1.0 + lum * white) / (1.0 + lum);
    const double Xd = Yd * cx / cy, Zd = Yd * (1.0 - cx - cy) / cy;
    double rgb[3];
    for (int k = 0; k < 3; ++k)
      rgb[k] = 255.0 * pow(kXyzToRgb[3 * k] * Xd + kXyzToRgb[3 * k + 1] * Yd + kXyzToRgb[3 * k + 2] * Zd, corr);
    unsigned char o[3];
    for (int k = 0; k < 3; ++k) {
      const double v = rgb[k];
      o[k] = v >= 255.0 ? 255 : (v <= 0.0 ? 0 : (v == v ? (unsigned char)v : 0));
    }
    out[i] = make_uchar4(o[0], o[1], o[2], 255);
  }
}

// Scratch of the film reads of one host thread, kept for its next read and released when the thread exits: a
// device buffer and a page-locked host buffer, each grown to the largest need.  A film read is
// synchronous, so the thread's next one finds them free.
struct ReadScratch {
  void *d = nullptr, *h = nullptr;
  size_t d_bytes = 0, h_bytes = 0;
  int device = -1;
  void release_device() {
    if (!d) return;
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != device) cudaSetDevice(device);
    cudaFree(d);
    if (cur != device) cudaSetDevice(cur);
    d = nullptr;
    d_bytes = 0;
  }
  cudaError_t device_buffer(size_t need, void **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (d && (dev != device || need > d_bytes)) release_device();
    if (!d) {
      if ((e = cudaMalloc(&d, need)) != cudaSuccess) {
        d = nullptr;
        return e;
      }
      d_bytes = need;
      device = dev;
    }
    *out = d;
    return cudaSuccess;
  }
  // portable and mapped: a kernel of any device writes there
  cudaError_t host_buffer(size_t need, void **out) {
    if (h && need > h_bytes) {
      cudaFreeHost(h);
      h = nullptr;
      h_bytes = 0;
    }
    if (!h) {
      const cudaError_t e = cudaHostAlloc(&h, need, cudaHostAllocPortable | cudaHostAllocMapped);
      if (e != cudaSuccess) {
        h = nullptr;
        return e;
      }
      h_bytes = need;
    }
    *out = h;
    return cudaSuccess;
  }
  ~ReadScratch() {
    release_device();
    if (h) cudaFreeHost(h);
  }
};
static thread_local ReadScratch t_read;

// Results up to this size are written by the kernel into page-locked staging of the thread and copied by the
// host, which takes 100 KB in the 10 us that a copy by the device costs more (means of 37 x 23 pixels 26.5 us,
// 72 x 72 32.0; by the device 76 x 76 40.8, 256 x 256 45).
constexpr size_t kStageBytes = (size_t)1 << 17;

// Makes the pages of a result array, while the stream still works; the array keeps its contents.  A copy by the
// device faults at every page that is not there, at 20 us each (24 MB: 2 to 9 ms), and at pages that are but
// that nobody has touched for a while (10 MB into memory of a result a second old: 2 to 3.4 ms, now 0.3).  So
// they are made in one request and then touched.  (Touched by a read first, a new page would be mapped
// twice, for reading and at the write, and the GPU's translations wait for that: 9 ms too.)  A system that
// does not know the request refuses it, and the copy faults as before.
static void make_pages(void *dst, size_t n) {
#ifndef MADV_POPULATE_WRITE
  constexpr int MADV_POPULATE_WRITE = 23;
#endif
  static const uintptr_t page = (uintptr_t)std::max(sysconf(_SC_PAGESIZE), 4096L);
  const uintptr_t first = (uintptr_t)dst / page * page, end = ((uintptr_t)dst + n + page - 1) / page * page;
  if (n < kStageBytes || madvise((void *)first, end - first, MADV_POPULATE_WRITE) != 0) return;
  for (uintptr_t p = first; p < end; p += page) (void)*(const volatile char *)std::max(p, (uintptr_t)dst);
}

// Device memory into the caller's array; returns when it is there.  Into ordinary memory whose pages exist a GB300
// copies as fast as into page-locked memory (24 MB: 0.19 ms), without staging.  An array that is
// page-locked in part is refused by the copy, and filled through page-locked staging.
static cudaError_t to_host(void *dst, const void *src, size_t n, cudaStream_t st) {
  make_pages(dst, n);
  cudaError_t e = cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st);
  if (e == cudaErrorInvalidValue) {
    cudaGetLastError();
    constexpr size_t kStage = (size_t)4 << 20;
    void *h = nullptr;
    e = t_read.host_buffer(std::min(n, kStage), &h);
    for (size_t k = 0; k < n && e == cudaSuccess; k += kStage) {
      const size_t m = std::min(kStage, n - k);
      e = cudaMemcpyAsync(h, (const char *)src + k, m, cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      if (e == cudaSuccess) memcpy((char *)dst + k, h, m);
    }
    return e;
  }
  return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

// Blocks of mgpu_host_alloc that are not freed: address, bytes.
static std::mutex g_host_mu;
static std::map<uintptr_t, size_t> &g_host_blocks = *new std::map<uintptr_t, size_t>;  // outlives the program's statics

// Whether the device may write the n bytes at p itself: they lie in one block of mgpu_host_alloc, aligned for
// its stores.  Other page-locked memory is not asked for: the runtime tells what the first byte is, not how
// far its registration reaches.  (Such a block has one address on host and device.)
static bool device_writes(const void *p, size_t n, size_t align) {
  const uintptr_t at = (uintptr_t)p;
  if (at % align) return false;
  std::lock_guard<std::mutex> lock(g_host_mu);
  auto it = g_host_blocks.upper_bound(at);
  if (it == g_host_blocks.begin()) return false;
  --it;
  const size_t off = at - it->first;
  return off <= it->second && n <= it->second - off;
}

}  // namespace mgpu

mgpu_accel::~mgpu_accel() {
  if (!registered) return;
  for (void *p : {(void *)dpairs.data(), (void *)ltris.data(), (void *)tris.data(), (void *)shade.data()})
    if (p) cudaHostUnregister(p);
  cudaGetLastError();
}

using namespace mgpu;

extern "C" {

const char *mgpu_last_error(void) { return t_last_error.c_str(); }
int mgpu_version(void) { return 1; }
uint64_t mgpu_launch_count(void) { return g_launches.load(); }

int mgpu_accel_build(const mgpu_scene_desc *desc, const mgpu_kd_params *params, mgpu_accel **out) {
  if (!desc || !out) return fail(MGPU_E_INVALID, "mgpu_accel_build: null argument");
  if (desc->ntri < 0 || (desc->ntri > 0 && !desc->tri_v)) return fail(MGPU_E_INVALID, "mgpu_accel_build: bad geometry");
  KdParams p;
  if (params) {
    p.min_prims = params->min_prims;
    p.max_depth = params->max_depth;
    p.cost_traversal = params->cost_traversal;
    p.empty_bias = params->empty_bias;
    p.threads = params->threads;
  }
  if (desc->ntri > 0 && !desc->tri_mat) return fail(MGPU_E_INVALID, "mgpu_accel_build: missing material indices");
  mgpu_accel *a = new (std::nothrow) mgpu_accel();
  if (!a) return fail(MGPU_E_NOMEM, "mgpu_accel_build: out of host memory");
  const char *err = nullptr;
  try {
    if (!kd_build(desc->tri_v, desc->ntri, p, a->tree, &err)) {
      delete a;
      return fail(MGPU_E_INVALID, std::string("mgpu_accel_build: ") + err);
    }
    a->ntri = desc->ntri;
    stage_device_arrays(desc, a);
  } catch (const std::bad_alloc &) {
    delete a;
    return fail(MGPU_E_NOMEM, "mgpu_accel_build: out of host memory");
  }
  *out = a;
  return MGPU_OK;
}

int mgpu_accel_stats(const mgpu_accel *a, mgpu_kd_stats *o) {
  if (!a || !o) return fail(MGPU_E_INVALID, "mgpu_accel_stats: null argument");
  const KdLog &l = a->tree.log;
  o->no_internal = l.no_internal;
  o->no_leaves = l.no_leaves;
  o->min_depth = l.min_depth;
  o->max_depth = l.max_depth;
  o->sum_depth = l.sum_depth;
  o->min_prims = l.min_prims;
  o->max_prims = l.max_prims;
  o->sum_prims = l.sum_prims;
  o->node_pairs = a->tree.pairs.size();
  o->refs = a->tree.refs.size();
  o->bytes_nodes = a->tree.pairs.size() * sizeof(Pair);
  o->bytes_refs = a->tree.refs.size() * sizeof(uint32_t);
  o->build_seconds = a->tree.build_seconds;
  return MGPU_OK;
}

int mgpu_accel_serialize(const mgpu_accel *a, int32_t *kind, float *split, int32_t *count, int32_t *prims,
                         int64_t *n_nodes, int64_t *n_prims) {
  if (!a) return fail(MGPU_E_INVALID, "mgpu_accel_serialize: null accel");
  kd_serialize(a->tree, kind, split, count, prims, n_nodes, n_prims);
  return MGPU_OK;
}

int mgpu_accel_destroy(mgpu_accel *a) {
  delete a;
  return MGPU_OK;
}

int mgpu_scene_create(const mgpu_scene_desc *desc, const mgpu_accel *accel, void *stream, mgpu_scene **out) {
  return scene_create(desc, accel, stream, UINT64_MAX, out);
}

}  // extern "C"

namespace mgpu {

int scene_create(const mgpu_scene_desc *desc, const mgpu_accel *accel, void *stream, uint64_t limit, mgpu_scene **out) {
  if (!desc || !accel || !out) return fail(MGPU_E_INVALID, "mgpu_scene_create: null argument");
  if (desc->ntri != accel->ntri) return fail(MGPU_E_INVALID, "mgpu_scene_create: accel built for another triangle count");
  if (desc->ntri > 0 && (!desc->tri_v || !desc->tri_mat)) return fail(MGPU_E_INVALID, "mgpu_scene_create: missing arrays");
  if (desc->nmat <= 0 || !desc->materials) return fail(MGPU_E_INVALID, "mgpu_scene_create: at least one material required");
  if (desc->nlight < 0 || (desc->nlight > 0 && !desc->lights)) return fail(MGPU_E_INVALID, "mgpu_scene_create: bad lights");
  const int64_t T = desc->ntri;
  for (int64_t t = 0; t < T; ++t) {
    if (desc->tri_mat[t] < 0 || desc->tri_mat[t] >= desc->nmat)
      return fail(MGPU_E_INVALID, "mgpu_scene_create: material index out of range at triangle " + std::to_string(t));
    if (desc->tri_light && (desc->tri_light[t] < -1 || desc->tri_light[t] >= desc->nlight))
      return fail(MGPU_E_INVALID, "mgpu_scene_create: light index out of range at triangle " + std::to_string(t));
  }
  for (int i = 0; i < desc->nmat; ++i) {
    float ty = desc->materials[16 * i];
    if (!(ty == 0.0f || ty == 1.0f || ty == 2.0f))
      return fail(MGPU_E_INVALID, "mgpu_scene_create: unknown material type at material " + std::to_string(i));
  }
  // device light records: the 16-float base record, then the 16-float extension
  std::vector<float> lrec((size_t)std::max(desc->nlight, 0) * 32, 0.0f);
  for (int i = 0; i < desc->nlight; ++i) {
    memcpy(&lrec[32 * (size_t)i], desc->lights + 16 * (size_t)i, 16 * sizeof(float));
    if (!desc->light_ext) continue;
    const float *x = desc->light_ext + 16 * (size_t)i;
    memcpy(&lrec[32 * (size_t)i + 16], x, 16 * sizeof(float));
    if (!(x[0] == 0.0f || x[0] == 1.0f || x[0] == 2.0f || x[0] == 3.0f || x[0] == 4.0f))
      return fail(MGPU_E_INVALID, "mgpu_scene_create: unknown light type at light " + std::to_string(i));
    if (x[0] == 2.0f) {
      uint32_t first, count;
      memcpy(&first, x + 8, 4);
      memcpy(&count, x + 9, 4);
      if (count == 0 || (uint64_t)first + count > (uint64_t)T)
        return fail(MGPU_E_INVALID, "mgpu_scene_create: mesh light " + std::to_string(i) + " has a bad triangle run");
    }
  }
  TexPlan tp;
  if (int rc = tex_plan(desc, tp)) return rc;
  // triangles cannot emit as a point light (it has no surface)
  if (desc->tri_light && desc->light_ext)
    for (int64_t t = 0; t < T; ++t)
      if (desc->tri_light[t] >= 0 && desc->light_ext[16 * (size_t)desc->tri_light[t]] == 3.0f)
        return fail(MGPU_E_INVALID, "mgpu_scene_create: triangle " + std::to_string(t) + " names a point light");
  // analytic spheres: records as the traversal reads them, shading records after the triangles'
  if (desc->nsphere < 0 || desc->nsphere > MGPU_MAX_SPHERES || (desc->nsphere > 0 && (!desc->spheres || !desc->sphere_mat)))
    return fail(MGPU_E_INVALID, "mgpu_scene_create: bad spheres (at most " + std::to_string(MGPU_MAX_SPHERES) + ")");
  std::vector<float4> sph((size_t)std::max(desc->nsphere, 0) * 2), sph_shade((size_t)std::max(desc->nsphere, 0) * 3);
  for (int i = 0; i < desc->nsphere; ++i) {
    const float *q = desc->spheres + 8 * (size_t)i;
    bool ok = q[3] > 0.0f;
    for (int k = 0; k < 8; ++k) ok = ok && std::isfinite(q[k]);
    if (!ok || desc->sphere_mat[i] < 0 || desc->sphere_mat[i] >= desc->nmat)
      return fail(MGPU_E_INVALID, "mgpu_scene_create: bad sphere " + std::to_string(i));
    sph[2 * i] = make_float4(q[0], q[1], q[2], q[3]);
    sph[2 * i + 1] = make_float4(q[4], q[5], q[6], q[7]);
    int32_t mat = desc->sphere_mat[i], li = desc->sphere_light ? desc->sphere_light[i] : -1;
    if (li < -1 || li >= desc->nlight)
      return fail(MGPU_E_INVALID, "mgpu_scene_create: light index out of range at sphere " + std::to_string(i));
    float4 a = make_float4(0, 0, 0, 0), b = a;
    memcpy(&a.w, &mat, 4);
    memcpy(&b.w, &li, 4);
    sph_shade[3 * i] = a;
    sph_shade[3 * i + 1] = b;
    sph_shade[3 * i + 2] = make_float4(0, 0, 0, 0);
  }
  const KdTree &tr = accel->tree;
  mgpu_accel *acc = const_cast<mgpu_accel *>(accel);
  register_staging(acc);
  const std::vector<Pair> &dpairs = accel->dpairs;
  const std::vector<F4> &ltris = accel->ltris, &tris = accel->tris;
  const std::vector<float4> &shade = accel->shade;
  SceneLayout L = scene_layout(accel, desc->nmat, desc->nlight, tp.uv ? T : 0, desc->ntex, tp.texels, desc->nsphere);

  mgpu_scene *s = new (std::nothrow) mgpu_scene();
  if (!s) return fail(MGPU_E_NOMEM, "mgpu_scene_create: out of host memory");
  cudaGetDevice(&s->device);
  bool wide = L.total <= limit;
  cudaError_t e = wide ? cudaMalloc(&s->d_block, L.total) : cudaErrorMemoryAllocation;
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();  // no room for the hierarchy: the kd-tree alone
    wide = false;
    L = scene_layout(accel, desc->nmat, desc->nlight, tp.uv ? T : 0, desc->ntex, tp.texels, desc->nsphere, false);
    e = cudaMalloc(&s->d_block, L.total);
  }
  if (e != cudaSuccess) {
    delete s;
    return cuda_fail(e, "mgpu_scene_create: cudaMalloc");
  }
  char *base = (char *)s->d_block;
  cudaStream_t st = as_stream(stream);
  auto up = [&](size_t off, const void *src, size_t n) -> cudaError_t {
    if (n == 0) return cudaSuccess;
    return cudaMemcpyAsync(base + off, src, n, cudaMemcpyHostToDevice, st);
  };
  s->view.tris = (const F4 *)(base + L.off_tris);
  s->view.ntri = T;
  s->view.wextent = 0.0f;
  for (int k = 0; k < 3; ++k) {
    s->view.bmin[k] = (float)tr.bmin[k];
    s->view.bmax[k] = (float)tr.bmax[k];
    const float c = 0.5f * s->view.bmin[k] + 0.5f * s->view.bmax[k];
    s->view.wcentre[k] = std::isfinite(c) ? c : 0.0f;
    // (a scene of points only has no bounds)
    const float lo = std::min(s->view.bmin[k], (float)tr.tmin[k]), hi = std::max(s->view.bmax[k], (float)tr.tmax[k]);
    s->view.wextent = std::max(s->view.wextent, std::max(hi - s->view.wcentre[k], s->view.wcentre[k] - lo));
  }
  e = up(L.off_tris, tris.data(), tris.size() * sizeof(F4));
  // the hierarchy's counters: beside the error words (256 bytes are 64)
  uint32_t *d_ctr = (uint32_t *)(base + L.off_err) + 16, ctr[kWideCounters];
  wide = wide && T > 0;
  if (e == cudaSuccess && wide) {
    if (int rc = wide_build(s->view.tris, T, s->view, base + L.off_wnodes, (F4 *)(base + L.off_wtris), base + L.off_pairs,
                            d_ctr, st)) {
      cudaFree(s->d_block);
      delete s;
      return rc;
    }
  }
  if (e == cudaSuccess) e = up(L.off_pairs, dpairs.data(), dpairs.size() * sizeof(Pair));
  if (e == cudaSuccess) e = up(L.off_refs, ltris.data(), ltris.size() * sizeof(F4));
  if (e == cudaSuccess) e = up(L.off_shade, shade.data(), shade.size() * sizeof(float4));
  if (e == cudaSuccess) e = up(L.off_mats, desc->materials, (size_t)desc->nmat * 16 * sizeof(float));
  if (e == cudaSuccess && desc->nlight > 0) e = up(L.off_lights, lrec.data(), lrec.size() * sizeof(float));
  if (e == cudaSuccess && tp.uv) e = up(L.off_uv, desc->tri_uv, (size_t)T * 6 * sizeof(float));
  if (e == cudaSuccess && desc->nsphere > 0) {
    e = up(L.off_sph, sph.data(), sph.size() * sizeof(float4));
    if (e == cudaSuccess)
      e = up(L.off_shade + shade.size() * sizeof(float4), sph_shade.data(), sph_shade.size() * sizeof(float4));
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(base + L.off_err, 0, 64, st);
  // the build of a small scene runs beside the uploads' staging: how it ended is read here (36 triangles: scene
  // creation 129 -> 115 us)
  if (e == cudaSuccess && wide) e = cudaMemcpyAsync(ctr, d_ctr, sizeof(ctr), cudaMemcpyDeviceToHost, st);
  // materials and lights are the caller's pageable arrays: wait for the copies
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaFree(s->d_block);
    delete s;
    return cuda_fail(e, "mgpu_scene_create: upload");
  }
  if (wide) wide_result(ctr, T, &s->wide_nodes, &wide, &s->outside);
  if (wide) {
    s->view.wnodes = (const uint32_t *)(base + L.off_wnodes);
    s->view.wtris = (const F4 *)(base + L.off_wtris);
  } else {
    s->view.wextent = INFINITY;
  }
  if (desc->ntex > 0) {
    if (int rc = tex_upload(desc, tp, (float4 *)(base + L.off_texrec), (float4 *)(base + L.off_texels), st)) {
      cudaFree(s->d_block);
      delete s;
      return rc;
    }
    s->d_texrec = (float4 *)(base + L.off_texrec);
    s->d_texels = (float4 *)(base + L.off_texels);
    s->tex_offset = tp.offset;
    for (int i = 0; i < desc->ntex; ++i) {
      s->tex_w.push_back(desc->textures[i].width);
      s->tex_h.push_back(desc->textures[i].height);
    }
  }
  if (tp.uv) s->d_uv = (float2 *)(base + L.off_uv);
  s->bg_tex = desc->background_tex;
  for (int k = 0; k < 3; ++k) s->bg_le[k] = desc->background_le[k];
  s->view.pairs = (const Pair *)(base + L.off_pairs);
  s->view.ltris = (const F4 *)(base + L.off_refs);
  s->view.npairs = tr.pairs.size();
  s->view.nrefs = ltris.size() / 3;
  s->view.spheres = desc->nsphere > 0 ? (const F4 *)(base + L.off_sph) : nullptr;
  s->view.nsphere = desc->nsphere;
  s->d_shade = (float4 *)(base + L.off_shade);
  s->d_mats = (float *)(base + L.off_mats);
  s->d_lights = (float *)(base + L.off_lights);
  s->nmat = desc->nmat;
  for (int i = 1; i < desc->nmat; ++i) s->mixed = s->mixed || desc->materials[16 * i] != desc->materials[0];
  s->nlight = desc->nlight;
  // staging the top of the tree in shared memory costs more occupancy than it saves on GB300
  // (the L1 keeps those pairs anyway); mgpu_scene_set_top_pairs turns it on
  s->top_pairs = 0;
  s->top_pairs_max = tr.top_pairs;
  s->d_err = (uint32_t *)(base + L.off_err);
  s->bytes = L.total;
  *out = s;
  return MGPU_OK;
}

int scene_device_bytes(const mgpu_scene_desc *desc, const mgpu_accel *a, bool wide, uint64_t *out) {
  TexPlan tp;
  if (int rc = tex_plan(desc, tp)) return rc;
  *out = scene_layout(a, desc->nmat, desc->nlight, tp.uv ? desc->ntri : 0, desc->ntex, tp.texels,
                      std::max(desc->nsphere, 0), wide).total;
  return MGPU_OK;
}

}  // namespace mgpu

extern "C" {

int mgpu_scene_destroy(mgpu_scene *s) {
  if (!s) return MGPU_OK;
  int cur = 0;
  cudaGetDevice(&cur);
  if (cur != s->device) cudaSetDevice(s->device);
  cudaError_t e = cudaFree(s->d_block);
  if (cur != s->device) cudaSetDevice(cur);
  delete s;
  if (e != cudaSuccess) return cuda_fail(e, "mgpu_scene_destroy: cudaFree");
  return MGPU_OK;
}

int mgpu_scene_set_top_pairs(mgpu_scene *s, uint32_t n) {
  if (!s) return fail(MGPU_E_INVALID, "mgpu_scene_set_top_pairs: null scene");
  if (n > s->top_pairs_max) n = s->top_pairs_max;
  if ((size_t)n * 16 > 96 * 1024) return fail(MGPU_E_INVALID, "mgpu_scene_set_top_pairs: more than 96 KiB of shared memory");
  s->top_pairs = n;
  return MGPU_OK;
}

int mgpu_scene_bytes(const mgpu_scene *s, uint64_t *out) {
  if (!s || !out) return fail(MGPU_E_INVALID, "mgpu_scene_bytes: null argument");
  *out = s->bytes;
  return MGPU_OK;
}

int mgpu_scene_hierarchy(const mgpu_scene *s, uint64_t *out) {
  if (!s || !out) return fail(MGPU_E_INVALID, "mgpu_scene_hierarchy: null argument");
  *out = s->wide_nodes;
  return MGPU_OK;
}

int mgpu_accel_device_bytes(const mgpu_accel *a, int32_t nmat, int32_t nlight, uint64_t *out) {
  if (!a || !out || nmat < 0 || nlight < 0) return fail(MGPU_E_INVALID, "mgpu_accel_device_bytes: bad argument");
  *out = scene_layout(a, nmat, nlight).total;
  return MGPU_OK;
}

int mgpu_scene_device_bytes(const mgpu_scene_desc *desc, const mgpu_accel *a, uint64_t *out) {
  if (!desc || !a || !out || desc->nmat < 0 || desc->nlight < 0)
    return fail(MGPU_E_INVALID, "mgpu_scene_device_bytes: bad argument");
  return scene_device_bytes(desc, a, true, out);
}

int mgpu_scene_read_texels(const mgpu_scene *s, int32_t tex, float *out, void *stream) {
  if (!s || !out || tex < 0 || tex >= (int32_t)s->tex_offset.size())
    return fail(MGPU_E_INVALID, "mgpu_scene_read_texels: bad argument");
  cudaStream_t st = as_stream(stream);
  const size_t n = (size_t)s->tex_w[tex] * s->tex_h[tex];
  MGPU_CUDA(cudaMemcpyAsync(out, s->d_texels + s->tex_offset[tex], n * sizeof(float4), cudaMemcpyDeviceToHost, st));
  MGPU_CUDA(cudaStreamSynchronize(st));
  return MGPU_OK;
}

int mgpu_film_create(int32_t width, int32_t height, void *stream, mgpu_film **out) {
  if (!out || width <= 0 || height <= 0 || (int64_t)width * height > (int64_t)1 << 31)
    return fail(MGPU_E_INVALID, "mgpu_film_create: bad size");
  mgpu_film *f = new (std::nothrow) mgpu_film();
  if (!f) return fail(MGPU_E_NOMEM, "mgpu_film_create: out of host memory");
  cudaGetDevice(&f->device);
  f->width = width;
  f->height = height;
  size_t n = (size_t)width * height;
  void *p = nullptr;
  cudaError_t e = cudaMalloc(&p, 2 * n * sizeof(float4));
  if (e != cudaSuccess) {
    delete f;
    return cuda_fail(e, "mgpu_film_create: cudaMalloc");
  }
  f->d_sum = (float4 *)p;
  f->d_c = f->d_sum + n;
  e = cudaMemsetAsync(p, 0, 2 * n * sizeof(float4), as_stream(stream));
  if (e != cudaSuccess) {
    cudaFree(p);
    delete f;
    return cuda_fail(e, "mgpu_film_create: clear");
  }
  *out = f;
  return MGPU_OK;
}

int mgpu_film_clear(mgpu_film *f, void *stream) {
  if (!f) return fail(MGPU_E_INVALID, "mgpu_film_clear: null film");
  MGPU_CUDA(cudaMemsetAsync(f->d_sum, 0, 2 * (size_t)f->width * f->height * sizeof(float4), as_stream(stream)));
  if (f->d_fx)
    MGPU_CUDA(cudaMemsetAsync(f->d_fx, 0, 4 * (size_t)f->width * f->height * sizeof(unsigned long long),
                              as_stream(stream)));
  return MGPU_OK;
}

int mgpu_film_set_filter(mgpu_film *f, int32_t type, float support, float p1, float p2, void *stream) {
  if (!f) return fail(MGPU_E_INVALID, "mgpu_film_set_filter: null film");
  if (type < kFilterNone || type > kFilterLanczos || (type != kFilterNone && !(support > 0.0f && support <= 64.0f)) ||
      (type == kFilterGaussian && !(p1 > 0.0f)) || (type == kFilterLanczos && !(p1 > 0.0f)))
    return fail(MGPU_E_INVALID, "mgpu_film_set_filter: bad filter type or parameters");
  if (f->d_fx) {
    cudaFree(f->d_fx);
    f->d_fx = nullptr;
  }
  f->filter = FilmFilter{type, type == kFilterNone ? 0 : (int)(((unsigned)ceilf(support) | 1u) >> 1), support, p1, p2};
  if (type == kFilterNone) return MGPU_OK;
  const size_t bytes = 4 * (size_t)f->width * f->height * sizeof(unsigned long long);
  MGPU_CUDA(cudaMalloc(&f->d_fx, bytes));
  MGPU_CUDA(cudaMemsetAsync(f->d_fx, 0, bytes, as_stream(stream)));
  return MGPU_OK;
}

int mgpu_film_destroy(mgpu_film *f) {
  if (!f) return MGPU_OK;
  cudaError_t e = cudaFree(f->d_sum);
  if (f->d_fx) cudaFree(f->d_fx);
  delete f;
  if (e != cudaSuccess) return cuda_fail(e, "mgpu_film_destroy: cudaFree");
  return MGPU_OK;
}

int mgpu_film_read_raw(mgpu_film *f, float *out8, void *stream) {
  if (!f || !out8) return fail(MGPU_E_INVALID, "mgpu_film_read_raw: null argument");
  size_t n = (size_t)f->width * f->height;
  cudaStream_t st = as_stream(stream);
  make_pages(out8, 2 * n * sizeof(float4));
  MGPU_CUDA(cudaMemcpyAsync(out8, f->d_sum, 2 * n * sizeof(float4), cudaMemcpyDeviceToHost, st));
  MGPU_CUDA(cudaStreamSynchronize(st));
  return MGPU_OK;
}

// The film's output in FP64 for pixels first .. first + count - 1, written by the kernel where the host reads
// it (page-locked memory): the per-pixel mean (sum - compensation) / count (ProgressiveFilterValue::
// getValue, ProgressiveFilterValue.h:26-31; 0 for a pixel without samples), or with a reconstruction
// filter sum(w L) / sum(w).  256 pixels at a time go through shared memory so that the stores to
// the host are whole lines.
__global__ void __launch_bounds__(256) k_film_mean(const float4 *__restrict__ sum, const float4 *__restrict__ comp,
                                                   const unsigned long long *__restrict__ fx, int64_t first,
                                                   int64_t count, double *__restrict__ out) {
  __shared__ double rgb[768];
  for (int64_t base = (int64_t)blockIdx.x * 256; base < count; base += (int64_t)gridDim.x * 256) {
    const int64_t i = base + threadIdx.x;
    if (i < count) {
      double r = 0.0, g = 0.0, b = 0.0;
      if (fx) {
        const unsigned long long *q = fx + 4 * (first + i);
        const double w = (double)q[3];
        if (w > 0) {
          r = (double)q[0] / w;
          g = (double)q[1] / w;
          b = (double)q[2] / w;
        }
      } else {
        const float4 s = sum[first + i], c = comp[first + i];
        const double cnt = s.w;
        if (cnt > 0) {
          r = ((double)s.x - (double)c.x) / cnt;
          g = ((double)s.y - (double)c.y) / cnt;
          b = ((double)s.z - (double)c.z) / cnt;
        }
      }
      rgb[3 * threadIdx.x] = r;
      rgb[3 * threadIdx.x + 1] = g;
      rgb[3 * threadIdx.x + 2] = b;
    }
    __syncthreads();
    const int64_t n = 3 * (count - base < 256 ? count - base : 256);
    for (int k = (int)threadIdx.x; k < n; k += 256) out[3 * base + k] = rgb[k];
    __syncthreads();
  }
}

int mgpu_film_read(mgpu_film *f, double *out_mean, void *stream) {
  if (!f || !out_mean) return fail(MGPU_E_INVALID, "mgpu_film_read: null argument");
  const int64_t n = (int64_t)f->width * f->height;
  cudaStream_t st = as_stream(stream);
  int cur = 0;
  MGPU_CUDA(cudaGetDevice(&cur));
  if (cur != f->device) {  // the kernel runs where the film is, after what the caller's stream holds
    MGPU_CUDA(cudaStreamSynchronize(st));
    MGPU_CUDA(cudaSetDevice(f->device));
    const int rc = mgpu_film_read(f, out_mean, nullptr);
    cudaSetDevice(cur);
    return rc;
  }
  auto launch = [&](int64_t first, int64_t count, double *dst) {
    const unsigned grid = (unsigned)std::min<int64_t>((count + 255) / 256, (int64_t)device_sm_count() * 8);
    k_film_mean<<<grid, 256, 0, st>>>(f->d_sum, f->d_c, f->d_fx, first, count, dst);
    g_launches.fetch_add(1);
    return cudaGetLastError();
  };
  // into the caller's array where the device can write it
  if (device_writes(out_mean, (size_t)n * 3 * sizeof(double), alignof(double))) {
    MGPU_CUDA(launch(0, n, out_mean));
    MGPU_CUDA(cudaStreamSynchronize(st));
    return MGPU_OK;
  }
  const size_t bytes = (size_t)n * 3 * sizeof(double);
  double *d = nullptr;
  if (bytes <= kStageBytes) {
    MGPU_CUDA(t_read.host_buffer(bytes, (void **)&d));
    MGPU_CUDA(launch(0, n, d));
    MGPU_CUDA(cudaStreamSynchronize(st));
    memcpy(out_mean, d, bytes);
    return MGPU_OK;
  }
  // taken in a device buffer that the thread keeps, at most kPiece pixels at a time
  constexpr int64_t kPiece = (int64_t)1 << 22;
  MGPU_CUDA(t_read.device_buffer((size_t)std::min(n, kPiece) * 3 * sizeof(double), (void **)&d));
  for (int64_t first = 0; first < n; first += kPiece) {
    const int64_t cnt = std::min(kPiece, n - first);
    MGPU_CUDA(launch(first, cnt, d));
    MGPU_CUDA(to_host(out_mean + 3 * first, d, (size_t)cnt * 3 * sizeof(double), st));
  }
  return MGPU_OK;
}

int mgpu_film_tonemap(mgpu_film *f, uint8_t *out_rgba, void *stream) {
  if (!f || !out_rgba) return fail(MGPU_E_INVALID, "mgpu_film_tonemap: null argument");
  const int64_t npix = (int64_t)f->width * f->height;
  ToneSrc ref{FilmRef{f->d_sum, f->d_c, npix, 0}, f->d_fx};
  const size_t bytes = (size_t)npix * sizeof(uchar4), b_part = align_up(kErrBlocks * sizeof(double2), 256);
  const bool direct = device_writes(out_rgba, bytes, sizeof(uchar4)), staged = !direct && bytes <= kStageBytes;
  char *d = nullptr;
  MGPU_CUDA(t_read.device_buffer(b_part + (direct || staged ? 0 : bytes), (void **)&d));
  double2 *part = (double2 *)d;
  uchar4 *img = direct ? (uchar4 *)out_rgba : (uchar4 *)(d + b_part);
  if (staged) MGPU_CUDA(t_read.host_buffer(bytes, (void **)&img));
  cudaStream_t st = as_stream(stream);
  k_tonemap_reduce<<<kErrBlocks, kErrThreads, 0, st>>>(ref, part);
  k_tonemap_map<<<device_sm_count() * 4, 256, 0, st>>>(ref, part, img);
  g_launches.fetch_add(2);
  MGPU_CUDA(cudaGetLastError());
  if (direct || staged) MGPU_CUDA(cudaStreamSynchronize(st));
  else MGPU_CUDA(to_host(out_rgba, img, bytes, st));
  if (staged) memcpy(out_rgba, img, bytes);
  return MGPU_OK;
}

int mgpu_film_error(mgpu_film *const *films, int32_t n, double *out_rmse, void *stream) {
  if (n < 0 || n > 65535 || (n > 0 && (!films || !out_rmse)))
    return fail(MGPU_E_INVALID, "mgpu_film_error: bad argument");
  if (n == 0) return MGPU_OK;
  // the films' records and their estimates in page-locked memory that the kernels read and write
  const size_t b_refs = align_up((size_t)n * sizeof(FilmRef), 256);
  char *h = nullptr;
  MGPU_CUDA(t_read.host_buffer(b_refs + (size_t)n * sizeof(double), (void **)&h));
  FilmRef *refs = (FilmRef *)h;
  double *est = (double *)(h + b_refs);
  int64_t blocks = 0;
  for (int32_t i = 0; i < n; ++i) {
    if (!films[i]) return fail(MGPU_E_INVALID, "mgpu_film_error: null film");
    const int64_t npix = (int64_t)films[i]->width * films[i]->height;
    refs[i] = FilmRef{films[i]->d_sum, films[i]->d_c, npix, blocks};
    blocks += err_blocks(npix);
  }
  double2 *part = nullptr;
  MGPU_CUDA(t_read.device_buffer((size_t)blocks * sizeof(double2), (void **)&part));
  cudaStream_t st = as_stream(stream);
  k_film_error_partial<<<(unsigned)blocks, kErrThreads, 0, st>>>(refs, n, part);
  k_film_error_final<<<n, kErrThreads, 0, st>>>(refs, part, est);
  g_launches.fetch_add(2);
  MGPU_CUDA(cudaGetLastError());
  MGPU_CUDA(cudaStreamSynchronize(st));
  memcpy(out_rmse, est, (size_t)n * sizeof(double));
  return MGPU_OK;
}

// Page-locked host memory that every device can write (results are then read without a staging copy).
int mgpu_host_alloc(uint64_t bytes, void **out) {
  if (!out || bytes == 0) return fail(MGPU_E_INVALID, "mgpu_host_alloc: bad argument");
  MGPU_CUDA(cudaHostAlloc(out, (size_t)bytes, cudaHostAllocPortable | cudaHostAllocMapped));
  try {
    std::lock_guard<std::mutex> lock(g_host_mu);
    g_host_blocks[(uintptr_t)*out] = (size_t)bytes;
  } catch (const std::bad_alloc &) {
    cudaFreeHost(*out);
    *out = nullptr;
    return fail(MGPU_E_NOMEM, "mgpu_host_alloc: out of host memory");
  }
  return MGPU_OK;
}

int mgpu_host_free(void *p) {
  {
    std::lock_guard<std::mutex> lock(g_host_mu);
    g_host_blocks.erase((uintptr_t)p);
  }
  if (p) MGPU_CUDA(cudaFreeHost(p));
  return MGPU_OK;
}

}  // extern "C"
