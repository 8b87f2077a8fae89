// kernels_pt.cu - raw ray batches and the wavefront path tracer.
//
// The reference's PathTracingIntegrator.rayColorRecursive
// (pkg/integrator/path_tracing.go:35-104) recurses once per bounce and
// returns emitted + direct + indirect radiance, every level scaled by its
// Russian-roulette compensation, and the indirect term scaled by the BSDF
// MIS weight.  Unrolled, the radiance of a sample is a sum over bounces of
//     W_k * (Le_k + Ld_k)
// where W_k is the product of the per-level factors of the levels above:
// rr compensation, and attenuation (specular) or attenuation*cos*w_bsdf/pdf
// (diffuse).  The wavefront keeps W_k, the Russian-roulette throughput and
// the gathered radiance per path and advances all paths one bounce per
// kernel sequence:  extend (closest hit) -> shade -> shadow (any hit).
#include <algorithm>

#include "device.cuh"
#include "kernels.h"
#include "pt_shade.cuh"

namespace gprt {

int launch_grid(uint32_t n, int block, int max_blocks) {
  uint32_t g = n / (uint32_t)block + (n % (uint32_t)block != 0);
  if (g < 1) g = 1;
  if (max_blocks > 0 && g > (uint32_t)max_blocks) g = (uint32_t)max_blocks;
  return (int)g;
}

// ----------------------------------------------------------------- raw batches
struct BatchSource {
  const gprt_ray* rays;
  gprt_hit* hits;
  uint32_t n;
  __device__ uint32_t count() const { return n; }
  int root;
  int* err;  // null: the hit records alone tell
  __device__ void load(uint32_t i, float3& o, float3& d, float& tmin, float& tmax, uint32_t& skip, int& rt) const {
    rt = root;
    const float4* r = reinterpret_cast<const float4*>(rays + i);
    float4 a = __ldg(r), b = __ldg(r + 1);
    o = f3(a);
    d = f3(b);
    tmin = a.w;
    tmax = b.w;
    skip = kNoHit;
  }
  __device__ void store(uint32_t i, const Hit& h) const {
    bool over = h.prim == kOverflowHit;
    if (over && err) atomicOr(err, kErrStackOverflow);
    bool any = h.prim != kNoHit && !over;
    reinterpret_cast<float4*>(hits)[i] =
        make_float4(any ? h.t : -1.f, __uint_as_float(any || over ? h.prim : kNoHit), any ? h.u : 0.f,
                    any ? h.v : 0.f);
  }
};

// Batches deal their rays out without a counter: calls on different streams share none.
template <bool kAny, bool kOneNode>
__global__ void __launch_bounds__(128, kTravBlocks) k_intersect(DevScene sc, BatchSource src, const __grid_constant__ Geom<kOneNode> g) {
  if constexpr (kOneNode) trace_batch_one_node<kAny, false>(g, src, nullptr, nullptr);
  else trace_persistent<kAny, false>(sc, src, nullptr, nullptr, nullptr);
}

int persistent_grid(int sm_count, int block) { return std::max(1, sm_count * kTravBlocks * 128 / block); }

void launch_intersect(const DevScene& sc, const gprt_ray* rays, uint32_t n, bool any_hit, gprt_hit* hits, int* err,
                      cudaStream_t st) {
  if (n == 0) return;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int grid = launch_grid(n, 128, persistent_grid(sms, 128));
  BatchSource src{rays, hits, n, sc.root, err};
  if (one_node(sc)) (any_hit ? k_intersect<true, true> : k_intersect<false, true>)<<<grid, 128, 0, st>>>(sc, src, *sc.one);
  else (any_hit ? k_intersect<true, false> : k_intersect<false, false>)<<<grid, 128, 0, st>>>(sc, src, NoGeom{});
}

// ----------------------------------------------------------------- raygen
// TileRenderer sample loop + Camera.GetRay (tile_renderer.go:55-59,
// camera.go:173-190): path p of the chunk is sample `layer` of pixel i.
__global__ void k_pt_raygen(DevScene sc, DevFilm film, DevPaths P, ChunkDesc ch) {
  uint32_t n = ch.npix * ch.layers;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    uint32_t layer = p / ch.npix, i = p - layer * ch.npix;
    uint32_t pix = ch.pix_list ? ch.pix_list[ch.pix0 + i] : ch.pix0 + i;
    uint32_t sample = film.count[pix] + layer;
    int x = (int)(pix % (uint32_t)film.width), y = (int)(pix / (uint32_t)film.width);
    Rng rng;
    rng.init(ch.seed, pix, sample);
    // Camera.GetRay(i, j, sampler.Get2D(), sampler.Get2D()) (tile_renderer.go:56)
    float2 lens = rng.next2();
    float2 jit = rng.next2();
    float3 o, d;
    camera_ray(sc.cam, x, y, lens, jit, o, d, true);
    const PathBuf& Q = P.q[0];
    store32(Q.ray + 2 * (size_t)p, make_float4(o.x, o.y, o.z, __uint_as_float(kNoHit)),
            make_float4(d.x, d.y, d.z, __int_as_float(sc.root)));
    store32(Q.st + 2 * (size_t)p, make_float4(1.f, 1.f, 1.f, __uint_as_float(p)),
            as_float4(make_uint4(pix, sample, rng.pos, 0u)));  // throughput 1 is implied at bounce 0
    P.Lout[p] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    P.counters[0] = n;
    P.counters[4] = 0;  // ray-fetch counters of the first extend and shadow launches
    P.counters[5] = 0;
  }
}

void launch_pt_raygen(const DevScene& sc, const DevFilm& film, const DevPaths& P, const ChunkDesc& ch, int block,
                      cudaStream_t st) {
  uint32_t n = ch.npix * ch.layers;
  k_pt_raygen<<<launch_grid(n, block, 0), block, 0, st>>>(sc, film, P, ch);
}

// ----------------------------------------------------------------- extend
// scene.BVH.Hit(ray, 0.001, +Inf) for every live path (path_tracing.go:67)

// Adds one thread's traversal work to the job's counters (one atomic per warp).
__device__ __forceinline__ void add_counts(unsigned long long* dst, uint32_t rays, const TraceStats& s) {
  unsigned long long v[4] = {rays, s.nodes, s.boxes, s.prims};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    unsigned long long x = v[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0 && x) atomicAdd(dst + k, x);
  }
}

// The rays of the current queue; built on the host and passed as a kernel
// argument, so its pointers stay in the constant bank.
struct ExtendSource {
  const float4* ray;
  float4* hit;
  const uint32_t* n;
  const float4* st;  // origin index of each path (first .w), read when reporting a bound
  ErrSink err;
  __device__ uint32_t count() const { return *n; }
  __device__ void load(uint32_t i, float3& o, float3& d, float& tmin, float& tmax, uint32_t& skip, int& rt) const {
    float4 a, b;
    load32(ray + 2 * (size_t)i, a, b);
    rt = __float_as_int(b.w);
    o = f3(a);
    d = f3(b);
    tmin = 0.001f;
    tmax = kInfF;
    skip = __float_as_uint(a.w);
  }
  // the marker hit of a stack overflow is stored as a miss and fails the
  // path's job
  __device__ void store(uint32_t i, const Hit& h) const {
    bool any = h.prim != kNoHit;
    if (h.prim == kOverflowHit) {
      err.report(__float_as_uint(st[2 * (size_t)i].w), kErrStackOverflow);
      any = false;
    }
    hit[i] = make_float4(any ? h.t : -1.f, __uint_as_float(any ? h.prim : kNoHit), h.u, h.v);
  }
};

// The error sink of a wavefront's paths (per job, or per item of a multi-job step).
static ErrSink err_sink(const DevPaths& P) { return ErrSink{P.counters + 3, P.item_err, P.item_start, P.n_items}; }

template <bool kCount, bool kOneNode>
__global__ void __launch_bounds__(128, kTravBlocks)
    k_pt_extend(DevScene sc, ExtendSource src, uint32_t* counters, int cur, unsigned long long* stats,
                const __grid_constant__ Geom<kOneNode> g) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counters[cur ^ 1] = 0;  // next queue and shadow queue start empty
    counters[2] = 0;
    counters[6] = 0;  // hit / miss counts of the slot order built after this launch
    counters[7] = 0;
  }
  TraceStats ts{0, 0, 0};
  uint32_t rays = 0;
  if constexpr (kOneNode) trace_batch_one_node<false, kCount>(g, src, &ts, &rays);
  else trace_persistent<false, kCount>(sc, src, counters + 4, &ts, &rays);
  if (kCount) {
    __syncwarp();
    add_counts(stats, rays, ts);
  }
}

// One ray per thread (grid-stride), the variant GPRT_JOB_SIMPLE_EXTEND selects.
template <bool kCount>
__global__ void __launch_bounds__(256)
    k_pt_extend_simple(DevScene sc, ExtendSource src, uint32_t* counters, int cur, unsigned long long* stats) {
  uint32_t n = src.count();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counters[cur ^ 1] = 0;
    counters[2] = 0;
    counters[6] = 0;
    counters[7] = 0;
  }
  TraceStats ts{0, 0, 0};
  uint32_t rays = 0;
  uint32_t end = kCount ? ((n + 31) & ~31u) : n;  // whole warps stay for the count reduction
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < end; i += gridDim.x * blockDim.x) {
    if (i < n) {
      float3 o, d;
      float tmin, tmax;
      uint32_t skip;
      int root;
      src.load(i, o, d, tmin, tmax, skip, root);
      Hit h;
      trace_from<false, kCount>(sc, root, o, d, tmin, tmax, skip, h, nullptr, &ts);
      src.store(i, h);
      rays++;
    }
  }
  if (kCount) add_counts(stats, rays, ts);
}

static int sm_count_current() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

void launch_pt_extend(const DevScene& sc, const DevPaths& P, int cur, int bounce, int block, int grid, cudaStream_t st) {
  ExtendSource src{P.q[cur].ray, P.hit, P.counters + cur, P.q[cur].st, err_sink(P)};
  if (P.variant & GPRT_JOB_SIMPLE_EXTEND) {
    int b = std::min(block, 256);
    if (P.stats) k_pt_extend_simple<true><<<grid, b, 0, st>>>(sc, src, P.counters, cur, P.stats);
    else k_pt_extend_simple<false><<<grid, b, 0, st>>>(sc, src, P.counters, cur, P.stats);
    return;
  }
  const int g = persistent_grid(sm_count_current(), 128);
  if (one_node(sc))
    (P.stats ? k_pt_extend<true, true> : k_pt_extend<false, true>)<<<g, 128, 0, st>>>(sc, src, P.counters, cur, P.stats,
                                                                                      *sc.one);
  else
    (P.stats ? k_pt_extend<true, false> : k_pt_extend<false, false>)<<<g, 128, 0, st>>>(sc, src, P.counters, cur,
                                                                                        P.stats, NoGeom{});
}

// ----------------------------------------------------------------- shade
// The shading order of queue `cur` (order_slots) for one scene.
__global__ void __launch_bounds__(1024) k_hit_order(DevScene sc, DevPaths P, int cur) {
  order_slots(P, cur, [&](uint32_t, uint32_t prim) { return prim_group(sc, prim); });
}

void launch_hit_order(const DevScene& sc, const DevPaths& P, int cur, uint32_t cap, int sms, cudaStream_t st) {
  if (!P.order) return;
  int g = std::max(1, std::min((int)((cap + 1023) / 1024), sms * 2));
  k_hit_order<<<g, 1024, 0, st>>>(sc, P, cur);
}

// One level of rayColorRecursive (path_tracing.go:35-104) with
// CalculateDirectLighting (:116-157), CalculateIndirectLighting (:160-189)
// and ApplyRussianRoulette (:193-220).  The Russian-roulette draw happens
// first at every level, as in the reference.
template <int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    k_pt_shade(DevScene sc, DevPaths P, ChunkDesc ch, int cur, int bounce) {
  uint32_t n = P.counters[cur];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    P.counters[4] = 0;  // ray-fetch counters of the next shadow and extend launches
    P.counters[5] = 0;
  }
  const uint32_t stride = gridDim.x * blockDim.x;
  uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t slot = first < n ? (P.order ? P.order[first] : first) : 0u;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    uint32_t i = base + threadIdx.x;
    // the slot of the next iteration, read now and prefetched into L2 after this one
    uint32_t inext = i + stride;
    uint32_t snext = inext < n ? (P.order ? P.order[inext] : inext) : 0u;
    ShadeOut o;
    o.cont = false;
    bool live = i < n;
    if (live) {
      float4 w4, ids;
      load32(P.q[cur].st + 2 * (size_t)slot, w4, ids);
      shade_path(sc, P, cur, slot, w4, as_uint4(ids), ch.seed, bounce, o);
    }
    push_shade_out(P, cur, live, o);
    if (inext < n) prefetch_slot(P.q[cur], P.hit, snext);
    slot = snext;
  }
}

void launch_pt_shade(const DevScene& sc, const DevPaths& P, const ChunkDesc& ch, int cur, int bounce, int block,
                     int grid, cudaStream_t st) {
  // the shading-group slot order pays where rays escape to an infinite
  // light (missed rays are then a large share) or where specular and
  // diffuse materials mix; in closed all-diffuse scenes it is overhead
  DevPaths Po = P;
  if (sc.has_infinite || sc.has_specular) launch_hit_order(sc, P, cur, P.capacity, sm_count_current(), st);
  else Po.order = nullptr;
  if (P.variant & GPRT_JOB_SHADE_OCCUPANCY) {
    int g = std::max(1, (int)((int64_t)grid * block / 192));
    k_pt_shade<192, 3><<<g, 192, 0, st>>>(sc, Po, ch, cur, bounce);
  } else {
    k_pt_shade<256, 2><<<grid, std::min(block, 256), 0, st>>>(sc, Po, ch, cur, bounce);
  }
}

// ----------------------------------------------------------------- shadow
// scene.BVH.Hit(shadowRay, 0.001, distance - 0.001) used as a boolean
// (path_tracing.go:143-148): the contribution is kept when nothing is hit.
struct ShadowSource {
  const float4* sh_o;
  const float4* sh_d;
  const float4* sh_c;
  const int* sh_root;  // null: every ray starts at `root`
  float4* Lout;        // radiance of the paths, by origin index
  const uint32_t* n;
  int root;
  ErrSink err;
  __device__ uint32_t count() const { return *n; }
  __device__ void load(uint32_t i, float3& o, float3& d, float& tmin, float& tmax, uint32_t& skip, int& rt) const {
    rt = sh_root ? sh_root[i] : root;
    float4 a = sh_o[i], b = sh_d[i];
    o = f3(a);
    d = f3(b);
    tmin = 0.001f;
    tmax = a.w;
    skip = __float_as_uint(b.w);
  }
  // one shadow ray per path and bounce: the read-modify-write of its origin
  // slot meets no other ray of the launch
  __device__ void store(uint32_t i, const Hit& h) const {
    if (h.prim == kOverflowHit) {  // the visibility is unknown: fail the path's job
      err.report(__float_as_uint(sh_c[i].w), kErrStackOverflow);
      return;
    }
    if (h.prim != kNoHit) return;  // occluded
    float4 c = sh_c[i];
    float4* dst = Lout + __float_as_uint(c.w);
    float4 L = *dst;
    *dst = make_float4(L.x + c.x, L.y + c.y, L.z + c.z, 0.f);
  }
};

template <bool kCount, bool kOneNode>
__global__ void __launch_bounds__(128, kTravBlocks)
    k_pt_shadow(DevScene sc, ShadowSource src, uint32_t* counters, unsigned long long* stats,
                const __grid_constant__ Geom<kOneNode> g) {
  TraceStats ts{0, 0, 0};
  uint32_t rays = 0;
  if constexpr (kOneNode) trace_batch_one_node<true, kCount>(g, src, &ts, &rays);
  else trace_persistent<true, kCount>(sc, src, counters + 5, &ts, &rays);
  if (kCount) {
    __syncwarp();
    add_counts(stats + 4, rays, ts);
  }
}

// One shadow ray per thread (grid-stride), the variant GPRT_JOB_SIMPLE_SHADOW selects.
template <bool kCount>
__global__ void __launch_bounds__(256)
    k_pt_shadow_simple(DevScene sc, ShadowSource src, uint32_t* counters, unsigned long long* stats) {
  uint32_t n = src.count();
  TraceStats ts{0, 0, 0};
  uint32_t rays = 0;
  uint32_t end = kCount ? ((n + 31) & ~31u) : n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < end; i += gridDim.x * blockDim.x) {
    if (i < n) {
      float3 o, d;
      float tmin, tmax;
      uint32_t skip;
      int root;
      src.load(i, o, d, tmin, tmax, skip, root);
      Hit h;
      trace_from<true, kCount>(sc, root, o, d, tmin, tmax, skip, h, nullptr, &ts);
      src.store(i, h);
      rays++;
    }
  }
  if (kCount) add_counts(stats + 4, rays, ts);
}

void launch_pt_shadow(const DevScene& sc, const DevPaths& P, int cur, int block, int grid, cudaStream_t st) {
  ShadowSource src{P.sh_o, P.sh_d, P.sh_c, P.sh_root, P.Lout, P.counters + 2, sc.root, err_sink(P)};
  if (P.variant & GPRT_JOB_SIMPLE_SHADOW) {
    int b = std::min(block, 256);
    if (P.stats) k_pt_shadow_simple<true><<<grid, b, 0, st>>>(sc, src, P.counters, P.stats);
    else k_pt_shadow_simple<false><<<grid, b, 0, st>>>(sc, src, P.counters, P.stats);
    return;
  }
  const int g = persistent_grid(sm_count_current(), 128);
  if (one_node(sc))
    (P.stats ? k_pt_shadow<true, true> : k_pt_shadow<false, true>)<<<g, 128, 0, st>>>(sc, src, P.counters, P.stats,
                                                                                      *sc.one);
  else
    (P.stats ? k_pt_shadow<true, false> : k_pt_shadow<false, false>)<<<g, 128, 0, st>>>(sc, src, P.counters, P.stats,
                                                                                        NoGeom{});
}

// ----------------------------------------------------------------- whole paths
// Small wavefronts in one launch: a lane takes a path from its camera ray to
// its end (trace the shadow ray of the last level and the path's ray, shade,
// repeat), keeping the state in registers that the queues of the wavefront
// pass through memory.  The wavefront's 3-4 launches cost 30-45 us a bounce on
// any number of paths (launches, and one ray's chain of dependent loads on an
// almost empty chip), and a scene of depth 50 pays that 50 times; here the
// chain of a path's bounces is all that is left: default scene, 90,000 paths of
// depth 50, 16 rounds 24.2 -> 7.18 ms, sphere scene 128 x 128 373 -> 125 us.
// What bounds that chain is fetching instructions: a bounce runs 2,600 of
// them, more than the caches near the scheduler hold, and warps at different
// places of the code evict each other's.  So the warps of a block trace together
// and shade together (two barriers a bounce) and share what they fetch: the
// default scene as above in blocks of 128 8.81 ms, 256 7.72, 512 7.18 (of 64
// without the barriers 9.96, before the pairing below).  Trees, whose traversals
// differ more in length, keep to 256 (128, 256 and 512: sphere scene 128 x 128
// 132, 125 and 125 us; 20,480 triangles 256 x 256 357, 367 and 389).
// It loses on large wavefronts, where lanes of a warp part ways and 16 warps
// per SM hide less than the traversal kernels' 32.
// Results are those of the wavefront, bit for bit: the same tests in the same
// order, the shading with the same roundings (dot_xy), and the radiance added
// up as the kernels of the wavefront add it (each unoccluded shadow ray, and
// what the path itself gathered when it ends).
// 512 threads per SM at 128 registers; a finished lane takes the warp's next
// path at once (waiting for 8 or 16 idle lanes: 2 and 14 % slower at 160,000
// paths).
constexpr int kPathsThreads = 512;  // per SM
constexpr int paths_block(bool one_node) { return one_node ? 512 : 256; }

// Paths of a wavefront at most that k_pt_paths renders: where both forms took
// the same time on GB300 (1 sample per pixel, depth 8; wavefront / whole paths
// in us).  Scenes with an infinite light, whose paths leave at different
// depths: sphere scene 526 / 404 at 360,000 paths, 639 / 572 at 589,824, 740 /
// 749 at 810,000; 20,480 triangles 1651 / 1516 at 589,824 and 1862 / 1924 at
// 810,000, 1.3 M triangles 2822 / 2396 and 3137 / 2991; quadrics 409 / 405 at
// 409,600 and 462 / 466 at 589,824; textured shapes 396 / 256 at 360,000, 533 /
// 471 at 810,000.  Closed scenes, where all lanes stay busy: Cornell box 334 /
// 317 at 176,400, 347 / 347 at 211,600, 455 / 509 at 360,000 (with spheres
// 423 / 391 there).
uint32_t pt_paths_max(const DevScene& sc, int sms) {
  return (uint32_t)sms * (sc.has_infinite ? 4096u : one_node(sc) ? 1536u : 2048u);
}

__device__ __forceinline__ float4 shfl4(float4 v, int src) {
  return make_float4(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                     __shfl_sync(0xffffffffu, v.z, src), __shfl_sync(0xffffffffu, v.w, src));
}

// kPair: a lane that has both a shadow ray and the path's ray hands the shadow
// ray to a lane of the warp that has neither, where there is one, and gets its
// answer back, so that both are on their way at once; without, and for the
// lanes that find none, one after the other.  (Sphere scene 128 x 128: 143 ->
// 125 us a pass; 20,480 triangles, 65,536 paths 399 -> 367.)
template <bool kOneNode, bool kPair>
__global__ void __launch_bounds__(paths_block(kOneNode), kPathsThreads / paths_block(kOneNode))
    k_pt_paths(DevScene sc, DevFilm film, DevPaths P, ChunkDesc ch, const __grid_constant__ Geom<kOneNode> g) {
  const uint32_t n = ch.npix * ch.layers;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  __shared__ uint8_t lane_of[paths_block(kOneNode) / 32][2][32];  // of the pairs: asking lane, answering lane
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t chunk = min(32u, (n + nw - 1) / nw);
  const ErrSink err{P.counters + 3, nullptr, nullptr, nullptr};
  uint64_t at = (uint64_t)w * chunk;
  uint32_t cur = (uint32_t)min((uint64_t)n, at), end = (uint32_t)min((uint64_t)n, at + chunk);
  bool more = cur < end;
  bool alive = false, shadow = false;  // the lane's path goes on; its last level left a shadow ray
  uint32_t path = 0;
  int bounce = 0;
  uint4 ids = make_uint4(0, 0, 0, 0);
  float4 o4 = make_float4(0.f, 0.f, 0.f, 0.f), d4 = o4, w4 = o4, sh_o = o4, sh_d = o4;
  float3 thr = f3(0.f, 0.f, 0.f), sh_c = thr;
  float3 Lo = thr;  // what the wavefront holds at the path's origin index
  TravEntry stack[kTraceStack];
  for (;;) {
    // new paths for the idle lanes
    unsigned idle = __ballot_sync(0xffffffffu, !alive && !shadow);
    if (more && idle) {
      if (cur == end) {
        at += (uint64_t)nw * chunk;
        cur = (uint32_t)min((uint64_t)n, at);
        end = (uint32_t)min((uint64_t)n, at + chunk);
      }
      if (cur == end) more = false;
      uint32_t take = min((uint32_t)__popc(idle), end - cur);
      uint32_t rank = (uint32_t)__popc(idle & ((1u << lane) - 1u));
      if (!alive && !shadow && rank < take) {
        path = cur + rank;
        uint32_t layer = path / ch.npix, i = path - layer * ch.npix;
        uint32_t pix = ch.pix_list ? ch.pix_list[ch.pix0 + i] : ch.pix0 + i;
        uint32_t sample = film.count[pix] + layer;
        int x = (int)(pix % (uint32_t)film.width), y = (int)(pix / (uint32_t)film.width);
        Rng rng;
        rng.init(ch.seed, pix, sample);
        float2 lens = rng.next2();
        float2 jit = rng.next2();
        float3 o, d;
        camera_ray(sc.cam, x, y, lens, jit, o, d, true);
        o4 = make_float4(o.x, o.y, o.z, __uint_as_float(kNoHit));
        d4 = make_float4(d.x, d.y, d.z, __int_as_float(sc.root));
        ids = make_uint4(pix, sample, rng.pos, 0u);
        w4 = make_float4(1.f, 1.f, 1.f, __uint_as_float(path));
        thr = f3(1.f, 1.f, 1.f);
        Lo = f3(0.f, 0.f, 0.f);
        bounce = 0;
        alive = true;
      }
      cur += take;
      if (take) idle = 0;
    }
    if (!__syncthreads_or(idle != 0xffffffffu || more)) break;
    // the shadow ray of the last step, then the path's ray
    bool helped = false, helper = false;
    int pairs = 0, peer = lane;
    float4 ao = make_float4(0.f, 0.f, 0.f, 0.f), ad = ao;  // a helper's ray
    if constexpr (kPair) {
      const unsigned below = (1u << lane) - 1u;
      const unsigned both = __ballot_sync(0xffffffffu, alive && shadow);
      const unsigned none = __ballot_sync(0xffffffffu, !alive && !shadow);
      pairs = min(__popc(both), __popc(none));
      if (pairs) {
        const int rank = __popc((alive ? both : none) & below);
        helped = alive && shadow && rank < pairs;
        helper = !alive && !shadow && rank < pairs;
        if (helped) lane_of[wp][0][rank] = (uint8_t)lane;
        if (helper) lane_of[wp][1][rank] = (uint8_t)lane;
        __syncwarp();
        if (helped || helper) peer = lane_of[wp][helped][rank];
        ao = shfl4(sh_o, peer);
        ad = shfl4(sh_d, peer);
      }
    }
    int lit = 0;  // the shadow ray traced here met nothing (2: its stack overflowed)
    Hit hit{-1.f, kNoHit, 0.f, 0.f};
    if constexpr (kOneNode) {
      // one copy of the loop for both rays: the kernel's code does not fit the
      // instruction caches
#pragma unroll 1
      for (int ray = 0; ray < 2; ray++) {
        const bool any = ray == 0 || (kPair && !alive);
        const bool live = !kPair ? (ray == 0 ? shadow : alive)
                                 : ray == 0 ? alive && shadow && !helped : alive || shadow || helper;
        if (!__any_sync(0xffffffffu, live)) continue;
        const float4 ro = helper ? ao : any ? sh_o : o4, rd = helper ? ad : any ? sh_d : d4;
        Hit h;
        trace_one_node<false>(g, live, any, f3(ro), f3(rd), 0.001f, any ? ro.w : kInfF,
                              __float_as_uint(any ? rd.w : ro.w), h);
        if (!any) hit = h;
        else if (live) lit = h.prim == kNoHit;
      }
    } else {
      Trav s;
      bool any = helper || (shadow && !helped), busy = any || alive;
      if (busy) {
        const float4 ro = helper ? ao : any ? sh_o : o4, rd = helper ? ad : any ? sh_d : d4;
        trav_init(s, f3(ro), f3(rd), 0.001f, any ? ro.w : kInfF, __float_as_uint(any ? rd.w : ro.w), sc.root, stack);
      }
      for (;;) {
        const bool testing = busy && s.testing();
        const unsigned busy_mask = __ballot_sync(0xffffffffu, busy), test_mask = __ballot_sync(0xffffffffu, testing);
        if (!busy_mask) break;
        if (trav_test_now(test_mask, busy_mask)) {
          if (testing) trav_prim<false>(sc, s, any, stack, nullptr);
        } else if (busy && !testing && s.node >= 0) {
          trav_visit<false>(sc, s, stack, nullptr);
        }
        if (busy && s.done()) {
          if (any) {
            lit = s.hit == kOverflowHit ? 2 : s.hit == kNoHit;
            any = false;
            busy = alive;
            if (busy) trav_init(s, f3(o4), f3(d4), 0.001f, kInfF, __float_as_uint(o4.w), sc.root, stack);
          } else {
            if (s.hit == kOverflowHit) {
              err.report(path, kErrStackOverflow);
              s.hit = kNoHit;
            }
            hit = s.result();
            busy = false;
          }
        }
      }
    }
    if (pairs) {
      const int answer = __shfl_sync(0xffffffffu, lit, peer);
      if (helped) lit = answer;
    }
    if (shadow) {
      if (lit == 2) err.report(path, kErrStackOverflow);
      else if (lit) Lo = f3(Lo.x + sh_c.x, Lo.y + sh_c.y, Lo.z + sh_c.z);
    }
    __syncthreads();
    if (shadow && !alive) P.Lout[path] = make_float4(Lo.x, Lo.y, Lo.z, 0.f);
    shadow = false;
    if (alive) {
      ShadeOut out;
      shade_step(sc, o4, d4, make_float4(hit.t, __uint_as_float(hit.prim), hit.u, hit.v), ids, w4, thr, ch.seed,
                 bounce, out, []() {}, [&](float3 p, float3 dir, float dist, uint32_t prim, float3 c) {
                   shadow = true;
                   sh_o = make_float4(p.x, p.y, p.z, dist - 0.001f);
                   sh_d = make_float4(dir.x, dir.y, dir.z, __uint_as_float(prim));
                   sh_c = c;
                 });
      o4 = out.o;
      d4 = out.d;
      w4 = out.w;
      thr = out.thr;
      ids = out.ids;
      bounce++;
      if (!out.cont || !is_zero(out.L)) Lo = f3(Lo.x + out.L.x, Lo.y + out.L.y, Lo.z + out.L.z);
      if (!out.cont) {
        alive = false;
        if (!shadow) P.Lout[path] = make_float4(Lo.x, Lo.y, Lo.z, 0.f);
      }
    }
  }
}

void launch_pt_paths(const DevScene& sc, const DevFilm& film, const DevPaths& P, const ChunkDesc& ch, int sms,
                     cudaStream_t st) {
  auto run = [&](auto kernel, int block, auto geo) {
    kernel<<<sms * (kPathsThreads / block), block, 0, st>>>(sc, film, P, ch, geo);
  };
  // In a one-node scene a ray's loop takes the time of its slowest lane anyway,
  // and pairing pays only while most lanes are idle (Cornell box without / with
  // it 125 / 112 us at 16,384 paths, 130 / 117 at 36,864, 137 / 141 at 65,536,
  // 258 / 269 at 147,456; textured shapes 345 / 357 at 449,790).
  const bool few = ch.npix * ch.layers <= (uint32_t)sms * 256u;
  if (!one_node(sc)) run(k_pt_paths<false, true>, paths_block(false), NoGeom{});
  else if (few) run(k_pt_paths<true, true>, paths_block(true), *sc.one);
  else run(k_pt_paths<true, false>, paths_block(true), *sc.one);
}

// ----------------------------------------------------------------- accumulate
// PixelStats.AddSample (pkg/renderer/stats.go:41-47), in sample order per pixel
__global__ void k_accumulate(DevFilm film, DevPaths P, ChunkDesc ch) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ch.npix; i += gridDim.x * blockDim.x) {
    uint32_t pix = ch.pix_list ? ch.pix_list[ch.pix0 + i] : ch.pix0 + i;
    float4 acc = film.rgbl[pix];
    float l2 = film.lum2[pix];
    for (uint32_t layer = 0; layer < ch.layers; layer++) {
      float4 c = P.Lout[layer * ch.npix + i];
      float lum = luminance(f3(c));
      acc.x += c.x;
      acc.y += c.y;
      acc.z += c.z;
      acc.w += lum;
      l2 += lum * lum;
    }
    film.rgbl[pix] = acc;
    film.lum2[pix] = l2;
    film.count[pix] += ch.layers;
  }
}

void launch_accumulate(const DevFilm& film, const DevPaths& P, const ChunkDesc& ch, int block, cudaStream_t st) {
  k_accumulate<<<launch_grid(ch.npix, block, 0), block, 0, st>>>(film, P, ch);
}

}  // namespace gprt

namespace gprt {

void carve_paths(unsigned char* base, uint32_t cap, bool multi, DevPaths& P) {
  size_t f4 = align256((size_t)cap * sizeof(float4)), f8 = align256((size_t)cap * 2 * sizeof(float4));
  unsigned char* p = base;
  auto take = [&](size_t n) {
    unsigned char* r = p;
    p += n;
    return r;
  };
  P.counters = reinterpret_cast<uint32_t*>(take(256));
  for (int k = 0; k < 2; k++) {
    PathBuf& Q = P.q[k];
    Q.ray = reinterpret_cast<float4*>(take(f8));
    Q.st = reinterpret_cast<float4*>(take(f8));
    Q.thr = reinterpret_cast<float4*>(take(f4));
  }
  P.hit = reinterpret_cast<float4*>(take(f4));
  P.Lout = reinterpret_cast<float4*>(take(f4));
  P.sh_o = reinterpret_cast<float4*>(take(f4));
  P.sh_d = reinterpret_cast<float4*>(take(f4));
  P.sh_c = reinterpret_cast<float4*>(take(f4));
  P.sh_root = multi ? reinterpret_cast<int*>(take(align256((size_t)cap * sizeof(int)))) : nullptr;
  P.order = reinterpret_cast<uint32_t*>(take(align256((size_t)cap * sizeof(uint32_t))));
  P.capacity = cap;
}

}  // namespace gprt
