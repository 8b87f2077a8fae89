// pt_shade.cuh - one level of the path tracer for one path, shared by the
// single-job wavefront (kernels_pt.cu) and the multi-job serving wavefront
// (server.cu).
#pragma once

#include "device.cuh"
#include "kernels.h"

namespace gprt {

// The state a shading step leaves: the continuing path (when `cont`).  Its
// shadow ray is queued as soon as next-event estimation produces it.
struct ShadeOut {
  bool cont;
  Reserve slot;  // its place in the next queue
  bool keep_thr;   // the throughput is part of the state
  float4 o, d, w;  // next ray origin (+ skip prim), direction (+ BVH root), weight (+ origin index)
  float3 thr, L;   // L: the radiance this level added
  uint4 ids;
};

// One level of rayColorRecursive (pkg/integrator/path_tracing.go:35-104) with
// CalculateDirectLighting (:116-157), CalculateIndirectLighting (:160-189)
// and ApplyRussianRoulette (:193-220), for a path at depth index `bounce`
// (= MaxDepth - depth) whose ray (o4, d4) met h4, with radiance weight w4 (and
// origin index) and roulette throughput thr.  The Russian-roulette draw
// happens first at every level, as in the reference.  out.L is the radiance
// the level adds; it is zero where the path continues (emitters do not
// scatter), unless the weight is not finite.
// The shadow ray of next-event estimation goes to
// `shadow(point, direction, light distance, primitive left, contribution)` as
// soon as it is known, so its state is not held to the end of the step.
// `goes_on()` is called when the path is known to continue, before next-event
// estimation: the wavefront reserves the path's place in the next queue there,
// and the atomic's way to L2 and back passes under it (reserved at the end
// instead: Cornell box 400^2 x 64 7.31 against 7.19 ms, 32 sphere scenes and
// 1.3 M triangles the same.  Shadow rays at the path's own index would need no
// atomic, but leave holes in their queue, which cost the Cornell box 10 %).
template <class Continue, class Shadow>
__device__ __forceinline__ void shade_step(const DevScene& sc, float4 o4, float4 d4, float4 h4, uint4 ids, float4 w4,
                                           float3 thr, uint64_t seed, int bounce, ShadeOut& out,
                                           Continue goes_on, Shadow shadow) {
  out.cont = false;
  float3 d = f3(d4);
  float3 W = f3(w4), L = f3(0.f, 0.f, 0.f);
  out.o = o4;
  out.d = d4;
  Rng rng;
  rng.init(seed, ids.x, ids.y, ids.z);
  // ApplyRussianRoulette: currentBounce = MaxDepth - depth = bounce
  float u = rng.next();
  bool dead = false;
  if (bounce >= sc.rr_min_bounces) {
    float surv = fminf(0.95f, fmaxf(0.5f, luminance_xy(thr)));
    if (u > surv) dead = true;
    else W *= 1.0f / surv;
  }
  bool cont = false;
  if (!dead) {
    uint32_t prim = __float_as_uint(h4.y);
    if (prim == kNoHit) {
      L += W * background(sc, d);  // infinite-light emission of a missed ray
    } else {
      Hit h{h4.x, prim, h4.z, h4.w};
      Surface s;
      surface_at(sc, f3(o4), d, h, s, true);
      DevMaterial m = load_material(sc, s.mat);
      L += W * emitted(m, s.front, d);  // getEmittedLight (:108-113)
      Scatter sc_;
      if (scatter(sc, m, d, s, rng, sc_)) {
        if (sc_.pdf <= 0.f) {
          // calculateSpecularColor (:88-97)
          W *= sc_.att;
          thr *= sc_.att;
          cont = true;
          if (bounce + 1 < sc.max_depth) goes_on();
        } else {
          float3 sd = normalize_yx(sc_.dir);
          float cosine_out = dot(sd, s.n);
          cont = cosine_out > 0.f;
          if (cont && bounce + 1 < sc.max_depth) goes_on();
          // CalculateDirectLighting: light choice + light sample
          if (sc.n_lights > 0) {
            int li = pick_light(sc, rng.next());
            DevLight Lt = sc.lights[li];
            LightSample ls = light_sample(sc, Lt, s.p, s.n, rng.next2());
            ls.pdf *= Lt.prob;
            if (luminance(ls.emission) > 0.f && ls.pdf > 0.f) {
              float cosine = dot(ls.dir, s.n);
              bool delta;
              float mp = mat_pdf(sc, m, d, ls.dir, s.n, delta);
              if (cosine > 0.f && !delta) {
                float w = power_heuristic(ls.pdf, mp);
                float3 f = brdf(sc, m, d, ls.dir, s, true);
                float3 c = W * (f * ls.emission) * (cosine * w / ls.pdf);
                if (!is_zero(c)) shadow(s.p, ls.dir, ls.dist, prim, c);
              }
            }
          }
          // CalculateIndirectLighting
          if (cont) {
            float lp = total_light_pdf(sc, s.p, s.n, sd);
            float w = power_heuristic(sc_.pdf, lp);
            W *= sc_.att * (cosine_out * w / sc_.pdf);
            thr *= sc_.att * (cosine_out / sc_.pdf);
          }
        }
        if (cont) {
          out.o = make_float4(s.p.x, s.p.y, s.p.z, __uint_as_float(prim));
          out.d = make_float4(sc_.dir.x, sc_.dir.y, sc_.dir.z, d4.w);
        }
      }
    }
  }
  out.cont = cont && (bounce + 1 < sc.max_depth);
  out.L = L;
  out.w = make_float4(W.x, W.y, W.z, w4.w);
  out.thr = thr;
  out.ids = make_uint4(ids.x, ids.y, rng.pos, ids.w);
}

// Whether roulette can end a path of the scene (its throughput is kept).
__device__ __forceinline__ bool roulette(const DevScene& sc) { return sc.rr_min_bounces < sc.max_depth; }

// shade_step for slot i of queue `cur`.  The shadow ray goes to P's shadow
// queue (its contribution, when unoccluded, is added to the path's radiance
// at its origin index).
__device__ __forceinline__ void shade_path(const DevScene& sc, const DevPaths& P, int cur, uint32_t i, float4 w4, uint4 ids,
                                           uint64_t seed, int bounce, ShadeOut& out) {
  const PathBuf& Q = P.q[cur];
  float4 o4, d4;
  load32(Q.ray + 2 * (size_t)i, o4, d4);
  const float4 h4 = P.hit[i];
  float3 thr = f3(1.f, 1.f, 1.f);
  if (bounce > 0 && roulette(sc)) thr = f3(Q.thr[i]);
  out.keep_thr = roulette(sc);
  shade_step(sc, o4, d4, h4, ids, w4, thr, seed, bounce, out,
             [&]() { out.slot = warp_reserve(&P.counters[cur ^ 1]); },
             [&](float3 p, float3 dir, float dist, uint32_t prim, float3 c) {
               // one warp-aggregated append among the lanes here
               uint32_t ss = warp_append(&P.counters[2], true);
               P.sh_o[ss] = make_float4(p.x, p.y, p.z, dist - 0.001f);
               P.sh_d[ss] = make_float4(dir.x, dir.y, dir.z, __uint_as_float(prim));
               P.sh_c[ss] = make_float4(c.x, c.y, c.z, w4.w);  // w4.w: the origin index
               if (P.sh_root) P.sh_root[ss] = __float_as_int(d4.w);
             });
}

// Brings the shading inputs of slot i of queue Q into L2 ahead of their use: a
// grid-stride shading loop issues this for its next slot at the end of the
// current one, so the next iteration's loads meet L2 instead of DRAM.
__device__ __forceinline__ void prefetch_slot(const PathBuf& Q, const float4* hits, uint32_t i) {
  const void* a[3] = {Q.ray + 2 * (size_t)i, Q.st + 2 * (size_t)i, hits + i};
#pragma unroll
  for (int k = 0; k < 3; k++) asm volatile("prefetch.global.L2 [%0];" ::"l"(a[k]));
}

// The shading group of primitive p, stored in its record by the builders.
__device__ __forceinline__ int prim_group(const DevScene& sc, uint32_t p) {
  if (p < sc.quad_base) return __float_as_int(__ldg(sc.tris + (size_t)p * 3 + 1).w);
  if (p < sc.sphere_base) return __float_as_int(__ldg(sc.quads + (size_t)(p - sc.quad_base) * 5 + 2).w);
  if (p < sc.quadric_base) return __float_as_int(__ldg(sc.spheres + (size_t)(p - sc.sphere_base) * 2 + 1).y);
  return __float_as_int(__ldg(sc.quadrics + (size_t)(p - sc.quadric_base) * 5 + 4).w);
}

// The slot order the shading kernels read for queue `cur`, by shading group
// (`group(i, prim)` for slot i's hit on primitive prim; missed rays, which
// only look up the background, are group 3): group 0 from the front, then,
// from the back, groups 1, 2 and 3.  Each block of 1,024 slots takes one
// range from the front and one from the back (one atomic each) and lays its
// back range out group by group, so warps run one kind of shading (next-event
// estimation on all lanes or on none; metal, glass or finished paths) instead
// of mixing them lane by lane.  Every path is shaded exactly as in queue
// order.
template <class Group>
__device__ __forceinline__ void order_slots(const DevPaths& P, int cur, Group group) {
  constexpr int G = kShadeGroups;
  __shared__ uint32_t wc[G][32];
  __shared__ uint32_t bfront, bback, boff[G];
  const uint32_t n = P.counters[cur];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  for (uint32_t base = blockIdx.x * 1024u; base < n; base += gridDim.x * 1024u) {
    uint32_t i = base + threadIdx.x;
    bool live = i < n;
    uint32_t prim = live ? __float_as_uint(P.hit[i].y) : kNoHit;
    int g = prim != kNoHit && prim != kOverflowHit ? group(i, prim) : G - 1;
    unsigned mine = 0;  // the lanes of this warp in group g
#pragma unroll
    for (int k = 0; k < G; k++) {
      unsigned m = __ballot_sync(0xffffffffu, live && g == k);
      if (g == k) mine = m;
      if (lane == 0) wc[k][w] = __popc(m);
    }
    __syncthreads();
    if (threadIdx.x < G) {  // exclusive scan of each group's warp counts
      uint32_t acc = 0;
      for (int k = 0; k < 32; k++) {
        uint32_t c = wc[threadIdx.x][k];
        wc[threadIdx.x][k] = acc;
        acc += c;
      }
      boff[threadIdx.x] = acc;  // the group's total, for now
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      // back-range entry j sits at n - 1 - (bback + j): the last group takes
      // the smallest j (the highest positions), group 1 the largest
      uint32_t back = 0;
      for (int k = G - 1; k >= 1; k--) {
        uint32_t t = boff[k];
        boff[k] = back;
        back += t;
      }
      bfront = boff[0] ? atomicAdd(&P.counters[6], boff[0]) : 0u;
      bback = back ? atomicAdd(&P.counters[7], back) : 0u;
    }
    __syncthreads();
    if (live) {
      uint32_t r = wc[g][w] + __popc(mine & below);
      if (g == 0) P.order[bfront + r] = i;
      else P.order[n - 1u - (bback + boff[g] + r)] = i;
    }
    __syncthreads();  // the counts and bases are rewritten for the next range
  }
}

// Moves a continuing path to the next queue; a finished path adds the
// radiance of its last level at its origin index (where its unoccluded shadow rays add
// theirs; raygen clears it).  `live` is false for lanes without a path.
__device__ __forceinline__ void push_shade_out(const DevPaths& P, int cur, bool live, const ShadeOut& o) {
  if (!live) return;
  if (o.cont) {
    const uint32_t slot = reserved_slot(o.slot);
    const PathBuf& N = P.q[cur ^ 1];
    store32(N.ray + 2 * (size_t)slot, o.o, o.d);
    store32(N.st + 2 * (size_t)slot, o.w, as_float4(o.ids));
    if (o.keep_thr) N.thr[slot] = make_float4(o.thr.x, o.thr.y, o.thr.z, 0.f);
    if (is_zero(o.L)) return;  // else it is not a number: the sum is not one either, whenever it is added
  }
  float4* dst = P.Lout + __float_as_uint(o.w.w);
  float4 a = *dst;
  *dst = make_float4(a.x + o.L.x, a.y + o.L.y, a.z + o.L.z, 0.f);
}

}  // namespace gprt
