// kernels_bdpt.cu - bidirectional path tracing.
//
// Restates BDPTIntegrator.RayColor (pkg/integrator/bdpt.go:73-102): a camera
// subpath and a light subpath are generated (generateCameraPath :106-135,
// generateLightPath :139-202, extendPath :206-291), every (s,t) strategy is
// evaluated (:294-561) and weighted by calculateMISWeight
// (pkg/integrator/bdpt_mis.go:13-335).  t=1 light-tracing contributions are
// splatted into the film's splat buffer with atomic adds and applied after
// the pass (processSplats, pkg/renderer/progressive.go:371-391).
//
// Every helper is inlined: an out-of-line call takes its vertex and scene
// arguments by reference, which puts them in each thread's local stack
// (3 KB per thread for the strategy kernel, 245 MB at full occupancy, more
// than L2), and that stack traffic went to DRAM.
//
// Per chunk of samples:
//   k_bdpt_camgen      the camera vertex and ray of every sample;
//   k_bdpt_trace       (per bounce) closest hits of the subpath queue;
//   k_bdpt_extend      (per bounce) each subpath's next vertex into a global
//                      vertex store (fields indexed [vertex][sample]) and the
//                      continuing subpaths compacted into the other queue; a
//                      camera subpath that ends starts its light subpath;
//   k_bdpt_subpaths    (small chunks, instead of the three above) both subpaths
//                      of every sample in one launch;
//   k_bdpt_list        lists, per strategy (s,t) and window of 16,384
//                      samples, the samples that have it;
//   k_bdpt_prefix      each strategy class's prefix sums of the list counts
//                      in (window, strategy) order;
//   k_bdpt_strategies  (small chunks: k_bdpt_strategies_all, one launch for the
//                      four classes; connections by run_connections, in three
//                      steps) one thread per listed (strategy, sample) item, in
//                      (window, strategy) order, so every strategy of a
//                      window runs while its vertices are in L2; the
//                      items of a strategy in consecutive threads: each warp
//                      runs a single (s,t) for 32 samples that have it, so
//                      control flow is uniform and neighbouring warps share
//                      code; its sampler position is the sample's position
//                      after the subpaths plus the draws of the strategies
//                      before it (draws_before);
//   k_bdpt_sum         adds each sample's strategy contributions in the
//                      reference's s-major order.
#include <algorithm>

#include "device.cuh"
#include "kernels.h"

namespace gprt {

namespace {


constexpr int kFlagLight = 1, kFlagCamera = 2, kFlagSpecular = 4, kFlagInfinite = 8, kFlagFront = 16;

struct BVert {  // bdpt.go:14-36
  float3 p, n, beta, Le, wi;
  float2 uv;  // surface UV (textured scenes)
  float fwd, rev;
  int mat;    // material index, -1 for none
  int light;  // index in the light table, -1 for none
  uint32_t prim;
  int flags;
  __device__ bool is(int f) const { return (flags & f) != 0; }
};

__device__ __forceinline__ bool light_is_area(const DevScene& sc, int li) {
  int k = sc.lights[li].kind;
  return k == kLightQuad || k == kLightSphere || k == kLightDisc || k == kLightDiscSpot;
}

// Vertex.IsOnSurface (bdpt.go:42-49)
__device__ __forceinline__ bool on_surface(const DevScene& sc, const BVert& v) {
  if (v.is(kFlagLight) && v.light >= 0) return light_is_area(sc, v.light);
  return v.mat >= 0;
}

// convertSolidAngleToAreaPdf (bdpt_mis.go:341-363)
__device__ __forceinline__ float to_area(const DevScene& sc, const BVert& from, const BVert& next, float pdf) {
  if (next.is(kFlagInfinite)) return pdf;
  float3 d = next.p - from.p;
  float d2 = dot(d, d);
  if (d2 == 0.f) return 0.f;
  float inv = 1.0f / d2;
  if (on_surface(sc, next)) pdf *= fabsf(dot(d * sqrtf(inv), next.n));
  return pdf * inv;
}

// ---------------------------------------------------------------- camera
// MapRayToPixel (camera.go:280-316)
__device__ __forceinline__ bool map_ray_to_pixel(const DevCamera& c, float3 o, float3 d, int& px, int& py) {
  float3 ipc = c.center - c.w * c.focus_distance;
  float t = dot(ipc - o, c.w) / dot(d, c.w);
  if (t <= 0.f) return false;
  float3 rel = o + d * t - ipc;
  float nx = (dot(rel, c.u) + c.viewport_width / 2.f) / c.viewport_width;
  float ny = (dot(rel, c.v) + c.viewport_height / 2.f) / c.viewport_height;
  float fx = nx * (float)c.width, fy = ny * (float)c.height;
  if (!(fx > -1.f && fx < (float)c.width + 1.f && fy > -1.f && fy < (float)c.height + 1.f)) return false;
  int x = (int)fx, y = (int)fy;  // Go int() truncates toward zero
  if (x >= 0 && x < c.width && y >= 0 && y < c.height) {
    px = x;
    py = y;
    return true;
  }
  return false;
}
// CalculateRayPDFs direction pdf (camera.go:194-216)
__device__ __forceinline__ float camera_dir_pdf(const DevCamera& c, float3 o, float3 d) {
  float ct = dot(d, c.forward);
  if (ct <= c.cos_total_width) return 0.f;
  int x, y;
  if (!map_ray_to_pixel(c, o, d, x, y)) return 0.f;
  return 1.0f / (c.image_plane_area * ct * ct * ct);
}
// EvaluateRayImportance (camera.go:263-277)
__device__ __forceinline__ float camera_importance(const DevCamera& c, float3 d) {
  float ct = dot(d, c.forward);
  if (ct < c.cos_total_width) return 0.f;
  float c2 = ct * ct;
  return 1.0f / (c.image_plane_area * c.lens_area * c2 * c2);
}

// ---------------------------------------------------------------- lights
// SampleEmission (quad_light.go:113-145, sphere_light.go:169-184,
// disc_light.go:103-110, disc_spot_light.go:210-240, point_spot_light.go:161-191,
// light_sampling.go:58-115 for the infinite lights)
__device__ __forceinline__ void sample_emission(const DevScene& sc, const DevLight& L, float2 sp, float2 sd, float3& p, float3& n,
                                float3& dir, float3& Le, float& area_pdf, float& dir_pdf) {
  if (L.kind == kLightQuad) {
    const float4* Q = sc.quads + (size_t)L.prim * 5;
    float3 c = f3(__ldg(Q)), U = f3(__ldg(Q + 1)), V = f3(__ldg(Q + 2)), N = f3(__ldg(Q + 3));
    p = c + U * sp.x + V * sp.y;
    dir = sample_cosine_hemisphere(N, sd);
    n = N;
    area_pdf = 1.0f / L.area;
    dir_pdf = dot_xy(dir, N) / kPi;
    Le = L.a;
    return;
  }
  if (L.kind == kLightSphere) {
    float4 S = make_float4(L.pos.x, L.pos.y, L.pos.z, L.radius);
    float z = 1.f - 2.f * sp.x;
    float r = sqrtf(fmaxf(0.f, 1.f - z * z));
    float s_, c_;
    sincosf(2.f * kPi * sp.y, &s_, &c_);
    float3 ld = f3(r * c_, r * s_, z);
    p = f3(S) + ld * S.w;
    n = ld;
    dir = sample_cosine_hemisphere(n, sd);
    dir_pdf = dot_xy(dir, n) / kPi;
    area_pdf = 1.0f / (4.f * kPi * S.w * S.w);
    Le = L.a;
    return;
  }
  if (L.kind == kLightDisc || L.kind == kLightDiscSpot || L.kind == kLightPointSpot) {
    if (L.kind == kLightPointSpot) {
      p = L.pos;
      area_pdf = 1.f;
    } else {
      const float4* Q = sc.quadrics + (size_t)L.prim * 5;
      p = disc_point(Q, sp);
      n = f3(__ldg(Q + 1));
      area_pdf = 1.0f / L.area;
    }
    if (L.kind == kLightDisc) {  // SampleEmissionDirection (light_sampling.go:58-80)
      dir = sample_cosine_hemisphere(n, sd);
      dir_pdf = dot_xy(dir, n) / kPi;
      Le = L.a;
      return;
    }
    dir = sample_cone(L.b, L.cos_total, sd);
    Le = L.a * spot_falloff(L, dot(dir, L.b));
    dir_pdf = 1.0f / (2.f * kPi * (1.f - L.cos_total));  // UniformConePDF (light_sampling.go:83-85)
    if (L.kind == kLightPointSpot) n = dir;
    return;
  }
  // SampleInfiniteLight (light_sampling.go:89-115)
  float3 d = sample_on_unit_sphere(sd);
  float3 up = fabsf(d.x) > 0.9f ? f3(0.f, 1.f, 0.f) : f3(1.f, 0.f, 0.f);
  float3 right = normalize(cross(d, up));
  up = normalize(cross(right, d));
  float2 ds = sample_unit_disk(sp);
  float R = sc.world_radius;
  float3 dp = sc.world_center + right * (ds.x * R) + up * (ds.y * R);
  p = dp + d * (-R);
  n = -d;
  dir = d;
  area_pdf = 1.0f / (kPi * R * R);
  dir_pdf = 1.0f / (4.f * kPi);
  Le = L.kind == kLightUniformInfinite ? L.a : gradient_emission(L, d);
}

// PDF_Le direction pdf (quad_light.go:148-185, sphere_light.go:187-209,
// disc_light.go:113-136, disc_spot_light.go:243-264, point_spot_light.go:194-214,
// uniform_infinite_light.go:94-106); pos receives the position pdf
__device__ __forceinline__ float pdf_le(const DevScene& sc, const DevLight& L, float3 p, float3 dir, float& pos) {
  pos = 0.f;
  if (L.kind == kLightQuad) {
    const float4* Q = sc.quads + (size_t)L.prim * 5;
    float3 c = f3(__ldg(Q)), U = f3(__ldg(Q + 1)), V = f3(__ldg(Q + 2)), N = f3(__ldg(Q + 3));
    float3 tp = p - c;
    float uu = dot(U, U), vv = dot(V, V), uv = dot(U, V);
    if (uu == 0.f || vv == 0.f) return 0.f;
    float det = uu * vv - uv * uv;
    if (fabsf(det) < 1e-8f) return 0.f;
    float tu = dot(tp, U), tv = dot(tp, V);
    float al = (vv * tu - uv * tv) / det, be = (uu * tv - uv * tu) / det;
    if (al < 0.f || al > 1.f || be < 0.f || be > 1.f) return 0.f;
    float3 rec = c + U * al + V * be;
    if (length(rec - p) > 0.001f * fmaxf(1.f, length(p) * 1e-3f)) return 0.f;
    pos = 1.0f / L.area;
    float ct = dot(dir, N);
    return ct <= 0.f ? 0.f : ct / kPi;
  }
  if (L.kind == kLightSphere) {
    float4 S = make_float4(L.pos.x, L.pos.y, L.pos.z, L.radius);
    float dc = length(p - f3(S));
    if (!(fabsf(dc - S.w) <= 0.001f * fmaxf(1.f, fabsf(S.w) * 1e-3f))) return 0.f;
    float3 n = normalize(p - f3(S));
    if (dot(dir, n) <= 0.f) return 0.f;
    pos = 1.0f / (4.f * kPi * S.w * S.w);
    return dot(dir, n) / kPi;
  }
  if (L.kind == kLightDisc || L.kind == kLightDiscSpot) {
    const float4* Q = sc.quadrics + (size_t)L.prim * 5;
    float4 g0 = __ldg(Q);
    float3 N = f3(__ldg(Q + 1));
    // validatePointOnDisc (disc_light.go:153-165), tolerance 0.001
    float3 tp = p - f3(g0);
    float h = dot(tp, N);
    if (fabsf(h) > 0.001f || length(tp - N * h) > g0.w) return 0.f;
    float ct = dot(dir, N);
    if (ct <= 0.f) return 0.f;
    if (L.kind == kLightDiscSpot && dot(dir, L.b) < L.cos_total) {
      pos = 1.0f / L.area;
      return 0.f;
    }
    pos = 1.0f / L.area;
    return ct / kPi;
  }
  if (L.kind == kLightPointSpot) {
    if (length(p - L.pos) > 0.001f || dot(dir, L.b) < L.cos_total) return 0.f;
    pos = 1.f;
    return 1.0f / (2.f * kPi * (1.f - L.cos_total));
  }
  if (sc.world_radius <= 0.f) return 0.f;
  pos = 1.0f / (kPi * sc.world_radius * sc.world_radius);
  return 1.0f / (4.f * kPi);
}

// calculateInfiniteLightDensity (bdpt_mis.go:313-335)
__device__ float infinite_density(const DevScene& sc, float3 p, float3 n, float3 dir) {
  float t = 0.f;
  for (int i = 0; i < sc.n_lights; i++) {
    DevLight L = sc.lights[i];
    if (L.kind == kLightUniformInfinite || L.kind == kLightGradientInfinite) {
      float c = dot(dir, n);
      t += (c <= 0.f ? 0.f : c / kPi) * L.prob;
    }
  }
  return t;
}

// ---------------------------------------------------------------- BRDF at a vertex
// evaluateBRDF (bdpt.go:564-583)
__device__ __forceinline__ float3 vertex_brdf(const DevScene& sc, const BVert& v, float3 out, bool radiance) {
  if (v.is(kFlagInfinite)) return f3(0.f, 0.f, 0.f);
  if (v.is(kFlagLight) && v.mat < 0) return f3(1.f, 1.f, 1.f);
  if (v.mat < 0) return f3(0.f, 0.f, 0.f);
  Surface s;
  s.p = v.p;
  s.n = v.n;
  s.front = v.is(kFlagFront);
  s.mat = v.mat;
  s.uv = v.uv;
  return brdf(sc, load_material(sc, v.mat), v.wi, out, s, radiance);
}

// calculateLightPdf (bdpt_mis.go:239-272)
__device__ __forceinline__ float vertex_light_pdf(const DevScene& sc, const BVert& cur, const BVert& to) {
  float3 w = to.p - cur.p;
  float inv = 1.0f / dot(w, w);
  w = w * sqrtf(inv);
  float pdf = 0.f;
  if (cur.is(kFlagLight)) {
    if (cur.is(kFlagInfinite)) {
      float r = sc.world_radius == 0.f ? 1.f : sc.world_radius;
      pdf = 1.0f / (kPi * r * r);
    } else if (cur.light >= 0) {
      float pos;
      pdf = pdf_le(sc, sc.lights[cur.light], cur.p, w, pos) * inv;
    }
  }
  if (on_surface(sc, to)) pdf *= fabsf(dot(to.n, w));
  return pdf;
}

// calculateVertexPdf (bdpt_mis.go:186-236)
__device__ __forceinline__ float vertex_pdf(const DevScene& sc, const BVert& cur, const BVert* prev, const BVert& next) {
  if (cur.is(kFlagLight)) return vertex_light_pdf(sc, cur, next);
  float3 wn = next.p - cur.p;
  if (dot(wn, wn) == 0.f) return 0.f;
  wn = normalize(wn);
  float3 wp = f3(0.f, 0.f, 0.f);
  if (prev) {
    wp = prev->p - cur.p;
    if (dot(wp, wp) == 0.f) return 0.f;
    wp = normalize(wp);
  } else if (!cur.is(kFlagCamera)) {
    return 0.f;
  }
  float pdf;
  if (cur.is(kFlagCamera)) {
    pdf = camera_dir_pdf(sc.cam, cur.p, wn);
    if (pdf == 0.f) return 0.f;
  } else if (cur.mat >= 0) {
    bool delta;
    pdf = mat_pdf(sc, load_material(sc, cur.mat), wp, wn, cur.n, delta);
    if (delta) return 0.f;
  } else {
    return 0.f;
  }
  return to_area(sc, cur, next, pdf);
}

// calculateLightOriginPdf (bdpt_mis.go:275-308)
__device__ __forceinline__ float light_origin_pdf(const DevScene& sc, const BVert& lv, const BVert& to) {
  float3 w = to.p - lv.p;
  if (dot(w, w) == 0.f) return 0.f;
  w = normalize(w);
  if (lv.is(kFlagInfinite)) return infinite_density(sc, to.p, to.n, -w);
  if (!lv.is(kFlagLight) || lv.light < 0) return 0.f;
  if (sc.n_lights == 0) return 0.f;
  float pos;
  pdf_le(sc, sc.lights[lv.light], lv.p, w, pos);
  return pos * sc.lights[lv.light].prob;
}

// Any-hit test of a connection / shadow ray (one call site for all strategies).
template <bool kOneNode>
__device__ __forceinline__ bool occluded(const DevScene& sc, const Geom<kOneNode>& geo, float3 o, float3 d, float tmax,
                                         uint32_t skip, int* err) {
  Hit hh;
  return trace<true, kOneNode>(sc, geo, o, d, 0.001f, tmax, skip, hh, err);
}

// ---------------------------------------------------------------- vertex store
// Subpath vertices live in global memory as 5 float4 fields indexed
// [vertex * ns + sample], so the 32 lanes of a warp (32 consecutive samples)
// read one field of one vertex in a single coalesced access: position and
// material | flags, normal and forward pdf, throughput and incoming direction
// (x), incoming direction (y, z), primitive and light, emission.  The first
// two are what a pdf request of the MIS weight reads of a vertex, the first
// four what a strategy reads of the vertex it ends at; the emission is read at
// a camera path's last vertex only.  What is known one bounce later (the
// reverse pdf and the MIS prefix) is the vertex's `pdf` record.
__device__ __forceinline__ void put_vert(const DevBdpt& B, int v, uint32_t i, const BVert& x) {
  size_t k = (size_t)v * B.ns + i;
  B.v[0][k] = make_float4(x.p.x, x.p.y, x.p.z, __int_as_float((x.mat + 1) | (x.flags << 24)));
  B.v[1][k] = make_float4(x.n.x, x.n.y, x.n.z, x.fwd);
  B.v[2][k] = make_float4(x.beta.x, x.beta.y, x.beta.z, x.wi.x);
  B.v[3][k] = make_float4(x.wi.y, x.wi.z, __uint_as_float(x.prim), __int_as_float(x.light));
  B.v[4][k] = make_float4(x.Le.x, x.Le.y, x.Le.z, 0.f);
  if (B.uv) B.uv[k] = x.mat >= 0 ? x.uv : make_float2(0.f, 0.f);
}

__device__ __forceinline__ BVert get_vert(const DevBdpt& B, int v, uint32_t i) {
  size_t k = (size_t)v * B.ns + i;
  float4 a = B.v[0][k], b = B.v[1][k], c = B.v[2][k], d = B.v[3][k], e = B.v[4][k];
  BVert x;
  x.p = f3(a);
  int mf = __float_as_int(a.w);
  x.mat = (mf & 0xFFFFFF) - 1;
  x.flags = (mf >> 24) & 0xFF;
  x.n = f3(b);
  x.fwd = b.w;
  x.rev = 0.f;
  x.beta = f3(c);
  x.wi = make_float3(c.w, d.x, d.y);
  x.prim = __float_as_uint(d.z);
  x.light = __float_as_int(d.w);
  x.Le = f3(e);
  x.uv = B.uv ? B.uv[k] : make_float2(0.f, 0.f);
  return x;
}

__device__ __forceinline__ float remap0(float f) { return f != 0.f ? f : 1.f; }

// The MIS prefix of a subpath, in each vertex's pdf record.
// calculateMISWeight (bdpt_mis.go:13-181) walks each subpath from the
// connection outwards, multiplying ratios r_i = remap0(rev_i) / remap0(fwd_i)
// and adding the running product at every connectible vertex; away from the
// two vertices next to the connection those ratios and flags do not depend on
// the strategy, so with the sum over vertices 0..k
//   A_k = r_k * q_k,   q_k = A_{k-1} + c_k
// (camera subpath: from vertex 1, c_k = neither vertex k nor k-1 specular;
// light subpath: from vertex 0, c_k also excludes delta lights) each strategy
// evaluates only its two connection-side steps, on top of q of the vertex
// before the connection's.
__device__ __forceinline__ float prefix_q(int k, bool ok, bool ok_before, float acc) {
  return acc + (ok && (k == 0 || ok_before) ? 1.f : 0.f);
}

// The q of a finished light subpath again (its forward pdfs have changed).
__device__ __forceinline__ void light_prefix(const DevScene& sc, const DevBdpt& B, int base, int len, uint32_t i) {
  float acc = 0.f;
  bool prev_ok = true;  // the previous vertex is neither specular nor a delta light
  for (int k = 0; k < len; k++) {
    size_t at = (size_t)(base + k) * B.ns + i;
    const int flags = __float_as_int(B.v[0][at].w) >> 24 & 0xFF, light = __float_as_int(B.v[3][at].w);
    const float fwd = B.v[1][at].w, rev = B.pdf[at].x;
    const bool ok = !(flags & kFlagSpecular) &&
                    !((flags & kFlagLight) && light >= 0 && sc.lights[light].kind == kLightPointSpot);
    const float q = prefix_q(k, ok, prev_ok, acc);
    B.pdf[at].y = q;
    acc = (remap0(rev) / remap0(fwd)) * q;
    prev_ok = ok;
  }
}

// The vertices of one sample's subpath (camera: base 0, light: base maxv).
struct SubpathRef {
  const DevBdpt* B;
  uint32_t i;
  int base;
  __device__ BVert operator[](int k) const { return get_vert(*B, base + k, i); }
  __device__ size_t at(int k) const { return (size_t)(base + k) * B->ns + i; }
  __device__ float fwd(int k) const { return B->v[1][at(k)].w; }
  __device__ float q(int k) const { return B->pdf[at(k)].y; }
  __device__ bool specular(int k) const { return __float_as_int(B->v[0][at(k)].w) >> 24 & kFlagSpecular; }
};

// ---------------------------------------------------------------- subpath wavefront
// generateCameraPath / generateLightPath / extendPath (bdpt.go:106-291) one
// bounce per launch over a compacted queue of subpaths: a persistent
// closest-hit traversal of the queue, then one thread per slot extends its
// subpath by the vertex hit, compacting the continuing subpaths into the
// other queue.  A sample's light subpath starts, in the same sampler stream,
// in the step that ends its camera subpath, so both kinds share the queue.
// Each vertex is stored when it is created; its reverse pdf (set by the
// scatter at the next vertex, bdpt.go:273-285) and its MIS prefix are stored
// one bounce later.

// A queue slot's state (BdQueue::st).  x: the subpath's length (5 bits),
// bounces (5), the bits below, and from kStLightMask the light vertices whose
// light tracing draws samples; y: the camera subpath's length (5), whether the
// light is infinite, and from kStCamMask the camera vertices whose direct
// lighting draws samples.  Bit s - 2 (t - 2) is strategy s (t): at most 17
// bits for 18 vertices.  Kept along with the subpath, the masks need no second
// pass over its vertices (of up to 2 x max_depth loads one after another, in
// the lane that ends the sample while its warp waits).
constexpr uint32_t kStCamera = 1u << 10, kStOkBefore = 1u << 11, kStOkLast = 1u << 12, kStSurfLast = 1u << 13,
                   kStInfLast = 1u << 14, kStInfinite = 1u << 5;
constexpr int kStLightMask = 15, kStCamMask = 6;

// The subpath vertex is neither specular nor (light subpaths) a delta light:
// it can take part in a connection (bdpt_mis.go:61-178).
__device__ __forceinline__ bool vertex_ok(const DevScene& sc, const BVert& v, bool camera) {
  bool ok = !v.is(kFlagSpecular);
  if (!camera) ok = ok && !(v.is(kFlagLight) && v.light >= 0 && sc.lights[v.light].kind == kLightPointSpot);
  return ok;
}

// convertSolidAngleToAreaPdf (bdpt_mis.go:341-363) towards a vertex known by
// its position, normal and kind.
__device__ __forceinline__ float to_area_at(float3 from, float3 p, float3 n, bool surface, bool infinite, float pdf) {
  if (infinite) return pdf;
  float3 d = p - from;
  float d2 = dot(d, d);
  if (d2 == 0.f) return 0.f;
  float inv = 1.0f / d2;
  if (surface) pdf *= fabsf(dot(d * sqrtf(inv), n));
  return pdf * inv;
}

// The reverse pdf and MIS prefix of a stored vertex, once final.
__device__ __forceinline__ void put_pdf(const DevBdpt& B, int v, uint32_t i, float rev, float q) {
  B.pdf[(size_t)v * B.ns + i] = make_float2(rev, q);
}

// The sample's record for the strategy kernels, once both subpaths are
// stored: lengths, and the strategies that draw uniform numbers
// (draws_before) from the state's masks.
__device__ __forceinline__ void finish_sample(const DevBdpt& B, uint32_t p, int nc, int nl, uint32_t pos, uint32_t pix,
                                              uint32_t sample, uint32_t light_mask, uint32_t cam_mask) {
  B.meta[p] = make_uint4((uint32_t)nc | ((uint32_t)nl << 8), pos, pix, sample);
  B.masks[p] = make_uint2(light_mask << 2, cam_mask << 2);
}

// The walk of calculateMISWeight (bdpt_mis.go:61-178) in prefix form, given
// the reverse pdfs it recomputes next to the connection: cam1, cam2 of camera
// vertices t - 1 and t - 2, lit1, lit2 of light vertices s - 1 and s - 2.
template <int CLS>
__device__ __forceinline__ float mis_walk(const SubpathRef& C, const SubpathRef& Lp, float sampled_fwd, int s, int t,
                                          float cam1, float cam2, float lit1, float lit2) {
  float sum = 0.f;
  if (t >= 2) {  // camera vertices t-1 .. 1
    const float r1 = remap0(cam1) / remap0(C.fwd(t - 1));
    const float inner = t >= 3 ? remap0(cam2) / remap0(C.fwd(t - 2)) * C.q(t - 2) : 0.f;
    sum += r1 * (inner + (C.specular(t - 2) ? 0.f : 1.f));
  }
  if (s >= 1) {  // light vertices s-1 .. 0
    const float q1 = remap0(lit1) / remap0(CLS == 2 ? sampled_fwd : Lp.fwd(s - 1));
    const float inner = s >= 2 ? remap0(lit2) / remap0(Lp.fwd(s - 2)) * Lp.q(s - 2) : 0.f;
    sum += q1 * (inner + 1.f);
  }
  return 1.f / (1.f + sum);
}

// The two reverse pdfs at the end x of a connection to vertex o, whose subpath
// comes from `own` (calculateVertexPdf, bdpt_mis.go:186-236): of x towards o
// coming from own, and towards own coming from o.
__device__ __forceinline__ void end_pdfs(const DevScene& sc, const BVert& x, const BVert& o, const BVert& own,
                                         float& to_o, float& to_own) {
  to_o = to_own = 0.f;
  if (x.is(kFlagLight)) {
#pragma unroll 1
    for (int r = 0; r < 2; r++) {
      float v = vertex_light_pdf(sc, x, r ? own : o);
      if (r) to_own = v;
      else to_o = v;
    }
    return;
  }
  float3 wo = o.p - x.p, wn = own.p - x.p;
  if (x.mat >= 0 && dot(wo, wo) != 0.f && dot(wn, wn) != 0.f) {
    wo = normalize(wo);
    wn = normalize(wn);
    const DevMaterial m = load_material(sc, x.mat);
    bool d1, d2;
    float p1 = mat_pdf(sc, m, wn, wo, x.n, d1), p2 = mat_pdf(sc, m, wo, wn, x.n, d2);
    if (!d1) to_o = to_area(sc, x, o, p1);
    if (!d2) to_own = to_area(sc, x, own, p2);
  }
}

// calculateMISWeight (bdpt_mis.go:13-181) of a strategy of class 0, 1 or 2
// whose stored vertex next to the connection is x: the reverse pdfs the walk
// recomputes there (:61-105 camera side, :140-178 light side), each
// calculateVertexPdf, or for s = 0 at t - 1 calculateLightOriginPdf.
template <int CLS>
__device__ __forceinline__ float mis_weight(const DevScene& sc, const SubpathRef& C, const SubpathRef& Lp,
                                            const BVert& x, const BVert& sampled, int s, int t) {
  if (s + t <= 2) return 1.f;
  float cam1 = 0.f, cam2 = 0.f, lit1 = 0.f, lit2 = 0.f;
  if (CLS == 0) {
    const BVert own = C[t - 2];
    cam1 = light_origin_pdf(sc, x, own);
    cam2 = vertex_pdf(sc, x, nullptr, own);
  } else if (CLS == 1) {
    lit1 = vertex_pdf(sc, sampled, nullptr, x);
    lit2 = vertex_pdf(sc, x, &sampled, Lp[s - 2]);
  } else {
    cam1 = vertex_light_pdf(sc, sampled, x);
    end_pdfs(sc, x, sampled, C[t - 2], lit1, cam2);
  }
  return mis_walk<CLS>(C, Lp, CLS == 2 ? sampled.fwd : 0.f, s, t, cam1, cam2, lit1, lit2);
}

// Uniform numbers the strategies before (s, t) draw, in the reference's
// s-major order: light tracing (s >= 2, t = 1) draws 2 when its light vertex
// is not specular (mask bit s); direct lighting (s = 1, t >= 2) draws 3 when
// its camera vertex is a non-specular surface and the scene has lights (mask
// bit t); every other strategy draws nothing.
__device__ __forceinline__ uint32_t draws_before(int s, int t, uint2 m) {
  if (s == 0) return 0;
  uint32_t lo_t = ((1u << t) - 1u) & ~3u;  // bits 2 .. t-1
  if (s == 1) return 3u * __popc(m.y & lo_t);
  uint32_t lo_s = ((1u << s) - 1u) & ~3u;  // bits 2 .. s-1
  return 3u * __popc(m.y) + 2u * __popc(m.x & lo_s) + (t > 1 ? 2u * ((m.x >> s) & 1u) : 0u);
}

// evaluateBDPTStrategy (bdpt.go:294-561) for strategy (s, t) of sample i;
// returns the weighted contribution to the sample (t = 1 splats instead).
template <int CLS, bool kOneNode>
__device__ __forceinline__ float3 eval_strategy(const DevScene& sc, const Geom<kOneNode>& geo, const DevFilm& film,
                                                const DevBdpt& B, uint32_t i, int s, int t, Rng& rs, int* err) {
  const float3 zero = f3(0.f, 0.f, 0.f);
  SubpathRef C{&B, i, 0}, Lp{&B, i, B.maxv};
  float3 Lc = zero;
  BVert sampled;
  bool splat = false;
  int spx = 0, spy = 0;
  bool test = false;
  float3 ro = zero, rd = f3(0.f, 0.f, 1.f);
  float rt = 0.f;
  uint32_t rskip = kNoHit;
  if (CLS == 0) {
    // evaluatePathTracingStrategy (bdpt.go:317-332): the caller passes t == nc only
    BVert last = C[t - 1];
    Lc = last.Le * last.beta;
  } else if (CLS == 1) {
    // evaluateLightTracingStrategy (bdpt.go:398-486)
    BVert lv = Lp[s - 1];
    if (s <= 1 || lv.is(kFlagSpecular)) return zero;
    float2 cs = rs.next2();
    float2 lens2 = sample_unit_disk(cs);
    float3 lp = sc.cam.center + sc.cam.u * (lens2.x * sc.cam.lens_radius) + sc.cam.v * (lens2.y * sc.cam.lens_radius);
    float3 toRef = lv.p - lp;
    float dist = length(toRef);
    float3 dir = normalize(toRef);
    float cpdf = (dist * dist) / (fabsf(dot(sc.cam.forward, dir)) * sc.cam.lens_area);
    float imp = camera_importance(sc.cam, dir);
    if (imp == 0.f) return zero;  // SampleCameraFromPoint returns nil
    float3 toCam = -dir;
    float3 f = vertex_brdf(sc, lv, toCam, false);
    float cb = imp / cpdf;
    float cosine = dot(toCam, lv.n);
    if (cosine <= 0.f) return zero;
    float3 c = f * cb * lv.beta;
    if (on_surface(sc, lv)) c = c * cosine;
    if (is_zero(c)) return zero;
    test = true;
    ro = lv.p;
    rd = toCam;
    rt = dist - 0.001f;
    rskip = lv.prim;
    sampled.p = lp;
    sampled.n = toCam;
    sampled.wi = dir;  // (scratch: the lens-to-vertex direction)
    sampled.beta = f3(cb, cb, cb);
    sampled.Le = zero;
    sampled.fwd = cpdf;
    sampled.rev = 0.f;
    sampled.mat = -1;
    sampled.light = -1;
    sampled.prim = kNoHit;
    sampled.flags = kFlagCamera;
    splat = true;
    Lc = c;
  } else {
    // evaluateDirectLightingStrategy (bdpt.go:334-394)
    BVert cv = C[t - 1];
    if (cv.is(kFlagSpecular) || cv.mat < 0) return zero;
    if (sc.n_lights == 0) return zero;
    int li = pick_light(sc, rs.next());
    DevLight L = sc.lights[li];
    LightSample ls = light_sample(sc, L, cv.p, cv.n, rs.next2());
    ls.pdf *= L.prob;
    if (is_zero(ls.emission) || ls.pdf <= 0.f) return zero;
    float ct = fabsf(dot_yx(ls.dir, cv.n));
    if (ct <= 0.f) return zero;
    float3 f = vertex_brdf(sc, cv, ls.dir, true);
    float3 lb = ls.emission * (1.f / ls.pdf);
    float3 c = f * cv.beta * lb * ct;
    if (is_zero(c)) return zero;
    test = true;
    ro = cv.p;
    rd = ls.dir;
    rt = ls.dist - 0.001f;
    rskip = cv.prim;
    sampled.p = ls.point;
    sampled.n = ls.normal;
    sampled.wi = zero;
    sampled.light = li;
    sampled.mat = -1;
    sampled.prim = kNoHit;
    sampled.fwd = ls.pdf;
    sampled.rev = 0.f;
    bool inf = L.kind == kLightUniformInfinite || L.kind == kLightGradientInfinite;
    sampled.flags = kFlagLight | (inf ? kFlagInfinite : 0);
    sampled.beta = lb;
    sampled.Le = ls.emission;
    Lc = c;
  }
  if (test && occluded<kOneNode>(sc, geo, ro, rd, rt, rskip, err)) return zero;
  if (splat) {
    // MapRayToPixel, then the light pdf of the camera vertex (bdpt.go:440-470)
    float3 dir = sampled.wi;
    sampled.wi = zero;
    if (!map_ray_to_pixel(sc.cam, sampled.p, dir, spx, spy)) return zero;
    sampled.rev = total_light_pdf(sc, sampled.p, sampled.n, normalize(Lp[s - 1].p - sampled.p));
  }
  if (is_zero(Lc) && !splat) return zero;
  const float w = mis_weight<CLS>(sc, C, Lp, CLS == 1 ? Lp[s - 1] : C[t - 1], sampled, s, t);
  if (splat) {
    float3 c = Lc * w;
    float4* dst = film.splat + (size_t)spy * film.width + spx;
    atomicAdd(&dst->x, c.x);
    atomicAdd(&dst->y, c.y);
    atomicAdd(&dst->z, c.z);
    return zero;
  }
  return Lc * w;
}

// Samples of a chunk per SM at most whose subpaths run in one launch and whose
// strategies share one: above it the wavefront is as fast (1 sample per pixel,
// depth 8, wavefront / one launch each in us: Cornell boxes 564 / 414 at
// 65,536 samples, 868 / 819 at 147,456, 1321 / 1423 at 262,144; spot scene
// 633 / 515 at 210,432, 866 / 839 at 374,272; sphere scene 500 / 334 at
// 147,456, 992 / 916 at 589,824; 20,480 triangles 1030 / 817 at 147,456,
// 1282 / 1293 at 262,144).
constexpr uint32_t kSmallBdptPerSm = 1024;
constexpr int kSubpathsBlock = 512, kSubpathsBlocksPerSm = 1;

// A subpath between bounces (one slot of BdQueue).
struct BdState {
  float4 o, d, beta, last;
  uint4 ids;
  uint2 st;
};

// generateCameraPath (bdpt.go:106-135): the camera vertex and ray of sample p
// of the chunk.
__device__ __forceinline__ BdState camera_start(const DevScene& sc, const DevFilm& film, const DevBdpt& B,
                                                const ChunkDesc& ch, uint32_t p) {
  uint32_t layer = p / ch.npix, i = p - layer * ch.npix;
  uint32_t pix = ch.pix_list ? ch.pix_list[ch.pix0 + i] : ch.pix0 + i;
  uint32_t sample = film.count[pix] + layer;
  int x = (int)(pix % (uint32_t)film.width), y = (int)(pix / (uint32_t)film.width);
  Rng rng;
  rng.init(ch.seed, pix, sample);
  float2 lens = rng.next2();
  float2 jit = rng.next2();
  float3 o, d;
  camera_ray(sc.cam, x, y, lens, jit, o, d, false);
  BVert c;
  c.p = o;
  c.n = -d;
  c.wi = f3(0.f, 0.f, 0.f);
  c.beta = f3(1.f, 1.f, 1.f);
  c.Le = f3(0.f, 0.f, 0.f);
  c.uv = make_float2(0.f, 0.f);
  c.fwd = 0.f;
  c.rev = 0.f;
  c.mat = -1;
  c.light = -1;
  c.prim = kNoHit;
  c.flags = kFlagCamera;
  put_vert(B, 0, p, c);
  BdState S;
  S.o = make_float4(o.x, o.y, o.z, __uint_as_float(kNoHit));
  S.d = make_float4(d.x, d.y, d.z, camera_dir_pdf(sc.cam, o, d));
  S.beta = make_float4(1.f, 1.f, 1.f, 0.f);
  S.last = make_float4(c.n.x, c.n.y, c.n.z, 0.f);
  S.ids = make_uint4(p, rng.pos, pix, sample);
  S.st = make_uint2(1u | kStCamera | kStOkBefore | kStOkLast, 0u);
  return S;
}

__device__ __forceinline__ void put_state(const BdQueue& Q, uint32_t i, const BdState& S) {
  Q.o[i] = S.o;
  Q.d[i] = S.d;
  Q.beta[i] = S.beta;
  Q.last[i] = S.last;
  Q.ids[i] = S.ids;
  Q.st[i] = S.st;
}

// The camera vertex and ray of every sample of the chunk, queue 0 slot p =
// sample p.
template <int MAXV>
__global__ void k_bdpt_camgen(DevScene sc, DevFilm film, DevPaths PS, ChunkDesc ch) {
  const DevBdpt& B = PS.bd;
  const uint32_t n = ch.npix * ch.layers;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
    put_state(B.q[0], p, camera_start(sc, film, B, ch, p));
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    PS.counters[0] = n;
    PS.counters[1] = 0;
    PS.counters[4] = 0;
  }
}

// The rays of the subpath queue; the marker hit of a stack overflow sets the
// job's error bits and is stored as a miss.
struct BdptSource {
  const float4* o;
  const float4* d;
  float4* hit;
  const uint32_t* n;
  int root;
  int* err;
  __device__ uint32_t count() const { return *n; }
  __device__ void load(uint32_t i, float3& ro, float3& rd, float& tmin, float& tmax, uint32_t& skip, int& rt) const {
    float4 a = o[i], b = d[i];
    ro = f3(a);
    rd = f3(b);
    tmin = 0.001f;
    tmax = kInfF;
    skip = __float_as_uint(a.w);
    rt = root;
  }
  __device__ void store(uint32_t i, const Hit& h) const {
    bool any = h.prim != kNoHit;
    if (h.prim == kOverflowHit) {
      atomicOr(err, kErrStackOverflow);
      any = false;
    }
    hit[i] = make_float4(any ? h.t : -1.f, __uint_as_float(any ? h.prim : kNoHit), h.u, h.v);
  }
};

template <bool kOneNode>
__global__ void __launch_bounds__(128, kTravBlocks) 
    k_bdpt_trace(DevScene sc, BdptSource src, uint32_t* counters, int cur, const __grid_constant__ Geom<kOneNode> geo) {
  if (blockIdx.x == 0 && threadIdx.x == 0) counters[cur ^ 1] = 0;  // the next queue starts empty
  if constexpr (kOneNode) trace_batch_one_node<false, false>(geo, src, nullptr, nullptr);
  else trace_persistent<false, false>(sc, src, counters + 4, nullptr, nullptr);
}

// One bounce of extendPath (bdpt.go:206-291) for one subpath whose ray met h4:
// the vertex hit (or the camera subpath's background vertex,
// createBackgroundVertex bdpt.go:585-601), its scatter, the reverse pdf of
// the vertex before it.  Returns whether the sample goes on, with S its next
// ray: a camera subpath that ends starts the sample's light subpath
// (generateLightPath, bdpt.go:139-202); a light subpath that ends gets the
// infinite-light pdf fix-ups and completes its sample.
template <int MAXV>
__device__ __forceinline__ bool extend_subpath(const DevScene& sc, const DevBdpt& B, uint64_t seed, BdState& S, float4 h4) {
  const float4 o4 = S.o, d4 = S.d, b4 = S.beta, l4 = S.last;
  const uint4 ids = S.ids;
  const uint2 st2 = S.st;
  const uint32_t p = ids.x;
  Rng rng;
  rng.init(seed, ids.z, ids.w, ids.y);
  const uint32_t bits = st2.x;
  bool camera = bits & kStCamera;
  int len = (int)(bits & 31u), b = (int)(bits >> 5 & 31u);
  uint32_t light_mask = bits >> kStLightMask, cam_mask = st2.y >> kStCamMask;
  const int vb = camera ? 0 : MAXV;  // vertex base of the subpath
  const int max_bounces = camera ? sc.max_depth : sc.max_depth - 1;
  float3 o = f3(o4), d = f3(d4), beta = f3(b4);
  float pdf_fwd = d4.w, acc = b4.w;
  bool ok_before = bits & kStOkBefore, ok_last = bits & kStOkLast;
  bool surf_last = bits & kStSurfLast, inf_last = bits & kStInfLast;
  float3 last_n = f3(l4);
  float last_fwd = l4.w;
  bool ended = true;
  uint32_t prim = __float_as_uint(h4.y);
  float rev_last = 0.f;  // the reverse pdf of the last vertex (0 unless the new vertex scatters)
  BVert v;
  bool has_v = false, v_ok = false;
  if (prim == kNoHit) {
    if (camera) {  // createBackgroundVertex (bdpt.go:585-601)
      float3 bg = background(sc, d);
      v.p = o + d * 1000.f;
      v.n = -d;
      v.wi = -d;
      v.fwd = pdf_fwd;
      v.rev = 0.f;
      v.beta = beta;
      v.Le = bg;
      v.uv = make_float2(0.f, 0.f);
      v.mat = -1;
      v.light = -1;
      v.prim = kNoHit;
      v.flags = kFlagInfinite | (is_zero(bg) ? 0 : kFlagLight);
      has_v = true;
    }
  } else {
    Hit h{h4.x, prim, h4.z, h4.w};
    Surface s;
    surface_at(sc, o, d, h, s, false);
    DevMaterial m = load_material(sc, s.mat);
    v.p = s.p;
    v.n = s.n;
    v.wi = -d;
    v.beta = beta;
    v.Le = emitted(m, s.front, d);
    v.mat = s.mat;
    v.uv = s.uv;
    v.light = -1;
    v.prim = prim;
    v.flags = (s.front ? kFlagFront : 0) | (is_zero(v.Le) ? 0 : kFlagLight);
    v.rev = 0.f;
    v.fwd = to_area_at(o, v.p, v.n, v.mat >= 0, false, pdf_fwd);
    has_v = true;
    Scatter scn;
    if (scatter(sc, m, d, s, rng, scn)) {
      float npdf = scn.pdf;
      if (scn.pdf <= 0.f) v.flags |= kFlagSpecular;
      float ct = fabsf(dot_yx_z(scn.dir, s.n));
      float3 nbeta = scn.pdf <= 0.f ? beta * scn.att : beta * scn.att * (ct / scn.pdf);
      bool rdelta;
      float pdf_rev = mat_pdf(sc, m, scn.dir, -d, s.n, rdelta);
      if (rdelta) {
        v.flags |= kFlagSpecular;
        pdf_rev = 0.f;
        npdf = 0.f;
      }
      rev_last = to_area_at(v.p, o, last_n, surf_last, inf_last, pdf_rev);
      if (b + 1 < max_bounces && len + 1 < MAXV) {
        ended = false;
        S.o = make_float4(s.p.x, s.p.y, s.p.z, __uint_as_float(prim));
        S.d = make_float4(scn.dir.x, scn.dir.y, scn.dir.z, npdf);
        beta = nbeta;
      }
    }
  }
  // the last vertex is final now: its reverse pdf and MIS prefix
  const float q_last = prefix_q(len - 1, ok_last, ok_before, acc);
  const float pre_last = camera && len == 1 ? 0.f : (remap0(rev_last) / remap0(last_fwd)) * q_last;
  put_pdf(B, vb + len - 1, p, rev_last, q_last);
  if (has_v) {
    v_ok = vertex_ok(sc, v, camera);
    put_vert(B, vb + len, p, v);
    if (ended) put_pdf(B, vb + len, p, 0.f, prefix_q(len, v_ok, ok_last, pre_last));  // no bounce follows
    const bool specular = v.is(kFlagSpecular);
    if (camera) cam_mask |= !specular && v.mat >= 0 && sc.n_lights > 0 ? 1u << (len - 1) : 0u;
    else light_mask |= specular ? 0u : 1u << (len - 1);
    len++;
  }
  if (!ended) {
    S.beta = make_float4(beta.x, beta.y, beta.z, pre_last);
    S.last = make_float4(v.n.x, v.n.y, v.n.z, v.fwd);
    S.ids = make_uint4(p, rng.pos, ids.z, ids.w);
    S.st = make_uint2((uint32_t)len | ((uint32_t)(b + 1) << 5) | (camera ? kStCamera : 0u) |
                         (ok_last ? kStOkBefore : 0u) | (v_ok ? kStOkLast : 0u) | (v.mat >= 0 ? kStSurfLast : 0u) |
                         light_mask << kStLightMask,
                     (st2.y & 63u) | cam_mask << kStCamMask);
    return true;
  } else if (camera) {
    const int nc = len;
    if (sc.n_lights > 0) {
      // generateLightPath (bdpt.go:139-202), in the same sampler stream
      int li = pick_light(sc, rng.next());
      DevLight L = sc.lights[li];
      float2 sp = rng.next2();
      float2 sd = rng.next2();
      float3 ep, en, ed, Le;
      float apdf, dpdf;
      sample_emission(sc, L, sp, sd, ep, en, ed, Le, apdf, dpdf);
      float ct = fabsf(dot_yx(ed, en));
      BVert lv;
      lv.p = ep;
      lv.n = en;
      lv.wi = f3(0.f, 0.f, 0.f);
      lv.uv = make_float2(0.f, 0.f);
      lv.light = li;
      lv.mat = -1;
      lv.prim = L.kind == kLightQuad     ? sc.quad_base + (uint32_t)L.prim
                : L.kind == kLightSphere ? (L.prim >= 0 ? sc.sphere_base + (uint32_t)L.prim : kNoHit)
                : (L.kind == kLightDisc || L.kind == kLightDiscSpot) ? sc.quadric_base + (uint32_t)L.prim
                                                                     : kNoHit;
      lv.fwd = apdf * L.prob;
      lv.rev = 0.f;
      bool inf = L.kind == kLightUniformInfinite || L.kind == kLightGradientInfinite;
      lv.flags = kFlagLight | (inf ? kFlagInfinite : 0);
      lv.beta = Le;
      lv.Le = Le;
      bool lok = vertex_ok(sc, lv, false);
      bool lsurf = light_is_area(sc, li);
      if (inf) {
        B.lorig[3 * (size_t)p] = make_float4(ep.x, ep.y, ep.z, apdf);
        B.lorig[3 * (size_t)p + 1] = make_float4(en.x, en.y, en.z, L.prob);
        B.lorig[3 * (size_t)p + 2] = make_float4(ed.x, ed.y, ed.z, 0.f);
      }
      if (0 < sc.max_depth - 1 && 1 < MAXV) {
        put_vert(B, MAXV, p, lv);
        float3 lb = Le * (ct / (L.prob * apdf * dpdf));
        S.o = make_float4(ep.x, ep.y, ep.z, __uint_as_float(lv.prim));
        S.d = make_float4(ed.x, ed.y, ed.z, dpdf);
        S.beta = make_float4(lb.x, lb.y, lb.z, 0.f);
        S.last = make_float4(en.x, en.y, en.z, lv.fwd);
        S.ids = make_uint4(p, rng.pos, ids.z, ids.w);
        S.st = make_uint2(1u | kStOkBefore | (lok ? kStOkLast : 0u) | (lsurf ? kStSurfLast : 0u) |
                             (inf ? kStInfLast : 0u),
                         (uint32_t)nc | (inf ? kStInfinite : 0u) | cam_mask << kStCamMask);
        return true;
      } else {  // a light subpath of the light vertex alone
        if (inf) lv.fwd = infinite_density(sc, ep, en, ed);  // the fix-up of the light vertex (bdpt.go:188-199)
        put_vert(B, MAXV, p, lv);
        put_pdf(B, MAXV, p, 0.f, prefix_q(0, lok, true, 0.f));
        finish_sample(B, p, nc, 1, rng.pos, ids.z, ids.w, 0u, cam_mask);
      }
    } else {
      finish_sample(B, p, nc, 0, rng.pos, ids.z, ids.w, 0u, cam_mask);
    }
  } else {
    int nl = len;
    if (st2.y & kStInfinite) {
      // the infinite-light fix-ups of generateLightPath (bdpt.go:188-199)
      float4 e0 = B.lorig[3 * (size_t)p], e1 = B.lorig[3 * (size_t)p + 1], e2 = B.lorig[3 * (size_t)p + 2];
      float3 ep = f3(e0), en = f3(e1), ed = f3(e2);
      float apdf = e0.w, lprob = e1.w;
      if (nl > 1) {
        const size_t at = (size_t)(MAXV + 1) * B.ns + p;
        const float4 n4 = B.v[1][at];
        float fwd = apdf * lprob;
        if ((__float_as_int(B.v[0][at].w) & 0xFFFFFF) > 0) fwd *= fabsf(dot(ed, f3(n4)));  // a surface
        B.v[1][at].w = fwd;
      }
      B.v[1][(size_t)MAXV * B.ns + p].w = infinite_density(sc, ep, en, ed);
      light_prefix(sc, B, MAXV, nl, p);  // the corrected pdfs change every prefix
    }
    finish_sample(B, p, (int)(st2.y & 31u), nl, rng.pos, ids.z, ids.w, light_mask, cam_mask);
  }
  return false;
}

// extend_subpath for every subpath of queue `cur`; continuing ones move to
// queue cur ^ 1.
template <int MAXV>
__global__ void __launch_bounds__(128, 4) k_bdpt_extend(DevScene sc, DevPaths PS, ChunkDesc ch, int cur) {
  const DevBdpt& B = PS.bd;
  const BdQueue& Q = B.q[cur];
  const uint32_t n = PS.counters[cur];
  if (blockIdx.x == 0 && threadIdx.x == 0) PS.counters[4] = 0;  // the next traversal's ray fetch counter
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    uint32_t i = base + threadIdx.x;
    bool cont = false;
    BdState S;
    if (i < n) {
      S = BdState{Q.o[i], Q.d[i], Q.beta[i], Q.last[i], Q.ids[i], Q.st[i]};
      cont = extend_subpath<MAXV>(sc, B, ch.seed, S, B.hit[i]);
    }
    // continuing subpaths to consecutive slots of the next queue (one atomic per warp)
    uint32_t slot = warp_append(&PS.counters[cur ^ 1], cont);
    if (cont) put_state(B.q[cur ^ 1], slot, S);
  }
}

// Both subpaths of every sample in one launch, for small chunks: a lane takes
// a sample from its camera ray to the end of its light subpath, with the state
// between bounces in registers.  The wavefront's 2 x max_depth pairs of
// launches each take a ray's or a shading step's chain of latencies, 8 and 22
// us, on any number of samples (49,000 samples of the spot scene: 448 us a
// frame, 225 so).  What is left is bound by fetching instructions, so the
// warps of a block trace together and extend together and share them (two
// barriers a bounce; the same frame in blocks of 128 276 us, 256 255, 512 225).
// The vertices are those of the wavefront, bit for bit (the roundings on which
// the compiler's contraction differs between the two are spelled out).
template <int MAXV, bool kOneNode>
__global__ void __launch_bounds__(kSubpathsBlock, kSubpathsBlocksPerSm)
    k_bdpt_subpaths(DevScene sc, DevFilm film, DevPaths PS, ChunkDesc ch, const __grid_constant__ Geom<kOneNode> geo) {
  const DevBdpt& B = PS.bd;
  const uint32_t n = ch.npix * ch.layers;
  const int lane = threadIdx.x & 31;
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t chunk = min(32u, (n + nw - 1) / nw);
  int* err = reinterpret_cast<int*>(PS.counters + 3);
  uint64_t at = (uint64_t)w * chunk;
  uint32_t cur = (uint32_t)min((uint64_t)n, at), end = (uint32_t)min((uint64_t)n, at + chunk);
  bool more = cur < end, alive = false;
  BdState S;
  S.o = S.d = S.beta = S.last = make_float4(0.f, 0.f, 0.f, 0.f);
  S.ids = make_uint4(0, 0, 0, 0);
  S.st = make_uint2(0, 0);
  TravEntry stack[kOneNode ? 1 : kTraceStack];
  for (;;) {
    unsigned idle = __ballot_sync(0xffffffffu, !alive);
    if (more && idle) {
      if (cur == end) {
        at += (uint64_t)nw * chunk;
        cur = (uint32_t)min((uint64_t)n, at);
        end = (uint32_t)min((uint64_t)n, at + chunk);
      }
      if (cur == end) more = false;
      uint32_t take = min((uint32_t)__popc(idle), end - cur);
      uint32_t rank = (uint32_t)__popc(idle & ((1u << lane) - 1u));
      if (!alive && rank < take) {
        S = camera_start(sc, film, B, ch, cur + rank);
        alive = true;
      }
      cur += take;
      if (take) idle = 0;
    }
    if (!__syncthreads_or(idle != 0xffffffffu || more)) break;
    Hit hit{-1.f, kNoHit, 0.f, 0.f};
    if constexpr (kOneNode) {
      trace_one_node<false>(geo, alive, false, f3(S.o), f3(S.d), 0.001f, kInfF, __float_as_uint(S.o.w), hit);
    } else {
      Trav s;
      bool busy = alive;
      if (busy) trav_init(s, f3(S.o), f3(S.d), 0.001f, kInfF, __float_as_uint(S.o.w), sc.root, stack);
      for (;;) {
        const bool testing = busy && s.testing();
        const unsigned busy_mask = __ballot_sync(0xffffffffu, busy), test_mask = __ballot_sync(0xffffffffu, testing);
        if (!busy_mask) break;
        if (trav_test_now(test_mask, busy_mask)) {
          if (testing) trav_prim<false>(sc, s, false, stack, nullptr);
        } else if (busy && !testing && s.node >= 0) {
          trav_visit<false>(sc, s, stack, nullptr);
        }
        if (busy && s.done()) {
          if (s.hit == kOverflowHit) {
            atomicOr(err, kErrStackOverflow);
            s.hit = kNoHit;
          }
          hit = s.result();
          busy = false;
        }
      }
    }
    __syncthreads();
    if (alive)
      alive = extend_subpath<MAXV>(sc, B, ch.seed, S,
                                   make_float4(hit.t, __uint_as_float(hit.prim), hit.u, hit.v));
  }
}

// The strategies (s, t) of a sample with s light vertices (s <= nl), as bits t:
// strategy k = s * MAXV + (t - 1) is evaluated when s <= nl and t <= nc, except
// (1,1) (bdpt.go:300-301) and s = 0 with t != nc (the path-tracing strategy
// contributes only at the full camera path).  Of these, the ones left out here
// return zero before drawing any number, so that changes neither a sampler
// position (draws_before) nor a sum: light tracing with a specular light
// vertex (mask bit s clear), direct lighting at a specular or material-less
// camera vertex or without lights (bit t clear), and a connection with either
// (bdpt.go:398-561).
__device__ __forceinline__ uint32_t strategy_row(int s, int nc, uint2 m) {
  if (s == 0) return 1u << nc;
  if (s == 1) return m.y;
  return (m.x >> s) & 1u ? m.y | 2u : 0u;
}

// Lists, per strategy, the samples that have it, so that the strategy kernel
// gives each warp 32 real (s, t, sample) items.  A block of 1,024 samples
// counts each strategy's items in shared memory (one shared atomic per warp
// and row of strategies, lane t for strategy (s, t): 228 -> 137 us per 2^20
// samples against one per strategy, whose answer lane 0 waited for), reserves its range of every list with one global atomic per
// strategy, then writes the items: per-warp global atomics on the
// (MAXV + 1) x MAXV list counters serialised in L2 (16.7 ms of a 200 ms
// Cornell-boxes frame).  The order within a list does not matter: every
// item writes its own contribution slot.
template <int MAXV>
__global__ void __launch_bounds__(1024) k_bdpt_list(DevPaths PS, ChunkDesc ch) {
  constexpr int K = (MAXV + 1) * MAXV;
  __shared__ uint32_t cnt[K], base[K];
  __shared__ uint16_t wofs[32][K];  // each warp's offset within the block's range (< 1,024)
  const DevBdpt& B = PS.bd;
  const uint32_t n = ch.npix * ch.layers;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  for (uint32_t start = blockIdx.x * 1024u; start < n; start += gridDim.x * 1024u) {
    const uint32_t w = start / kBdWindow;  // the block's samples lie in one window
    for (int k = threadIdx.x; k < K; k += blockDim.x) cnt[k] = 0;
    __syncthreads();
    uint32_t i = start + threadIdx.x;
    int nc = 0, nl = -1;
    uint2 mk = make_uint2(0u, 0u);
    if (i < n) {
      uint32_t m = B.meta[i].x;
      nc = (int)(m & 0xFF);
      nl = (int)(m >> 8);
      mk = B.masks[i];
    }
    // a warp visits only the strategies that some lane of it has, the same in
    // both loops, so wofs is written and read for those only
    const int wnl = __reduce_max_sync(0xFFFFFFFFu, nl);
    for (int s = 0; s <= wnl; s++) {
      const uint32_t mine = s <= nl ? strategy_row(s, nc, mk) : 0u;
      const uint32_t all = __reduce_or_sync(0xFFFFFFFFu, mine);
      uint32_t c = 0;  // lane t: the row's count of strategy t
      for (uint32_t left = all; left; left &= left - 1u) {
        const int t = __ffs(left) - 1;
        const unsigned mask = __ballot_sync(0xFFFFFFFFu, (mine >> t) & 1u);
        if (lane == t) c = __popc(mask);
      }
      if (c) wofs[wp][s * MAXV + lane - 1] = (uint16_t)atomicAdd(&cnt[s * MAXV + lane - 1], c);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += blockDim.x)
      base[k] = cnt[k] ? w * kBdWindow + atomicAdd(B.scount + w * K + k, cnt[k]) : 0u;
    __syncthreads();
    for (int s = 0; s <= wnl; s++) {
      const uint32_t mine = s <= nl ? strategy_row(s, nc, mk) : 0u;
      const uint32_t all = __reduce_or_sync(0xFFFFFFFFu, mine);
      for (uint32_t left = all; left; left &= left - 1u) {
        const int t = __ffs(left) - 1, k = s * MAXV + t - 1;
        const bool has = (mine >> t) & 1u;
        const unsigned mask = __ballot_sync(0xFFFFFFFFu, has);
        if (has) B.slist[(size_t)k * B.ns + base[k] + wofs[wp][k] + __popc(mask & below)] = i;
      }
    }
    __syncthreads();  // cnt, base and wofs are rewritten for the next range
  }
}

// The strategy classes, each evaluated by its own launch so that a launch
// holds only its class's code: 0 the path-tracing strategy (s = 0, t = nc),
// 1 light tracing (s >= 2, t = 1), 2 direct lighting (s = 1, t >= 2),
// 3 connections (s, t >= 2).
__host__ __device__ constexpr int strategy_class(int s, int t) {
  return s == 0 ? 0 : t == 1 ? 1 : s == 1 ? 2 : 3;
}

// The per-class prefix sums of the list counts in (window, strategy) order,
// which map a strategy kernel's class-wide item index g to the entry
// e = w * K + k with sprefix[e] <= g < sprefix[e + 1].  One block: each
// thread sums a contiguous run of entries for the four classes, and a
// block-wide scan of the runs gives their offsets.
template <int MAXV>
__global__ void __launch_bounds__(1024) k_bdpt_prefix(DevPaths PS) {
  constexpr int K = (MAXV + 1) * MAXV;
  __shared__ uint32_t part[4][1024];
  const DevBdpt& B = PS.bd;
  const uint32_t E = B.nw * K;
  const uint32_t per = (E + 1023u) / 1024u;
  const uint32_t t = threadIdx.x;
  const uint32_t lo = min(E, t * per), hi = min(E, lo + per);
  uint32_t s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  for (uint32_t e = lo; e < hi; e++) {
    int k = (int)(e % K), c = strategy_class(k / MAXV, k % MAXV + 1);
    uint32_t v = B.scount[e];
    s0 += c == 0 ? v : 0u;
    s1 += c == 1 ? v : 0u;
    s2 += c == 2 ? v : 0u;
    s3 += c == 3 ? v : 0u;
  }
  part[0][t] = s0;
  part[1][t] = s1;
  part[2][t] = s2;
  part[3][t] = s3;
  __syncthreads();
  for (uint32_t d = 1; d < 1024u; d <<= 1) {  // inclusive scan (Hillis-Steele)
    uint32_t a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    if (t >= d) {
      a0 = part[0][t - d];
      a1 = part[1][t - d];
      a2 = part[2][t - d];
      a3 = part[3][t - d];
    }
    __syncthreads();
    part[0][t] += a0;
    part[1][t] += a1;
    part[2][t] += a2;
    part[3][t] += a3;
    __syncthreads();
  }
  uint32_t r0 = part[0][t] - s0, r1 = part[1][t] - s1, r2 = part[2][t] - s2, r3 = part[3][t] - s3;
  uint32_t* P = B.sprefix;
  for (uint32_t e = lo; e < hi; e++) {
    P[e] = r0;
    P[(E + 1) + e] = r1;
    P[2 * (E + 1) + e] = r2;
    P[3 * (E + 1) + e] = r3;
    int k = (int)(e % K), c = strategy_class(k / MAXV, k % MAXV + 1);
    uint32_t v = B.scount[e];
    r0 += c == 0 ? v : 0u;
    r1 += c == 1 ? v : 0u;
    r2 += c == 2 ? v : 0u;
    r3 += c == 3 ? v : 0u;
  }
  if (t == 1023u) {
    P[E] = part[0][t];
    P[(E + 1) + E] = part[1][t];
    P[2 * (E + 1) + E] = part[2][t];
    P[3 * (E + 1) + E] = part[3][t];
  }
}

// The entry e = w * K + k of item g of class-prefix P (E entries, P[e] <= g <
// P[e + 1]) for the warp's 32 consecutive items from `base`: 32 probes a
// round for the first item's, and a search of their own for the lanes whose
// items lie past its end.  (A binary search per lane took 13 dependent loads.)
__device__ __forceinline__ uint32_t item_entry(const uint32_t* P, uint32_t E, uint32_t base, uint32_t g, int lane) {
  uint32_t lo = 0, len = E;
  while (len > 1) {
    const uint32_t step = (len + 31) >> 5, at = lane * step;
    const bool le = at < len && __ldg(P + lo + at) <= base;
    const uint32_t c = (uint32_t)__popc(__ballot_sync(0xffffffffu, le)) - 1u;  // P[lo] <= base
    lo += c * step;
    len = min(step, len - c * step);
  }
  if (__ldg(P + lo + 1) > g) return lo;
  uint32_t hi = E;
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (__ldg(P + mid) <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

// One thread per listed (strategy, sample) item of class CLS, in (window,
// strategy) order: a warp evaluates one (s, t) for 32 samples of one window
// that have it (uniform control flow, neighbouring warps on the same code),
// and every strategy of a window of samples runs before the next window, so
// the vertex reads of the window's later strategies hit L2.  The work is
// latency-bound: 8 blocks per SM and at most 64 registers, a few spilled.
// Whole warps run it, for classes 0, 1 and 2.
template <int MAXV, int CLS, bool kOneNode>
__device__ __forceinline__ void run_strategies(const DevScene& sc, const DevFilm& film, const DevPaths& PS,
                                               const ChunkDesc& ch, const Geom<kOneNode>& geo) {
  constexpr int K = (MAXV + 1) * MAXV;
  const DevBdpt& B = PS.bd;
  const uint32_t n = ch.npix * ch.layers;
  const uint32_t E = B.nw * K;
  const uint32_t* P = B.sprefix + (size_t)CLS * (E + 1);
  const uint32_t total = __ldg(P + E);
  const int lane = threadIdx.x & 31;
  int* err = reinterpret_cast<int*>(PS.counters + 3);
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total; base += gridDim.x * blockDim.x) {
    const uint32_t g = min(base + lane, total - 1);
    const uint32_t lo = item_entry(P, E, base, g, lane);
    if (base + lane < total) {
      const uint32_t w = lo / K;
      const int k = (int)(lo - w * K);
      const uint32_t i = B.slist[(size_t)k * B.ns + w * kBdWindow + (g - __ldg(P + lo))];
      const int s = k / MAXV, t = k % MAXV + 1;
      uint4 m = B.meta[i];
      Rng rs;
      rs.init(ch.seed, m.z, m.w, m.y + draws_before(s, t, B.masks[i]));
      float3 c = eval_strategy<CLS, kOneNode>(sc, geo, film, B, i, s, t, rs, err);
      B.contrib[(size_t)k * n + i] = make_float4(c.x, c.y, c.z, 0.f);
    }
    __syncwarp();
  }
}

// The segment that joins light vertex pl to camera vertex pc.
struct Connection {
  float3 d;  // from pc to pl, unit length
  float dist;
};
__device__ __forceinline__ Connection connect(float3 pl, float3 pc) {
  Connection c;
  c.d = pl - pc;
  c.dist = sqrtf(dot_xy(c.d, c.d));
  c.d = c.d * (1.f / c.dist);
  return c;
}

// The connection strategy (evaluateConnectionStrategy, bdpt.go:502-561) of
// light vertex s - 1 and camera vertex t - 1 of sample i, neither of them
// specular, in three steps.  First: whether the vertices face each other.
__device__ __forceinline__ bool connection_faces(const DevBdpt& B, uint32_t i, int s, int t) {
  const size_t kl = (size_t)(B.maxv + s - 1) * B.ns + i, kc = (size_t)(t - 1) * B.ns + i;
  const float3 nl = f3(B.v[1][kl]), nc = f3(B.v[1][kc]);
  const Connection c = connect(f3(B.v[0][kl]), f3(B.v[0][kc]));
  return !(c.dist < 0.001f) && !(dot_xy(c.d, nc) <= 0.f) && !(dot_yx(-c.d, nl) <= 0.f);
}

// Second: whether they see each other.
template <bool kOneNode>
__device__ __forceinline__ bool connection_visible(const DevScene& sc, const Geom<kOneNode>& geo, const DevBdpt& B,
                                                   uint32_t i, int s, int t, int* err) {
  const size_t kl = (size_t)(B.maxv + s - 1) * B.ns + i, kc = (size_t)(t - 1) * B.ns + i;
  const float3 pc = f3(B.v[0][kc]);
  const Connection c = connect(f3(B.v[0][kl]), pc);
  return !occluded<kOneNode>(sc, geo, pc, c.d, c.dist - 0.001f, __float_as_uint(B.v[3][kc].z), err);
}

// Third: the weighted contribution.  The four reverse pdfs of the MIS weight
// (bdpt_mis.go:61-105, 140-178) are two at each end: from the own subpath
// towards the other end's vertex, and back.
__device__ __forceinline__ float3 connection_value(const DevScene& sc, const DevBdpt& B, uint32_t i, int s, int t) {
  const SubpathRef C{&B, i, 0}, Lp{&B, i, B.maxv};
  float3 bl = f3(0.f, 0.f, 0.f), bc = bl, wl = bl, wc = bl;  // BRDFs and throughputs at the two ends
  float cc = 0.f, cl = 0.f, dist = 0.f;
  float cam1 = 0.f, cam2 = 0.f, lit1 = 0.f, lit2 = 0.f;
#pragma unroll 1
  for (int q = 0; q < 2; q++) {  // the light end, the camera end
    const int kx = q ? t - 1 : B.maxv + s - 1, ko = q ? B.maxv + s - 1 : t - 1;
    const BVert x = get_vert(B, kx, i), o = get_vert(B, ko, i), own = get_vert(B, kx - 1, i);
    const Connection c = connect(q ? o.p : x.p, q ? x.p : o.p);
    const float3 f = vertex_brdf(sc, x, q ? c.d : -c.d, q == 1);
    float to_o, to_own;
    end_pdfs(sc, x, o, own, to_o, to_own);
    dist = c.dist;
    if (q) {
      bc = f;
      wc = x.beta;
      cc = dot_xy(c.d, x.n);
      lit1 = to_o;
      cam2 = to_own;
    } else {
      bl = f;
      wl = x.beta;
      cl = dot_yx(-c.d, x.n);
      cam1 = to_o;
      lit2 = to_own;
    }
  }
  const float g = (cc * cl) / (dist * dist);
  const float3 v = wl * bl * bc * wc * g;
  if (is_zero(v)) return v;
  return v * mis_walk<3>(C, Lp, 0.f, s, t, cam1, cam2, lit1, lit2);
}

// The connections, by whole warps.  Of the pairs 74 % face each other and
// 54 % see each other (Cornell boxes): the items that pass a step are
// collected per warp until 32 of them take the next, so that every step runs
// on full warps (25 of 32 lanes active instead of 19; 28.7 -> 24.5 ms of the
// Cornell-boxes frame of 512 x 512 x 64 samples when it came in).  Then bound
// by the latency of the vertex reads: 6 blocks per SM and 80 registers are
// faster than 4 or 8 (70.5 ms the whole frame, 71.8 and 72.7), and a grid that
// is resident at once than two waves of it, which read each window of vertices
// twice (3 ms of the frame).
constexpr int kConnectBlocks = 6;
template <int MAXV, bool kOneNode>
__device__ __forceinline__ void run_connections(const DevScene& sc, const DevPaths& PS, const ChunkDesc& ch,
                                                const Geom<kOneNode>& geo) {
  constexpr int K = (MAXV + 1) * MAXV;
  __shared__ uint2 facing[4][64], seen[4][64];  // {sample, strategy}; fewer than 32 are left before 32 are added
  const DevBdpt& B = PS.bd;
  const uint32_t n = ch.npix * ch.layers;
  const uint32_t E = B.nw * K;
  const uint32_t* P = B.sprefix + (size_t)3 * (E + 1);
  const uint32_t total = __ldg(P + E);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  int* err = reinterpret_cast<int*>(PS.counters + 3);
  uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
  int nf = 0, ns = 0;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  for (;;) {
    const bool more = base < total;
    if (ns >= 32 || (ns > 0 && !more && nf == 0)) {
      const int take = min(ns, 32);
      ns -= take;
      if (lane < take) {
        const uint2 it = seen[wp][ns + lane];
        const int s = (int)it.y / MAXV, t = (int)it.y % MAXV + 1;
        const float3 c = connection_value(sc, B, it.x, s, t);
        B.contrib[(size_t)it.y * n + it.x] = make_float4(c.x, c.y, c.z, 0.f);
      }
      __syncwarp();
    } else if (nf >= 32 || (nf > 0 && !more)) {
      const int take = min(nf, 32);
      nf -= take;
      bool pass = false;
      uint2 it = make_uint2(0u, 0u);
      if (lane < take) {
        it = facing[wp][nf + lane];
        pass = connection_visible<kOneNode>(sc, geo, B, it.x, (int)it.y / MAXV, (int)it.y % MAXV + 1, err);
        if (!pass) B.contrib[(size_t)it.y * n + it.x] = zero;
      }
      const unsigned m = __ballot_sync(0xffffffffu, pass);
      if (pass) seen[wp][ns + __popc(m & below)] = it;
      ns += __popc(m);
      __syncwarp();
    } else if (more) {
      const uint32_t g = min(base + lane, total - 1);
      const uint32_t lo = item_entry(P, E, base, g, lane);
      const uint32_t w = lo / K;
      uint2 it = make_uint2(0u, lo - w * K);
      bool pass = false;
      if (base + lane < total) {
        it.x = B.slist[(size_t)it.y * B.ns + w * kBdWindow + (g - __ldg(P + lo))];
        pass = connection_faces(B, it.x, (int)it.y / MAXV, (int)it.y % MAXV + 1);
        if (!pass) B.contrib[(size_t)it.y * n + it.x] = zero;
      }
      const unsigned m = __ballot_sync(0xffffffffu, pass);
      if (pass) facing[wp][nf + __popc(m & below)] = it;
      nf += __popc(m);
      base += gridDim.x * blockDim.x;
      __syncwarp();
    } else {
      break;
    }
  }
}

template <int MAXV, int CLS, bool kOneNode>
__global__ void __launch_bounds__(128, CLS == 3 ? kConnectBlocks : 8)
    k_bdpt_strategies(DevScene sc, DevFilm film, DevPaths PS, ChunkDesc ch, const __grid_constant__ Geom<kOneNode> geo) {
  if constexpr (CLS == 3) run_connections<MAXV, kOneNode>(sc, PS, ch, geo);
  else run_strategies<MAXV, CLS, kOneNode>(sc, film, PS, ch, geo);
}

// The four classes in one launch (blockIdx.y), for small chunks, whose launches
// each take the time of one item (22-25 us; together 28).
template <int MAXV, bool kOneNode>
__global__ void __launch_bounds__(128, 8)
    k_bdpt_strategies_all(DevScene sc, DevFilm film, DevPaths PS, ChunkDesc ch,
                          const __grid_constant__ Geom<kOneNode> geo) {
  switch (blockIdx.y) {
    case 0: run_connections<MAXV, kOneNode>(sc, PS, ch, geo); break;
    case 1: run_strategies<MAXV, 1, kOneNode>(sc, film, PS, ch, geo); break;
    case 2: run_strategies<MAXV, 2, kOneNode>(sc, film, PS, ch, geo); break;
    default: run_strategies<MAXV, 0, kOneNode>(sc, film, PS, ch, geo); break;
  }
}

template <int MAXV>
__global__ void k_bdpt_sum(DevPaths PS, ChunkDesc ch) {
  const DevBdpt& B = PS.bd;
  uint32_t n = ch.npix * ch.layers;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint4 m = B.meta[i];
    const uint2 mk = B.masks[i];
    int nc = (int)(m.x & 0xFF), nl = (int)(m.x >> 8);
    float3 total = f3(0.f, 0.f, 0.f);
    for (int s = 0; s <= nl; s++) {
      const uint32_t row = strategy_row(s, nc, mk);  // the others contribute nothing: not evaluated
      for (int t0 = 1; t0 <= nc; t0 += 4) {
        // four reads on their way at once, each of one strategy (the warp's are
        // neighbours), added in the reference's order
        float4 c[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (row >> (t0 + k) & 1u) c[k] = B.contrib[(size_t)(s * MAXV + t0 + k - 1) * n + i];
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (row >> (t0 + k) & 1u) total += f3(c[k]);
      }
    }
    PS.Lout[i] = make_float4(total.x, total.y, total.z, 0.f);
  }
}

template <int MAXV, bool kOneNode>
void launch_bdpt_maxv(const DevScene& sc, const DevFilm& film, const DevPaths& P, const ChunkDesc& ch, int sms,
                      cudaStream_t st) {
  Geom<kOneNode> geo{};
  if constexpr (kOneNode) geo = *sc.one;
  const uint32_t n = ch.npix * ch.layers;
  const int gs = launch_grid(n, 128, std::max(1, sms * 8));  // grid-stride kernels over the queue
  const int gt = std::max(1, sms * kTravBlocks);                       // persistent traversal
  const int g2 = std::max(1, sms * 16);
  const int g3 = launch_grid(n, 256, 0);
  const int gl = std::min(launch_grid(n, 1024, 0), std::max(1, sms * 2));
  const bool small = n <= (uint32_t)sms * kSmallBdptPerSm;
  if (small) {
    k_bdpt_subpaths<MAXV, kOneNode><<<sms * kSubpathsBlocksPerSm, kSubpathsBlock, 0, st>>>(sc, film, P, ch, geo);
  } else {
    k_bdpt_camgen<MAXV><<<g3, 256, 0, st>>>(sc, film, P, ch);
    int cur = 0;
    // at most max_depth camera bounces, then max_depth - 1 light bounces
    for (int it = 0; it < 2 * sc.max_depth; it++) {
      BdptSource src{P.bd.q[cur].o, P.bd.q[cur].d, P.bd.hit, P.counters + cur, sc.root,
                     reinterpret_cast<int*>(P.counters + 3)};
      k_bdpt_trace<kOneNode><<<gt, 128, 0, st>>>(sc, src, P.counters, cur, geo);
      k_bdpt_extend<MAXV><<<gs, 128, 0, st>>>(sc, P, ch, cur);
      cur ^= 1;
    }
  }
  k_bdpt_list<MAXV><<<gl, 1024, 0, st>>>(P, ch);
  k_bdpt_prefix<MAXV><<<1, 1024, 0, st>>>(P);
  if (small) {
    k_bdpt_strategies_all<MAXV, kOneNode><<<dim3(sms * 4, 4), 128, 0, st>>>(sc, film, P, ch, geo);
  } else {
    k_bdpt_strategies<MAXV, 0, false><<<g2, 128, 0, st>>>(sc, film, P, ch, NoGeom{});
    k_bdpt_strategies<MAXV, 1, kOneNode><<<g2, 128, 0, st>>>(sc, film, P, ch, geo);
    k_bdpt_strategies<MAXV, 2, kOneNode><<<g2, 128, 0, st>>>(sc, film, P, ch, geo);
    k_bdpt_strategies<MAXV, 3, kOneNode><<<sms * kConnectBlocks, 128, 0, st>>>(sc, film, P, ch, geo);
  }
  k_bdpt_sum<MAXV><<<g3, 256, 0, st>>>(P, ch);
}

}  // namespace

// Subpaths as a wavefront (camera rays, then per bounce: traversal and
// extension over the compacted queue), per-strategy lists, one launch per
// strategy class, the per-sample sums.
void launch_bdpt(const DevScene& sc, const DevFilm& film, const DevPaths& P, const ChunkDesc& ch, int block,
                 cudaStream_t st) {
  (void)block;
  if (sc.max_depth <= 0) {
    // No ray leaves the camera: the one strategy with a camera subpath of its
    // single vertex sees no emission.  The kernels below take at least one
    // bounce to have written each sample's record (meta, masks).
    cudaMemsetAsync(P.Lout, 0, (size_t)ch.npix * ch.layers * sizeof(float4), st);
    return;
  }
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaMemsetAsync(P.bd.scount, 0, sizeof(uint32_t) * P.bd.nw * (P.bd.maxv + 1) * P.bd.maxv, st);
  const bool one = one_node(sc);
  auto launch = P.bd.maxv == 10 ? (one ? launch_bdpt_maxv<10, true> : launch_bdpt_maxv<10, false>)
                                : (one ? launch_bdpt_maxv<18, true> : launch_bdpt_maxv<18, false>);
  launch(sc, film, P, ch, sms, st);
}

}  // namespace gprt
