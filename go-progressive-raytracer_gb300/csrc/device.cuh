// device.cuh - device-side core of the GB300 rendering path: FP32 vector
// math, the counter-based sampler, primitive intersection, 4-wide BVH
// traversal, materials, lights and the camera.  Each routine restates the
// reference function cited beside it (paths relative to the reference
// project root) in FP32.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "deal.h"
#include "layout.h"

namespace gprt {

// ----------------------------------------------------------------- float3
__device__ __forceinline__ float3 f3(float a, float b, float c) { return make_float3(a, b, c); }
__device__ __forceinline__ float3 f3(float4 v) { return make_float3(v.x, v.y, v.z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator-(float3 a) { return f3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 operator*(float s, float3 a) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 operator*(float3 a, float3 b) { return f3(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ float3& operator+=(float3& a, float3 b) { a = a + b; return a; }
__device__ __forceinline__ float3& operator*=(float3& a, float3 b) { a = a * b; return a; }
__device__ __forceinline__ float3& operator*=(float3& a, float s) { a = a * s; return a; }
__device__ __forceinline__ float dot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// The path tracer and BDPT each have their shading in two kernels (the
// wavefront's and the one that takes small chunks whole), which have to render
// the same films.  The compiler contracts products and sums into multiply-adds
// kernel by kernel, and in most places alike; where the two did not agree the
// order is spelled out, as the wavefront's kernel of that integrator rounds:
// _xy rounds y y first, _yx x x (dot_yx_z also z z).  That the rest agrees is a
// property of the build, held by the tests that compare the films bit for bit.
__device__ __forceinline__ float dot_xy(float3 a, float3 b) {
  return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
}
__device__ __forceinline__ float dot_yx_z(float3 a, float3 b) {  // z z rounded as well
  return __fadd_rn(__fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ float dot_yx(float3 a, float3 b) {
  return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)));
}
__device__ __forceinline__ float3 cross(float3 a, float3 b) {
  return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float length(float3 a) { return sqrtf(dot(a, a)); }
// core.Vec3.Normalize (pkg/core/vec3.go:97-103): zero stays zero
__device__ __forceinline__ float3 normalize(float3 a) {
  float l = length(a);
  return l == 0.f ? f3(0.f, 0.f, 0.f) : f3(a.x / l, a.y / l, a.z / l);
}
// normalize with the rounding of the squared length spelled out, as dot_xy.
__device__ __forceinline__ float3 normalize_by(float3 a, float l2) {
  float l = sqrtf(l2);
  return l == 0.f ? f3(0.f, 0.f, 0.f) : f3(a.x / l, a.y / l, a.z / l);
}
__device__ __forceinline__ float3 normalize_xy(float3 a) {
  return normalize_by(a, __fmaf_rn(a.z, a.z, __fmaf_rn(a.x, a.x, __fmul_rn(a.y, a.y))));
}
__device__ __forceinline__ float3 normalize_yx(float3 a) {
  return normalize_by(a, __fmaf_rn(a.z, a.z, __fmaf_rn(a.y, a.y, __fmul_rn(a.x, a.x))));
}
// core.Vec3.Luminance (pkg/core/vec3.go:134-136)
__device__ __forceinline__ float luminance(float3 c) { return 0.2126f * c.x + 0.7152f * c.y + 0.0722f * c.z; }
// with its roundings spelled out (as dot_xy)
__device__ __forceinline__ float luminance_xy(float3 c) {
  return __fmaf_rn(0.0722f, c.z, __fmaf_rn(0.2126f, c.x, __fmul_rn(0.7152f, c.y)));
}
__device__ __forceinline__ bool is_zero(float3 c) { return c.x == 0.f && c.y == 0.f && c.z == 0.f; }

constexpr float kPi = 3.14159265358979323846f;
#define kInfF (__int_as_float(0x7f800000))

// 32-byte records (32-byte aligned) in one 256-bit access
__device__ __forceinline__ void load32(const float4* p, float4& a, float4& b) {
  asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p)
      : "memory");
}
__device__ __forceinline__ void store32(float4* p, float4 a, float4 b) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
               "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}
__device__ __forceinline__ float4 as_float4(uint4 v) {
  return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ uint4 as_uint4(float4 v) {
  return make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
}

// ----------------------------------------------------------------- sampler
// Counter-based sampler: every value is a pure function of (job seed, pixel,
// sample index, dimension), so a sample renders identically alone, batched
// with other jobs, or split across chunks.  The hash is the "pcg4d" mix of
// Jarzynski & Olano, "Hash Functions for GPU Rendering", JCGT 9(3), 2020.
// It replaces the per-tile math/rand stream of pkg/renderer/progressive.go:444.
__device__ __forceinline__ uint4 pcg4d(uint4 v) {
  v.x = v.x * 1664525u + 1013904223u;
  v.y = v.y * 1664525u + 1013904223u;
  v.z = v.z * 1664525u + 1013904223u;
  v.w = v.w * 1664525u + 1013904223u;
  v.x += v.y * v.w;
  v.y += v.z * v.x;
  v.z += v.x * v.y;
  v.w += v.y * v.z;
  v.x ^= v.x >> 16;
  v.y ^= v.y >> 16;
  v.z ^= v.z >> 16;
  v.w ^= v.w >> 16;
  v.x += v.y * v.w;
  v.y += v.z * v.x;
  v.z += v.x * v.y;
  v.w += v.y * v.z;
  return v;
}
__device__ __forceinline__ float u01(uint32_t x) { return (float)(x >> 8) * (1.0f / 16777216.0f); }

// 32-bit finalizer of MurmurHash3 (fmix32, Austin Appleby): every input bit
// affects every output bit.
__host__ __device__ __forceinline__ uint32_t fmix32(uint32_t h) {
  h ^= h >> 16;
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  h ^= h >> 16;
  return h;
}

// The fourth pcg4d coordinate of a 64-bit job seed.  The seed is a
// coordinate of its own, hashed first: keying it into the pixel (pixel ^
// seed) would give seed s the streams seed 0 gives pixel ^ s, so renders with
// nearby seeds would reuse each other's random numbers on shuffled pixels.
__host__ __device__ __forceinline__ uint32_t seed_word(uint64_t seed) {
  return fmix32((uint32_t)seed ^ fmix32((uint32_t)(seed >> 32) ^ 0x9e3779b9u));
}

// The uniform numbers of one pixel sample, consumed sequentially in the
// reference's draw order (RandomSampler, pkg/core/sampling.go:17-39): draw k
// is word k % 4 of pcg4d(pixel, sample, k / 4, seed_word(seed)).  `pos`
// (draws consumed) is all the state a wavefront path carries between
// kernels.
struct Rng {
  uint32_t k0, k1, k3, pos;
  bool valid;
  uint4 buf;
  __device__ __forceinline__ void init(uint64_t seed, uint32_t pixel, uint32_t sample, uint32_t start = 0) {
    k0 = pixel;
    k1 = sample;
    k3 = seed_word(seed);
    pos = start;
    valid = false;
  }
  __device__ __forceinline__ float next() {
    uint32_t lane = pos & 3u;
    if (lane == 0 || !valid) {
      buf = pcg4d(make_uint4(k0, k1, pos >> 2, k3));
      valid = true;
    }
    uint32_t r = lane == 0 ? buf.x : lane == 1 ? buf.y : lane == 2 ? buf.z : buf.w;
    pos++;
    return u01(r);
  }
  __device__ __forceinline__ float2 next2() {
    float a = next();
    float b = next();
    return make_float2(a, b);
  }
};

// ----------------------------------------------------------------- warps
// SampleCosineHemisphere (pkg/core/sampling.go:42-67)
__device__ __forceinline__ float3 sample_cosine_hemisphere(float3 n, float2 s) {
  float sa, ca;
  sincosf(2.0f * kPi * s.x, &sa, &ca);
  float r = sqrtf(s.y);
  float x = r * ca, y = r * sa, z = sqrtf(1.0f - s.y);
  float3 nt = fabsf(n.x) > 0.1f ? f3(0.f, 1.f, 0.f) : f3(1.f, 0.f, 0.f);
  float3 t = normalize(cross(nt, n));
  float3 b = cross(n, t);
  return t * x + b * y + n * z;
}
// SampleCone (sampling.go:70-94): uniform direction within the cone of
// cosine cos_total about the unit direction w
__device__ __forceinline__ float3 sample_cone(float3 w, float cos_total, float2 s) {
  float3 u = fabsf(w.x) > 0.1f ? f3(0.f, 1.f, 0.f) : f3(1.f, 0.f, 0.f);
  u = normalize(cross(u, w));
  float3 v = cross(w, u);
  float ct = 1.0f - s.x * (1.0f - cos_total);
  float st = sqrtf(fmaxf(0.f, 1.0f - ct * ct));
  float sp, cp;
  sincosf(2.0f * kPi * s.y, &sp, &cp);
  return u * (st * cp) + v * (st * sp) + w * ct;
}
// SampleOnUnitSphere (sampling.go:97-104)
__device__ __forceinline__ float3 sample_on_unit_sphere(float2 s) {
  float z = 1.0f - 2.0f * s.x;
  float r = sqrtf(fmaxf(0.f, 1.0f - z * z));
  float sp, cp;
  sincosf(2.0f * kPi * s.y, &sp, &cp);
  return f3(r * cp, r * sp, z);
}
// SamplePointInUnitDisk, concentric (sampling.go:108-126)
__device__ __forceinline__ float2 sample_unit_disk(float2 s) {
  float ux = 2.f * s.x - 1.f, uy = 2.f * s.y - 1.f;
  if (ux == 0.f && uy == 0.f) return make_float2(0.f, 0.f);
  float theta, r;
  if (fabsf(ux) > fabsf(uy)) {
    r = ux;
    theta = kPi / 4.f * (uy / ux);
  } else {
    r = uy;
    theta = kPi / 2.f - kPi / 4.f * (ux / uy);
  }
  float st, ct;
  sincosf(theta, &st, &ct);
  return make_float2(r * ct, r * st);
}
// SamplePointInUnitSphere (sampling.go:130-147); pow(x, 1/3) == cbrt(x)
__device__ __forceinline__ float3 sample_in_unit_sphere(float3 s) {
  float r = cbrtf(s.x);
  float sp, cp;
  sincosf(2.f * kPi * s.y, &sp, &cp);
  float ct = 2.f * s.z - 1.f;
  float st = sqrtf(fmaxf(0.f, 1.f - ct * ct));
  return f3(r * st * cp, r * st * sp, r * ct);
}

// ----------------------------------------------------------------- hit record
struct Hit {
  float t;
  uint32_t prim;  // global primitive id or kNoHit
  float u, v;
};

// The primitive tests below spell out every rounding (explicit fma / mul /
// add / div intrinsics): kernels that inline them in different contexts -- the
// traversal variants, the single-job and the batched wavefronts -- then
// return bit-identical hits.
__device__ __forceinline__ float dot_rn(float3 a, float3 b) {
  return __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, __fmul_rn(a.z, b.z)));
}
__device__ __forceinline__ float3 cross_rn(float3 a, float3 b) {
  return make_float3(__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)),
                     __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float3 sub_rn(float3 a, float3 b) {
  return make_float3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}

// ----------------------------------------------------------------- primitives
// Triangle.Hit, Moller-Trumbore, epsilon 1e-8 (pkg/geometry/triangle.go:107-175)
// Triangles are stored as (v0, e1 = v1 - v0, e2 = v2 - v0).
__device__ __forceinline__ bool hit_triangle(float3 o, float3 d, float4 a, float4 b, float4 c, float tmin,
                                             float tmax, float& t, float& uu, float& vv) {
  float3 v0 = f3(a), e1 = f3(b), e2 = f3(c);
  float3 h = cross_rn(d, e2);
  float det = dot_rn(e1, h);
  if (det > -1e-8f && det < 1e-8f) return false;
  float f = __frcp_rn(det);
  float3 s = sub_rn(o, v0);
  float u = __fmul_rn(f, dot_rn(s, h));
  if (u < 0.f || u > 1.f) return false;
  float3 q = cross_rn(s, e1);
  float v = __fmul_rn(f, dot_rn(d, q));
  if (v < 0.f || __fadd_rn(u, v) > 1.f) return false;
  float tt = __fmul_rn(f, dot_rn(e2, q));
  if (tt < tmin || tt > tmax) return false;
  t = tt;
  uu = u;
  vv = v;
  return true;
}

// Quad.Hit (pkg/geometry/quad.go:133-180).  Stored as 5 float4:
// (corner, D) (u, mat) (v, id) (normal, -) (W, -).
__device__ __forceinline__ bool hit_quad(float3 o, float3 d, const float4* q, float tmin, float tmax, float& t,
                                         float& alpha, float& beta) {
  float4 c = q[0];
  float3 n = f3(q[3]);
  float den = dot_rn(d, n);
  if (fabsf(den) < 1e-8f) return false;
  float tt = __fdiv_rn(__fsub_rn(c.w, dot_rn(o, n)), den);
  if (tt < tmin || tt > tmax) return false;
  float3 p = make_float3(__fmaf_rn(d.x, tt, o.x), __fmaf_rn(d.y, tt, o.y), __fmaf_rn(d.z, tt, o.z));
  float3 hv = sub_rn(p, f3(c));
  float3 U = f3(q[1]), V = f3(q[2]), W = f3(q[4]);
  float a = dot_rn(W, cross_rn(hv, V));
  float b = dot_rn(W, cross_rn(U, hv));
  if (a < 0.f || a > 1.f || b < 0.f || b > 1.f) return false;
  t = tt;
  alpha = a;
  beta = b;
  return true;
}

// Sphere.Hit (pkg/geometry/sphere.go:27-81): nearer root first, then the
// farther.  The discriminant uses the formulation of Haines, Guenther &
// Akenine-Moller, "Precision Improvements for Ray/Sphere Intersection"
// (Ray Tracing Gems, 2019, ch. 7) to keep FP32 usable for radius-1000
// spheres; the roots are the same quantities as (-halfB -/+ sqrt(D)) / a.
__device__ __forceinline__ bool hit_sphere(float3 o, float3 d, float4 s, float tmin, float tmax, float& t) {
  float3 f = sub_rn(o, f3(s));
  float a = dot_rn(d, d);
  float halfB = dot_rn(f, d);
  float k = __fdiv_rn(halfB, a);
  float3 l = make_float3(__fmaf_rn(-d.x, k, f.x), __fmaf_rn(-d.y, k, f.y), __fmaf_rn(-d.z, k, f.z));
  float r2 = __fmul_rn(s.w, s.w);
  float disc = __fmul_rn(a, __fsub_rn(r2, dot_rn(l, l)));
  if (disc < 0.f) return false;
  float sq = __fsqrt_rn(disc);
  float qq = __fsub_rn(-halfB, copysignf(sq, halfB));
  float c = __fsub_rn(dot_rn(f, f), r2);
  float t0, t1;
  if (qq == 0.f) {
    t0 = t1 = __fdiv_rn(-halfB, a);
  } else {
    float ra = __fdiv_rn(c, qq), rb = __fdiv_rn(qq, a);
    t0 = fminf(ra, rb);
    t1 = fmaxf(ra, rb);
  }
  float root = t0;
  if (root < tmin || root > tmax) {
    root = t1;
    if (root < tmin || root > tmax) return false;
  }
  t = root;
  return true;
}

// Disc (disc.go:49-92) and the circular caps of cylinders and cones
// (cylinder.go:224-266, cone.go:306-350): plane hit, |n.d| < eps rejected,
// inside when |p - c|^2 <= r^2.
__device__ __forceinline__ bool hit_cap_plane(float3 o, float3 d, float3 c, float3 n, float r, float eps, float tmin,
                                              float tmax, float& t) {
  float den = dot_rn(d, n);
  if (fabsf(den) < eps) return false;
  float tt = __fdiv_rn(dot_rn(sub_rn(c, o), n), den);
  if (tt < tmin || tt > tmax) return false;
  float3 p = make_float3(__fmaf_rn(d.x, tt, o.x), __fmaf_rn(d.y, tt, o.y), __fmaf_rn(d.z, tt, o.z));
  float3 cp = sub_rn(p, c);
  if (dot_rn(cp, cp) > __fmul_rn(r, r)) return false;
  t = tt;
  return true;
}

__device__ __forceinline__ float axial_height(float3 o, float3 d, float t, float3 base, float3 axis) {
  float3 p = make_float3(__fmaf_rn(d.x, t, o.x), __fmaf_rn(d.y, t, o.y), __fmaf_rn(d.z, t, o.z));
  return dot_rn(sub_rn(p, base), axis);
}

// Cylinder, cone and disc (cylinder.go:97-221, cone.go:128-303, disc.go:49).
// The quadratics are solved in the plane normal to the axis (cylinder) or
// with the half-b form and q = -(b' + sign(b') sqrt(D)) (cone), which keep
// FP32 roots accurate when the ray starts far away; the candidate order and
// the height / nappe checks are the reference's.  `part` tells the surface
// code which piece was hit: 0 body (or disc), 1 base cap, 2 top cap.
template <class Load>
__device__ __forceinline__ bool hit_quadric(float3 o, float3 d, const float4* Q, Load ld, float tmin, float tmax,
                                            float& t, float& part) {
  float4 g0 = ld(Q), g1 = ld(Q + 1), g4 = ld(Q + 4);
  int kind = __float_as_int(g4.x);
  float3 p0 = f3(g0), axis = f3(g1);
  if (kind == kQuadricDisc) {
    if (!hit_cap_plane(o, d, p0, axis, g0.w, 1e-6f, tmin, tmax, t)) return false;
    part = 0.f;
    return true;
  }
  float4 g2 = ld(Q + 2);
  float height = g1.w, best = tmax;
  bool any = false;
  if (kind == kQuadricCylinder) {
    float3 delta = sub_rn(o, p0);
    float DV = dot_rn(d, axis), dV = dot_rn(delta, axis);
    float3 dp = make_float3(__fmaf_rn(-axis.x, DV, d.x), __fmaf_rn(-axis.y, DV, d.y), __fmaf_rn(-axis.z, DV, d.z));
    float3 Dp = make_float3(__fmaf_rn(-axis.x, dV, delta.x), __fmaf_rn(-axis.y, dV, delta.y),
                            __fmaf_rn(-axis.z, dV, delta.z));
    float A = dot_rn(dp, dp);
    if (A >= 1e-8f) {
      float hb = dot_rn(Dp, dp);
      float k = __fdiv_rn(hb, A);
      float3 l = make_float3(__fmaf_rn(-dp.x, k, Dp.x), __fmaf_rn(-dp.y, k, Dp.y), __fmaf_rn(-dp.z, k, Dp.z));
      float r2 = __fmul_rn(g0.w, g0.w);
      float disc = __fmul_rn(A, __fsub_rn(r2, dot_rn(l, l)));
      if (disc >= 0.f) {
        float sq = __fsqrt_rn(disc);
        float q = __fsub_rn(-hb, copysignf(sq, hb));
        float C = __fsub_rn(dot_rn(Dp, Dp), r2);
        float t1, t2;
        if (q == 0.f) {
          t1 = t2 = __fdiv_rn(-hb, A);
        } else {
          float ra = __fdiv_rn(C, q), rb = __fdiv_rn(q, A);
          t1 = fminf(ra, rb);
          t2 = fmaxf(ra, rb);
        }
        float tc = t1;
        bool ok = true;
        if (tc < tmin || tc > best) {
          tc = t2;
          if (tc < tmin || tc > best) ok = false;
        }
        if (ok) {
          float h = axial_height(o, d, tc, p0, axis);
          if (h < 0.f || h > height) {
            ok = false;
            if (tc == t1) {
              tc = t2;
              if (!(tc < tmin || tc > best)) {
                h = axial_height(o, d, tc, p0, axis);
                ok = !(h < 0.f || h > height);
              }
            }
          }
        }
        if (ok) {
          best = tc;
          part = 0.f;
          any = true;
        }
      }
    }
  } else {
    float4 g3 = ld(Q + 3);
    float3 apex = f3(g3);
    float kk = __fadd_rn(1.f, g3.w);  // 1 + tan^2
    float3 CO = sub_rn(o, apex);
    float DV = dot_rn(d, axis), COV = dot_rn(CO, axis);
    float A = __fsub_rn(dot_rn(d, d), __fmul_rn(kk, __fmul_rn(DV, DV)));
    if (fabsf(A) >= 1e-8f) {
      float hb = __fsub_rn(dot_rn(d, CO), __fmul_rn(kk, __fmul_rn(DV, COV)));
      float C = __fsub_rn(dot_rn(CO, CO), __fmul_rn(kk, __fmul_rn(COV, COV)));
      float disc = __fmaf_rn(hb, hb, -__fmul_rn(A, C));
      if (disc >= 0.f) {
        float sq = __fsqrt_rn(disc);
        float q = __fsub_rn(-hb, copysignf(sq, hb));
        float ra, rb;
        if (q == 0.f) {
          ra = rb = __fdiv_rn(-hb, A);
        } else {
          ra = __fdiv_rn(C, q);
          rb = __fdiv_rn(q, A);
        }
        // the reference tries (-b - sqrt D) / 2a first: the smaller root when
        // a > 0, the larger when a < 0
        float first = A > 0.f ? fminf(ra, rb) : fmaxf(ra, rb);
        float second = A > 0.f ? fmaxf(ra, rb) : fminf(ra, rb);
        for (int pass = 0; pass < 2 && !any; pass++) {
          float tc = pass == 0 ? first : second;
          if (tc < tmin || tc > best) continue;
          float3 p = make_float3(__fmaf_rn(d.x, tc, o.x), __fmaf_rn(d.y, tc, o.y), __fmaf_rn(d.z, tc, o.z));
          float h = dot_rn(sub_rn(p, p0), axis);
          if (h < -1e-8f || h > height + 1e-8f) continue;
          if (dot_rn(sub_rn(p, apex), axis) > 1e-8f) continue;
          best = tc;
          part = 0.f;
          any = true;
        }
      }
    }
  }
  if (g4.z != 0.f) {  // caps: base (-axis), top (+axis) when it has a radius
    float tc;
    float3 na = make_float3(-axis.x, -axis.y, -axis.z);
    if (hit_cap_plane(o, d, p0, na, g0.w, 1e-8f, tmin, best, tc)) {
      best = tc;
      part = 1.f;
      any = true;
    }
    if (g2.w > 0.f && hit_cap_plane(o, d, f3(g2), axis, g2.w, 1e-8f, tmin, best, tc)) {
      best = tc;
      part = 2.f;
      any = true;
    }
  }
  if (any) t = best;
  return any;
}

// ----------------------------------------------------------------- BVH traversal
// Replaces geometry.BVH.Hit / hitNode (pkg/geometry/bvh.go:183-239).  The
// tree is this library's own 4-wide SAH BVH (layout.h) instead of the
// reference's binary midpoint BVH; the closest hit is the same, except that
// among candidates at exactly equal t the reference keeps the later one in
// its depth-first order while this traversal keeps the first one it meets.
struct TraceStats {
  uint32_t nodes, boxes, prims;
};

// What bounds the traversal and how it is laid out.  On a mesh the kernels
// are bound by instruction issue at a fraction of the lanes (IPC 2.0-2.4,
// 10-17 of 32 lanes per instruction with the boxes and leaves of a node in one
// loop), on a handful of rays by the chain of loads of a node visit.  So a
// visit is four 256-bit loads issued together and four box tests without a
// branch (packed multiply-adds: two planes per instruction; three-input
// minima and maxima, as the ALU is now the busiest pipe, at 65-75 %), and a
// primitive test is a step of its own, taken when enough lanes wait for it.
// The leaves of a visited node come before any node below it, in slot order,
// each checked against the hit so far when its turn comes: the primitives are
// tested in the order, and culled by the comparisons, of a loop that
// intersects each leaf as it meets it, so ties between equal distances fall
// the same way.  (The stack holds children that such a hit hides until they are
// popped: fit_stack in scene.cpp.)  Measured on GB300 against that loop, back
// to back: 2^24 rays on 1.3 M triangles (closest hit) 16.9 -> 9.2 ms, 300,007
// rays (any hit) on 81,920 triangles 130 -> 81 us, the 1024^2 x 16 frame of the
// 1.3 M triangles 28.6 -> 20.6 ms.

// State of one ray's traversal; `skip` is the primitive the ray leaves from:
// a ray cannot re-enter the plane of the triangle or quad it starts on, and
// for the sphere it starts on hits closer than 2e-4 x radius are rounding
// noise of the FP32 origin.
//
// A ray is in one of two steps: it tests primitives [prim, end) of a leaf, or
// (prim == end) it visits node `node`; node < 0 with no primitive left ends it.
// The leaves a visited node's boxes let through are tested before any node
// below it: `leaves` holds those of node `lnode` still to come (bit = child
// slot), and `node` / `node_t` meanwhile the child to visit after them
// (kPopNext: the top of the stack).
struct Trav {
  float3 o, d, inv, nood;  // nood = -(origin * inv)
  float tmin, best;        // best: the hit distance so far (tmax before a hit)
  uint32_t skip;
  int node, sp;
  float node_t;  // entry distance of `node`
  int lnode;
  unsigned leaves;
  int prim, end, type;
  uint32_t hit;  // primitive hit so far (kNoHit, or the marker kOverflowHit)
  float hu, hv;
  __device__ __forceinline__ bool testing() const { return prim < end; }
  __device__ __forceinline__ bool done() const { return prim >= end && node < 0; }
  __device__ __forceinline__ Hit result() const { return Hit{hit < kOverflowHit ? best : -1.f, hit, hu, hv}; }
};
constexpr int kPopNext = -2;

// One entry of a traversal stack: a node and the distance at which the ray
// enters its box.
struct TravEntry {
  int node;
  float t;
};

// 1 / d per axis, finite for directions along a plane.
__device__ __forceinline__ float3 ray_inverse(float3 d) {
  return f3(1.0f / (fabsf(d.x) > 1e-20f ? d.x : copysignf(1e-20f, d.x)),
            1.0f / (fabsf(d.y) > 1e-20f ? d.y : copysignf(1e-20f, d.y)),
            1.0f / (fabsf(d.z) > 1e-20f ? d.z : copysignf(1e-20f, d.z)));
}

// `root` is the BVH node the ray starts at (-1: nothing to intersect).  A
// root carrying kRootStackCap starts the ray with only kTestStackCap free
// stack entries (the stack is entered near its top, below a -1 sentinel that
// ends the traversal when popped), so that tests can drive the stack-overflow
// path of one job on an ordinary scene.
__device__ __forceinline__ void trav_init(Trav& s, float3 o, float3 d, float tmin, float tmax, uint32_t skip,
                                          int root, TravEntry* stack) {
  s.o = o;
  s.d = d;
  s.inv = ray_inverse(d);
  s.nood = -(o * s.inv);
  s.tmin = tmin;
  s.best = tmax;
  s.skip = skip;
  s.node = root;
  s.sp = 0;
  s.leaves = 0;
  s.prim = s.end = 0;
  if (root >= 0 && (root & kRootStackCap)) {
    s.node = root & ~kRootStackCap;
    s.sp = kTraceStack - kTestStackCap;
    stack[s.sp - 1] = TravEntry{-1, -kInfF};
  }
  s.hit = kNoHit;
  s.hu = s.hv = 0.f;
}

// The two planes of each axis of a child box, the child's reference and meta
// (layout.h), as four 64-bit words read in a single 256-bit load.
struct ChildRec {
  unsigned long long x, y, z, rm;
  __device__ __forceinline__ int ref() const { return (int)(unsigned)rm; }
  __device__ __forceinline__ int meta() const { return (int)(rm >> 32); }
};
__device__ __forceinline__ ChildRec ldg_child(const float4* p) {
  ChildRec c;
  asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(c.x), "=l"(c.y), "=l"(c.z), "=l"(c.rm) : "l"(p));
  return c;
}
// Both planes of one axis in one packed multiply-add: distances at which the
// ray meets them, each rounded as fmaf(plane, inv, nood).
__device__ __forceinline__ float2 slab(unsigned long long planes, float inv, float nood) {
  unsigned long long k, c, r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(k) : "f"(inv));
  asm("mov.b64 %0, {%1, %1};" : "=l"(c) : "f"(nood));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(planes), "l"(k), "l"(c));
  float2 t;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(t.x), "=f"(t.y) : "l"(r));
  return t;
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
// Entry and exit distance of the ray in a child box, before the ray's own
// far end.  Rounding is monotonic, so the nearer plane of each axis is the
// smaller distance.
__device__ __forceinline__ void span_of(float2 x, float2 y, float2 z, float tmin, float& tn, float& tf) {
  tn = max3(fminf(x.x, x.y), fminf(y.x, y.y), fmaxf(fminf(z.x, z.y), tmin));
  tf = min3(fmaxf(x.x, x.y), fmaxf(y.x, y.y), fmaxf(z.x, z.y));
}
__device__ __forceinline__ void child_span(float3 inv, float3 nood, float tmin, const ChildRec& c, float& tn,
                                           float& tf) {
  span_of(slab(c.x, inv.x, nood.x), slab(c.y, inv.y, nood.y), slab(c.z, inv.z, nood.z), tmin, tn, tf);
}
__device__ __forceinline__ void child_span(float3 inv, float3 nood, float tmin, const NodeChild& c, float& tn,
                                           float& tf) {
  auto axis = [](const float* p, float k, float c0) { return make_float2(__fmaf_rn(p[0], k, c0), __fmaf_rn(p[1], k, c0)); };
  span_of(axis(c.x, inv.x, nood.x), axis(c.y, inv.y, nood.y), axis(c.z, inv.z, nood.z), tmin, tn, tf);
}

// Moves the ray to the nearest entry left on its stack, leaving out those
// whose box starts behind the hit (nothing below them can be nearer).
__device__ __forceinline__ void trav_pop(Trav& s, const TravEntry* stack) {
  int node = -1;
  while (s.sp > 0) {
    const TravEntry e = stack[--s.sp];
    if (!(e.t > s.best)) {
      node = e.node;
      break;
    }
  }
  s.node = node;
}

// The first leaf of the node just visited, whose box was tested there.
__device__ __forceinline__ void trav_first_leaf(const DevScene& sc, Trav& s) {
  const int i = __ffs(s.leaves) - 1;
  s.leaves &= s.leaves - 1;
  const int2 rm = __ldg(reinterpret_cast<const int2*>(sc.nodes + (size_t)s.lnode * 8 + 2 * i + 1) + 1);
  s.prim = rm.x;
  s.end = rm.x + (rm.y & kLeafCountMask);
  s.type = (rm.y >> kLeafTypeShift) & 3;
}

// A ray that has met something at a distance which is not a number (the ray or
// the primitive is not one either): no node is known to be near enough then, so
// the children of `lnode`, whose leaves it has tested, are taken off the stack
// (they are its top entries), and it tests only the leaves of the nodes below
// them there, instead of visiting every node that those lead to.  A node is
// visited in full if a hit in its leaves is at a distance again.
__device__ __forceinline__ void trav_leaves_only(const DevScene& sc, Trav& s, const TravEntry* stack) {
  bool left = true;  // the top entry may be a child of lnode
  while (s.sp > 0 && stack[s.sp - 1].node >= 0) {  // negative: the sentinel of trav_init
    const int node = stack[s.sp - 1].node, from = left ? s.lnode : node;
    bool child = false;
    s.leaves = 0;
#pragma unroll 1
    for (int i = 0; i < 4; i++) {
      const ChildRec c = ldg_child(sc.nodes + (size_t)from * 8 + 2 * i);
      if (c.ref() == kEmptyChild) break;
      float tn, tf;
      child_span(s.inv, s.nood, s.tmin, c, tn, tf);
      if (c.meta() == 0) child |= c.ref() == node;
      else if (!(tn > tf)) s.leaves |= 1u << i;
    }
    if (left && !child) {
      left = false;
      continue;
    }
    s.sp--;
    if (!left && s.leaves) {
      s.node = s.lnode = node;
      s.node_t = -kInfF;
      trav_first_leaf(sc, s);
      return;
    }
  }
  s.leaves = 0;
  s.node = -1;
}

// The ray's next leaf of node `lnode`, or, when none is left, its next node.
// A leaf whose box starts behind a hit in a leaf before it is left out.
__device__ __forceinline__ void trav_next_leaf(const DevScene& sc, Trav& s, const TravEntry* stack) {
  while (s.leaves) {
    const int i = __ffs(s.leaves) - 1;
    s.leaves &= s.leaves - 1;
    const ChildRec c = ldg_child(sc.nodes + (size_t)s.lnode * 8 + 2 * i);
    float tn, tf;
    child_span(s.inv, s.nood, s.tmin, c, tn, tf);
    if (tn > s.best) continue;
    s.prim = c.ref();
    s.end = s.prim + (c.meta() & kLeafCountMask);
    s.type = (c.meta() >> kLeafTypeShift) & 3;
    return;
  }
  if (s.node == kPopNext || !(s.node_t <= s.best)) {
    if (s.best == s.best) trav_pop(s, stack);
    else trav_leaves_only(sc, s, stack);
  }
}

// The ray (o, d) against the record R (read through `ld`) of a primitive of
// type `type` with global id gid: a hit with t in [tmin, best].
template <class Load>
__device__ __forceinline__ bool hit_record(int type, const float4* R, Load ld, float3 o, float3 d, float tmin, float best,
                                           uint32_t skip, uint32_t gid, float& t, float& u, float& v) {
  u = v = 0.f;
  if (type == kPrimTriangle) {
    if (gid == skip) return false;
    return hit_triangle(o, d, ld(R), ld(R + 1), ld(R + 2), tmin, best, t, u, v);
  }
  if (type == kPrimQuad) {
    if (gid == skip) return false;
    float4 qq[5] = {ld(R), ld(R + 1), ld(R + 2), ld(R + 3), ld(R + 4)};
    return hit_quad(o, d, qq, tmin, best, t, u, v);
  }
  if (type == kPrimSphere) {
    float4 S = ld(R);
    float lo = gid == skip ? fmaxf(tmin, 2e-4f * fabsf(S.w)) : tmin;
    return hit_sphere(o, d, S, lo, best, t);
  }
  // a ray leaving a quadric may hit it again (the other side of a
  // cylinder); hits closer than 2e-4 x radius are its own surface
  float lo = tmin;
  if (gid == skip) {
    float4 g0 = ld(R);
    if (__float_as_int(ld(R + 4).x) == kQuadricDisc) return false;  // planar
    lo = fmaxf(tmin, 2e-4f * g0.w);
  }
  return hit_quadric(o, d, R, ld, lo, best, t, u);
}

// The ray against primitive p of type `type` of the scene.
__device__ __forceinline__ bool hit_prim(const DevScene& sc, int type, int p, float3 o, float3 d, float tmin, float best,
                                         uint32_t skip, uint32_t& gid, float& t, float& u, float& v) {
  auto ld = [](const float4* x) { return __ldg(x); };
  if (type == kPrimTriangle) {
    gid = (uint32_t)p;
    return hit_record(kPrimTriangle, sc.tris + (size_t)p * 3, ld, o, d, tmin, best, skip, gid, t, u, v);
  }
  if (type == kPrimQuad) {
    gid = sc.quad_base + (uint32_t)p;
    return hit_record(kPrimQuad, sc.quads + (size_t)p * 5, ld, o, d, tmin, best, skip, gid, t, u, v);
  }
  if (type == kPrimSphere) {
    gid = sc.sphere_base + (uint32_t)p;
    return hit_record(kPrimSphere, sc.spheres + (size_t)p * 2, ld, o, d, tmin, best, skip, gid, t, u, v);
  }
  gid = sc.quadric_base + (uint32_t)p;
  return hit_record(kPrimQuadric, sc.quadrics + (size_t)p * 5, ld, o, d, tmin, best, skip, gid, t, u, v);
}

// Tests the ray against primitive `prim` of its leaf and moves on: to the
// leaf's next primitive, the node's next leaf or the ray's next node.
template <bool kCount>
__device__ __forceinline__ void trav_prim(const DevScene& sc, Trav& s, bool any_hit, const TravEntry* stack,
                                          TraceStats* st) {
  uint32_t gid;
  float t, u, v;
  if (kCount) st->prims++;
  if (hit_prim(sc, s.type, s.prim++, s.o, s.d, s.tmin, s.best, s.skip, gid, t, u, v)) {
    s.best = t;
    s.hu = u;
    s.hv = v;
    s.hit = gid;
    if (any_hit) {
      s.node = -1;
      s.prim = s.end;
      return;
    }
  }
  if (s.prim == s.end) trav_next_leaf(sc, s, stack);
}

// Visits node s.node: tests its four children, pushes the farther internal
// ones, and moves the ray to the first leaf it meets there, else to the
// nearest internal child, else to the top of the stack.  When the farther
// children do not fit on the stack the ray ends at once with the marker hit
// (kOverflowHit): its result is not the closest hit, and the caller reports
// the bound against the ray's job.
template <bool kCount>
__device__ __forceinline__ void trav_visit(const DevScene& sc, Trav& s, TravEntry* stack, TraceStats* st) {
  const float4* N = sc.nodes + (size_t)s.node * 8;
  if (kCount) st->nodes++;
  ChildRec c[4];
#pragma unroll
  for (int i = 0; i < 4; i++) c[i] = ldg_child(N + 2 * i);
  float tn[4];  // entry distances of the internal children hit, else infinite
  int ref[4];
  unsigned leaves = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    float tf;
    child_span(s.inv, s.nood, s.tmin, c[i], tn[i], tf);
    ref[i] = c[i].ref();
    const bool used = ref[i] != kEmptyChild;
    if (kCount) st->boxes += used;
    const bool hit = used && !(tn[i] > fminf(tf, s.best));
    const bool leaf = c[i].meta() != 0;
    if (hit && leaf) leaves |= 1u << i;
    if (!hit || leaf) tn[i] = kInfF;
  }
  // nearest first: an odd-even transposition network, stable as only a
  // strictly greater neighbour changes places
  auto order = [&](int i, int j) {
    const bool swap = tn[i] > tn[j];
    const float t0 = swap ? tn[j] : tn[i], t1 = swap ? tn[i] : tn[j];
    const int r0 = swap ? ref[j] : ref[i], r1 = swap ? ref[i] : ref[j];
    tn[i] = t0;
    tn[j] = t1;
    ref[i] = r0;
    ref[j] = r1;
  };
  order(0, 1);
  order(2, 3);
  order(1, 2);
  order(0, 1);
  order(2, 3);
  order(1, 2);
  const bool p1 = tn[1] < kInfF, p2 = tn[2] < kInfF, p3 = tn[3] < kInfF;
  if (s.sp + p1 + p2 + p3 > kTraceStack) {
    s.node = -1;
    s.hit = kOverflowHit;
    return;
  }
  if (p3) stack[s.sp++] = TravEntry{ref[3], tn[3]};
  if (p2) stack[s.sp++] = TravEntry{ref[2], tn[2]};
  if (p1) stack[s.sp++] = TravEntry{ref[1], tn[1]};
  s.lnode = s.node;
  s.node = tn[0] < kInfF ? ref[0] : kPopNext;
  s.node_t = tn[0];
  s.leaves = leaves;
  if (leaves) trav_first_leaf(sc, s);
  else if (s.node == kPopNext) trav_pop(s, stack);
}

// Whole traversal of one ray from BVH node `root`.  A stack overflow returns
// no hit and, when `err` is given, sets kErrStackOverflow there.
template <bool kAnyHit, bool kCount>
__device__ __forceinline__ bool trace_from(const DevScene& sc, int root, float3 o, float3 d, float tmin, float tmax,
                                           uint32_t skip, Hit& hit, int* err, TraceStats* st = nullptr) {
  Trav s;
  TravEntry stack[kTraceStack];
  trav_init(s, o, d, tmin, tmax, skip, root, stack);
  while (s.node >= 0) {
    trav_visit<kCount>(sc, s, stack, st);
    while (s.testing()) trav_prim<kCount>(sc, s, kAnyHit, stack, st);
  }
  if (s.hit == kOverflowHit) {
    if (err) atomicOr(err, kErrStackOverflow);
    s.hit = kNoHit;
  }
  hit = s.result();
  return s.hit != kNoHit;
}

__host__ __device__ __forceinline__ bool one_node(const DevScene& sc) { return sc.one != nullptr; }

// What a kernel takes beside the scene: the one node, or nothing.
struct NoGeom {};
template <bool kOneNode>
struct GeomOf {
  using type = NoGeom;
};
template <>
struct GeomOf<true> {
  using type = OneNode;
};
template <bool kOneNode>
using Geom = typename GeomOf<kOneNode>::type;

// Whole traversal of one ray of a one-node scene: its leaves in slot order,
// each primitive by every lane of the warp at once, so that the loop, the
// type and the record's address are the same for all lanes; a lane whose ray
// misses the leaf's box (or without a ray: !live) sits it out.  The tests and
// their order are those of trav_visit / trav_prim, whose step per primitive
// costs more here than the lanes it fills.  The records come from the launch's
// constant bank: a 128-bit global load returns 512 bytes a warp, though all
// lanes read the same 16, and those loads kept the load pipe at 65-71 %; now
// issue bounds the loop.  Against the steps on global records: Cornell box (18
// quads) 400^2 x 64 10.26 -> 7.19 ms, Cornell boxes BDPT 512^2 x 64 86.0 -> 70.5
// ms, textured shapes 517 x 290 x 3 527 -> 345 us (of the 3 ms of the Cornell
// box the constant bank gave 0.25).
template <bool kCount>
__device__ __forceinline__ bool trace_one_node(const OneNode& g, bool live, bool any_hit, float3 o, float3 d, float tmin,
                                               float tmax, uint32_t skip, Hit& hit, TraceStats* st = nullptr) {
  const float3 inv = ray_inverse(d);
  const float3 nood = -(o * inv);
  auto ld = [](const float4* x) { return *x; };
  float best = tmax, hu = 0.f, hv = 0.f;
  uint32_t prim = kNoHit;
  if (kCount && live) st->nodes++;
  for (int i = 0; i < 4; i++) {
    const int ref = g.child[i].ref, meta = g.child[i].meta;
    if (ref == kEmptyChild) break;
    if (kCount && live) st->boxes++;
    float tn, tf;
    child_span(inv, nood, tmin, g.child[i], tn, tf);
    bool in = live && !(tn > fminf(tf, best)) && !(any_hit && prim != kNoHit);
    auto leaf = [&](int type, int stride) {
      const float4* R = g.rec + g.off[type] + ref * stride;
      uint32_t gid = g.base[type] + (uint32_t)ref;
      for (int k = meta & kLeafCountMask; k > 0; k--, R += stride, gid++) {
        float t, u, v;
        if (kCount && in) st->prims++;
        if (in && hit_record(type, R, ld, o, d, tmin, best, skip, gid, t, u, v)) {
          best = t;
          hu = u;
          hv = v;
          prim = gid;
          in = !any_hit;
        }
      }
    };
    const int type = (meta >> kLeafTypeShift) & 3;
    if (type == kPrimTriangle) leaf(kPrimTriangle, 3);
    else if (type == kPrimQuad) leaf(kPrimQuad, 5);
    else if (type == kPrimSphere) leaf(kPrimSphere, 2);
    else leaf(kPrimQuadric, 5);
  }
  hit = Hit{prim != kNoHit ? best : -1.f, prim, hu, hv};
  return prim != kNoHit;
}

// Whole traversal of one ray of the scene (the BDPT strategy kernels), in the
// form for one_node(sc): a kernel holds one form, as both together spill.
template <bool kAnyHit, bool kOneNode>
__device__ __forceinline__ bool trace(const DevScene& sc, const Geom<kOneNode>& g, float3 o, float3 d, float tmin,
                                      float tmax, uint32_t skip, Hit& hit, int* err) {
  if constexpr (kOneNode) return trace_one_node<false>(g, true, kAnyHit, o, d, tmin, tmax, skip, hit);
  else return trace_from<kAnyHit, false>(sc, sc.root, o, d, tmin, tmax, skip, hit, err);
}

// A batch of rays of a one-node scene, one ray per thread (every ray costs
// the same, so there is nothing to refill).
template <bool kAnyHit, bool kCount, class Source>
__device__ __forceinline__ void trace_batch_one_node(const OneNode& g, Source& src, TraceStats* st, uint32_t* traced) {
  const uint32_t n = src.count();
  deal_blocks(n, blockIdx.x * blockDim.x, gridDim.x * blockDim.x, [&](uint64_t base) {
    const bool live = base + threadIdx.x < n;
    const uint32_t i = (uint32_t)base + threadIdx.x;
    float3 o = f3(0.f, 0.f, 0.f), d = f3(0.f, 0.f, 1.f);
    float tmin = 0.f, tmax = 0.f;
    uint32_t skip = kNoHit;
    int root;
    if (live) src.load(i, o, d, tmin, tmax, skip, root);
    Hit h;
    trace_one_node<kCount>(g, live, kAnyHit, o, d, tmin, tmax, skip, h, st);
    if (live) {
      src.store(i, h);
      if (kCount) (*traced)++;
    }
  });
}

// The step of a warp whose lanes `busy` are on a ray and `testing` wait for a
// primitive test: a test costs about a third of a node visit, so it is taken
// once more than a third of the lanes wait for it (1/2 and 1/4: 21.0 and 20.8
// against 20.6 ms for the frame of 1.3 M triangles; 68.0 and 68.4 against 67.9
// ms for 32 sphere scenes).
__device__ __forceinline__ bool trav_test_now(unsigned testing, unsigned busy) {
  return 3 * __popc(testing) > __popc(busy);
}

// Persistent traversal of a batch of rays: every warp loops until its work
// is exhausted, one step per iteration (trav_test_now), and lanes whose ray
// finished take new rays once at least 16 lanes are idle (8 and 24: 69.6 and
// 69.6 against 67.9 ms on the sphere batch, 20.4 and 22.0 against 20.6 ms on
// 1.3 M triangles), so warps stay full instead of waiting for their slowest
// ray.  Rays are dealt in chunks of up to 64 (deal.h).  Warp w of W
// starts on chunk w; with `work` != null the chunks after the first W come
// from that counter (zeroed by the previous kernel on the same stream),
// otherwise warp w goes on with chunks w + W, w + 2 W, ... (calls on
// different streams share no counter; one contiguous range per warp left the
// warps of the cheap half of a batch idle).  A batch of fewer than 64 rays per
// warp is dealt out in one smaller chunk per warp, so that it spreads over
// the chip and draws nothing from the counter.  Source provides count(),
// load(i, o, d, tmin, tmax, skip, root) and store(i, hit); store() sees the
// marker hit of a ray that overflowed its stack and reports it.
constexpr uint32_t kFetchChunk = 64;
constexpr uint32_t kNoRay = 0xffffffffu;  // no ray in a batch has this number
constexpr int kRefillIdle = 16;
// 128-thread blocks per SM of the traversal kernels: 64 registers, up to 54
// bytes spilled; 7 blocks (72 registers) and 6 (80) measured 2 and 8 % slower
// on the sphere batch and on the frame of 1.3 M triangles (its raw batch of
// 2^24 rays 4 % faster and 2 % slower).
constexpr int kTravBlocks = 8;

template <bool kAnyHit, bool kCount, class Source>
__device__ __forceinline__ void trace_persistent(const DevScene& sc, Source& src, uint32_t* work, TraceStats* st,
                                                 uint32_t* traced) {
  const uint32_t n = src.count();
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t chunk = deal_chunk(n, nw, kFetchChunk);
  // the warp's current chunk [cur, end), warp-uniform
  uint32_t cur = deal_at(n, (uint64_t)w * chunk), end = deal_at(n, (uint64_t)cur + chunk);
  bool more = cur < end;  // the warp may still draw rays
  uint32_t next = w;      // without `work`: the chunk it holds
  Trav s;
  TravEntry stack[kTraceStack];
  uint32_t ray = kNoRay;
  for (;;) {
    const bool idle = ray == kNoRay, testing = !idle && s.testing();
    const unsigned idle_mask = __ballot_sync(0xffffffffu, idle), test_mask = __ballot_sync(0xffffffffu, testing);
    if (more && __popc(idle_mask) >= kRefillIdle) {
      if (cur == end) {
        uint64_t at;
        if (work) {
          uint32_t base = 0;
          if (n > (uint64_t)nw * chunk && lane == 0) base = atomicAdd(work, chunk);
          at = (uint64_t)nw * chunk + __shfl_sync(0xffffffffu, base, 0);
        } else {
          next += nw;
          at = (uint64_t)next * chunk;
        }
        cur = deal_at(n, at);
        end = deal_at(n, at + chunk);
      }
      if (cur == end) {
        more = false;
      } else {
        uint32_t take = min((uint32_t)__popc(idle_mask), end - cur);
        uint32_t rank = (uint32_t)__popc(idle_mask & lt);
        if (idle && rank < take) {
          float3 o, d;
          float tmin, tmax;
          uint32_t skip;
          int root;
          uint32_t mine = cur + rank;
          src.load(mine, o, d, tmin, tmax, skip, root);
          trav_init(s, o, d, tmin, tmax, skip, root, stack);
          ray = mine;
          if (kCount) (*traced)++;
        }
        cur += take;
      }
      continue;
    }
    if (idle_mask == 0xffffffffu) break;
    if (trav_test_now(test_mask, ~idle_mask)) {
      if (testing) trav_prim<kCount>(sc, s, kAnyHit, stack, st);
    } else if (!idle && !testing && s.node >= 0) {
      trav_visit<kCount>(sc, s, stack, st);
    }
    if (!idle && s.done()) {
      src.store(ray, s.result());
      ray = kNoRay;
    }
  }
}

// Warp-aggregated append: one atomic per warp, lanes get consecutive slots.
__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool want) {
  unsigned mask = __ballot_sync(__activemask(), want);
  if (!want) return 0;
  int lane = threadIdx.x & 31;
  int leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
  base = __shfl_sync(mask, base, leader);
  return base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

// The same in two parts: the lanes that call warp_reserve together take
// consecutive places (one atomic), and each reads its own where it needs it,
// so that what lies between hides the atomic's way to L2 and back.
struct Reserve {
  unsigned mask;  // the lanes that reserved together
  uint32_t base;  // the first place, in their lowest lane
};
__device__ __forceinline__ Reserve warp_reserve(uint32_t* counter) {
  Reserve r;
  r.mask = __activemask();
  r.base = 0;
  if ((threadIdx.x & 31) == (unsigned)(__ffs(r.mask) - 1)) r.base = atomicAdd(counter, (uint32_t)__popc(r.mask));
  return r;
}
__device__ __forceinline__ uint32_t reserved_slot(const Reserve& r) {
  return __shfl_sync(r.mask, r.base, __ffs(r.mask) - 1) + (uint32_t)__popc(r.mask & ((1u << (threadIdx.x & 31)) - 1u));
}

// Largest k < n with start[k] <= x (start[0] = 0, start ascending).
__device__ __forceinline__ uint32_t find_range(const uint32_t* start, uint32_t n, uint32_t x) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (__ldg(start + mid) <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Where a wavefront reports a device bound of one path: the job's error
// word, or, in a multi-job wavefront, the error word of the work item whose
// path range [start[k], start[k+1]) holds the path's origin index, so that
// only that job fails.
struct ErrSink {
  uint32_t* word;           // single job: its error word
  uint32_t* items;          // multi-job: one error word per item (else null)
  const uint32_t* start;    // multi-job: first origin index of each item
  const uint32_t* n_items;  // multi-job: items of the step
  __device__ void report(uint32_t origin, uint32_t bits) const {
    if (items) atomicOr(items + find_range(start, *n_items, origin), bits);
    else atomicOr(word, bits);
  }
};

// ----------------------------------------------------------------- surface data
// Resolves a hit into the SurfaceInteraction of the reference: point,
// front-face shading normal (SetFaceNormal, pkg/material/interfaces.go:58-65)
// and material.
struct Surface {
  float3 p, n;
  bool front;
  int mat;
  float2 uv;  // SurfaceInteraction.UV, set when the scene has textures
};

// UV of a point on a cylinder / cone body (cylinder.go:187-205, cone.go:234-253)
__device__ __forceinline__ float2 axial_uv(float3 axis, float3 radial, float h, float height) {
  float3 ref = fabsf(axis.y) < 0.9f ? f3(0.f, 1.f, 0.f) : f3(1.f, 0.f, 0.f);
  float3 tangent = normalize(cross(axis, ref));
  float3 bitangent = cross(axis, tangent);
  float a = atan2f(dot(radial, bitangent), dot(radial, tangent));
  return make_float2((a + kPi) / (2.f * kPi), h / height);
}
// UV of a point on a cap of outward normal n (cylinder.go:241-255, cone.go:322-339)
__device__ __forceinline__ float2 cap_uv(float3 n, float3 c, float r, float3 p) {
  float3 ref = fabsf(n.y) < 0.9f ? f3(0.f, 1.f, 0.f) : f3(1.f, 0.f, 0.f);
  float3 tangent = normalize(cross(n, ref));
  float3 bitangent = cross(n, tangent);
  float3 l = p - c;
  return make_float2((dot(l, tangent) / r + 1.f) * 0.5f, (dot(l, bitangent) / r + 1.f) * 0.5f);
}

// `yx`: the rounding of a cylinder or cone body's normal (normalize_yx, the
// path tracer's; else normalize_xy, the BDPT subpaths').
__device__ __forceinline__ void surface_at(const DevScene& sc, float3 o, float3 d, const Hit& h, Surface& s, bool yx) {
  s.p = o + d * h.t;  // Ray.At (pkg/core/vec3.go:216-218)
  float3 outward;
  uint32_t p = h.prim;
  const bool uv = sc.has_textures;
  if (p < sc.quad_base) {
    const float4* T = sc.tris + (size_t)p * 3;
    float4 a = __ldg(T);
    float4 nn = __ldg(sc.tri_normals + p);
    outward = f3(nn);  // precomputed normalize(e1 x e2) (triangle.go:92-99)
    s.mat = __float_as_int(a.w);
    if (uv) {  // per-vertex UVs interpolated with the barycentrics, else the barycentrics (triangle.go:151-161)
      s.uv = make_float2(h.u, h.v);
      if (sc.tri_uvs) {
        float4 A = __ldg(sc.tri_uvs + 2 * (size_t)p), Bq = __ldg(sc.tri_uvs + 2 * (size_t)p + 1);
        if (Bq.z != 0.f) {
          float w = 1.f - h.u - h.v;
          s.uv = make_float2(A.x * w + A.z * h.u + Bq.x * h.v, A.y * w + A.w * h.u + Bq.y * h.v);
        }
      }
    }
  } else if (p < sc.sphere_base) {
    const float4* Q = sc.quads + (size_t)(p - sc.quad_base) * 5;
    outward = f3(__ldg(Q + 3));
    s.mat = __float_as_int(__ldg(Q + 1).w);
    if (uv) s.uv = make_float2(h.u, h.v);  // (alpha, beta) (quad.go:165-166)
  } else if (p < sc.quadric_base) {
    const float4* S = sc.spheres + (size_t)(p - sc.sphere_base) * 2;
    float4 c = __ldg(S);
    outward = (s.p - f3(c)) * (1.0f / c.w);  // (p - c) / r (sphere.go:62)
    s.mat = __float_as_int(__ldg(S + 1).x);
    if (uv) {  // spherical angles (sphere.go:64-68)
      float theta = acosf(fminf(1.f, fmaxf(-1.f, -outward.y)));
      float phi = atan2f(-outward.z, outward.x) + kPi;
      s.uv = make_float2(phi / (2.f * kPi), theta / kPi);
    }
  } else {
    const float4* Q = sc.quadrics + (size_t)(p - sc.quadric_base) * 5;
    float4 g0 = __ldg(Q), g1 = __ldg(Q + 1), g4 = __ldg(Q + 4);
    float3 axis = f3(g1);
    int kind = __float_as_int(g4.x);
    s.mat = __float_as_int(g4.y);
    if (kind == kQuadricDisc) {
      outward = axis;
      if (uv) {  // disc.go:68-73
        float3 l = s.p - f3(g0);
        s.uv = make_float2((dot(l, f3(__ldg(Q + 2))) / g0.w + 1.f) * 0.5f,
                           (dot(l, f3(__ldg(Q + 3))) / g0.w + 1.f) * 0.5f);
      }
    } else if (h.u == 2.f) {
      outward = axis;  // top cap
      if (uv) {
        float4 g2 = __ldg(Q + 2);
        s.uv = cap_uv(axis, f3(g2), g2.w, s.p);
      }
    } else if (h.u == 1.f) {
      outward = -axis;  // base cap
      if (uv) s.uv = cap_uv(-axis, f3(g0), g0.w, s.p);
    } else {
      // body: radial from the axis (cylinder.go:188-191), tilted by the
      // cone's slope (cone.go:240-248)
      float3 base = f3(g0);
      float hh = dot(s.p - base, axis);
      float3 radial = s.p - (base + axis * hh);
      if (uv) s.uv = axial_uv(axis, radial, hh, g1.w);
      if (kind == kQuadricCone) radial = radial + axis * ((g0.w - __ldg(Q + 2).w) / g1.w);
      outward = yx ? normalize_yx(radial) : normalize_xy(radial);
    }
  }
  s.front = dot(d, outward) < 0.f;
  s.n = s.front ? outward : -outward;
}

// ----------------------------------------------------------------- materials
__device__ __forceinline__ DevMaterial load_material(const DevScene& sc, int m) { return sc.materials[m]; }

// ImageTexture.Evaluate (image_texture.go:25-52): u, v wrapped into [0,1)
// (Go's int() truncates toward zero), nearest texel, v = 0 at the last row
__device__ __forceinline__ float3 tex_eval(const DevScene& sc, int t, float2 uv) {
  uint4 ti = __ldg(sc.tex_info + t);
  float u = uv.x - truncf(uv.x), v = uv.y - truncf(uv.y);
  if (u < 0.f) u += 1.f;
  if (v < 0.f) v += 1.f;
  int x = (int)(u * (float)ti.y), y = (int)((1.f - v) * (float)ti.z);
  x = min(max(x, 0), (int)ti.y - 1);
  y = min(max(y, 0), (int)ti.z - 1);
  return f3(__ldg(sc.texels + ti.x + (size_t)y * ti.y + (uint32_t)x));
}
// ColorSource.Evaluate of a Lambertian / Metal albedo (color_source.go)
__device__ __forceinline__ float3 albedo_at(const DevScene& sc, const DevMaterial& m, const Surface& s) {
  return m.tex >= 0 ? tex_eval(sc, m.tex, s.uv) : m.albedo;
}

__device__ __forceinline__ float3 reflect(float3 v, float3 n) { return v - n * (2.f * dot(v, n)); }
// refractVector (pkg/material/dielectric.go:158-163)
__device__ __forceinline__ float3 refract(float3 uv, float3 n, float eta) {
  float ct = fminf(-dot(uv, n), 1.0f);
  float3 perp = (uv + n * ct) * eta;
  float3 par = n * (-sqrtf(fabsf(1.0f - dot(perp, perp))));
  return perp + par;
}
// Reflectance, Schlick (dielectric.go:166-172); pow(x,5) as a product
__device__ __forceinline__ float schlick(float c, float ratio) {
  float r0 = (1.f - ratio) / (1.f + ratio);
  r0 = r0 * r0;
  float x = 1.f - c;
  float x2 = x * x;
  return r0 + (1.f - r0) * (x2 * x2 * x);
}

struct Scatter {
  float3 dir;  // scattered direction (not normalised for metal, like the reference)
  float3 att;
  float pdf;   // <= 0: specular (ScatterResult.IsSpecular, interfaces.go:42-45)
};

// Material.Scatter for Lambertian / Metal / Dielectric / Emissive / Layered
// (lambertian.go:25-49, metal.go:38-62, dielectric.go:20-59,
// emissive.go:17-21, layered.go:24-79).  Returns didScatter.
__device__ __forceinline__ bool scatter_basic(const DevScene& sc, const DevMaterial& m, float3 din, const Surface& s,
                                              Rng& rng, Scatter& out) {
  switch (m.kind) {
    case kMatLambertian: {
      float2 u = rng.next2();
      float3 dir = sample_cosine_hemisphere(s.n, u);
      float c = fmaxf(0.f, dot(normalize_xy(dir), s.n));
      out.dir = dir;
      out.att = albedo_at(sc, m, s) * (1.0f / kPi);
      out.pdf = c / kPi;
      return true;
    }
    case kMatMetal: {
      float3 r = reflect(normalize_xy(din), s.n);
      if (m.fuzz > 0.f) {
        float a = rng.next(), b = rng.next(), c = rng.next();
        r = r + sample_in_unit_sphere(f3(a, b, c)) * m.fuzz;
      }
      out.dir = r;
      out.att = albedo_at(sc, m, s);
      out.pdf = 0.f;
      return dot(r, s.n) > 0.f;
    }
    case kMatDielectric: {
      float ratio = s.front ? 1.0f / m.ior : m.ior;
      float3 ud = normalize_xy(din);
      float ct = fminf(-dot(ud, s.n), 1.0f);
      float st = sqrtf(1.0f - ct * ct);
      bool cannot = ratio * st > 1.0f;
      // no sample is drawn under total internal reflection (Go's || short-circuit)
      if (cannot || schlick(ct, ratio) > rng.next())
        out.dir = reflect(ud, s.n);
      else
        out.dir = refract(ud, s.n, ratio);
      out.att = f3(1.f, 1.f, 1.f);
      out.pdf = 0.f;
      return true;
    }
    default:
      return false;  // Emissive absorbs
  }
}

__device__ __forceinline__ bool scatter(const DevScene& sc, const DevMaterial& m, float3 din, const Surface& s,
                                        Rng& rng, Scatter& out) {
  if (m.kind == kMatMix)  // Mix.Scatter (mix.go:30-37): material 2 below the ratio
    return scatter_basic(sc, load_material(sc, rng.next() < m.fuzz ? m.inner : m.outer), din, s, rng, out);
  if (m.kind != kMatLayered) return scatter_basic(sc, m, din, s, rng, out);
  DevMaterial mo = load_material(sc, m.outer);
  Scatter o;
  if (!scatter_basic(sc, mo, din, s, rng, o)) return false;
  float3 sd = normalize(o.dir);
  if (!(dot(sd, s.n) < 0.f)) {
    out = o;
    return true;
  }
  DevMaterial mi = load_material(sc, m.inner);
  Scatter in;
  if (!scatter_basic(sc, mi, sd, s, rng, in)) {
    out = o;
    return true;
  }
  out.dir = in.dir;
  out.att = o.att * in.att;
  out.pdf = in.pdf;
  return true;
}

// EvaluateBRDF (lambertian.go:52-62, metal.go:65-77, dielectric.go:62-142,
// emissive.go:35-38, layered.go:81-95)
__device__ __forceinline__ float3 brdf_basic(const DevScene& sc, const DevMaterial& m, float3 in, float3 out,
                                             const Surface& s, bool radiance) {
  switch (m.kind) {
    case kMatLambertian:
      if (dot(out, s.n) <= 0.f) return f3(0.f, 0.f, 0.f);
      return albedo_at(sc, m, s) * (1.0f / kPi);
    case kMatMetal: {
      float3 r = reflect(-in, s.n);
      if (length(out - r) < 0.001f) return albedo_at(sc, m, s);
      return f3(0.f, 0.f, 0.f);
    }
    case kMatDielectric: {
      float3 wi = normalize(in), wo = normalize(out), n = normalize(s.n);
      float wiN = dot(wi, n), woN = dot(wo, n);
      bool same = (wiN > 0.f) == (woN > 0.f);
      float ratio = s.front ? 1.0f / m.ior : m.ior;
      if (!same) {
        float3 r = reflect(wi, n);
        if (length(wo - r) < 0.001f) {
          float f = schlick(fabsf(wiN), ratio);
          return f3(f, f, f);
        }
      } else {
        float3 rf = refract(wi, n, ratio);
        if (length(wo - rf) < 0.001f) {
          float tr = 1.f - schlick(fabsf(wiN), ratio);
          if (radiance) {
            float etap = s.front ? m.ior : 1.0f / m.ior;
            tr /= etap * etap;
          }
          return f3(tr, tr, tr);
        }
      }
      return f3(0.f, 0.f, 0.f);
    }
    default:
      return f3(0.f, 0.f, 0.f);
  }
}

// isReflectionPath (layered.go:110-119)
__device__ __forceinline__ bool is_reflection_path(float3 in, float3 out, float3 n) {
  float3 inc = -in;
  float3 r = inc - n * (2.f * dot(inc, n));
  return length(out - r) < 0.1f;
}

__device__ __forceinline__ float3 brdf(const DevScene& sc, const DevMaterial& m, float3 in, float3 out,
                                       const Surface& s, bool radiance) {
  if (m.kind == kMatMix)  // Mix.EvaluateBRDF (mix.go:40-46)
    return brdf_basic(sc, load_material(sc, m.outer), in, out, s, radiance) * (1.f - m.fuzz) +
           brdf_basic(sc, load_material(sc, m.inner), in, out, s, radiance) * m.fuzz;
  if (m.kind != kMatLayered) return brdf_basic(sc, m, in, out, s, radiance);
  int sub = is_reflection_path(in, out, s.n) ? m.outer : m.inner;
  return brdf_basic(sc, load_material(sc, sub), in, out, s, radiance);
}

// Material.PDF (lambertian.go:65-72, metal.go:80-84, dielectric.go:145-149,
// emissive.go:41-44, layered.go:98-107).  Returns pdf; sets delta.
__device__ __forceinline__ float pdf_basic(const DevMaterial& m, float3 out, float3 n, bool& delta) {
  switch (m.kind) {
    case kMatLambertian: {
      delta = false;
      float c = dot(out, n);
      return c <= 0.f ? 0.f : c / kPi;
    }
    case kMatMetal:
    case kMatDielectric:
      delta = true;
      return 0.f;
    default:
      delta = false;
      return 0.f;
  }
}
__device__ __forceinline__ float mat_pdf(const DevScene& sc, const DevMaterial& m, float3 in, float3 out, float3 n,
                                         bool& delta) {
  if (m.kind == kMatMix) {  // Mix.PDF (mix.go:49-59): never delta
    bool d;
    float p1 = pdf_basic(load_material(sc, m.outer), out, n, d);
    float p2 = pdf_basic(load_material(sc, m.inner), out, n, d);
    delta = false;
    return p1 * (1.f - m.fuzz) + p2 * m.fuzz;
  }
  if (m.kind != kMatLayered) return pdf_basic(m, out, n, delta);
  int sub = is_reflection_path(in, out, n) ? m.outer : m.inner;
  bool d;
  float p = pdf_basic(load_material(sc, sub), out, n, d);
  delta = false;
  return p;
}

// Material Emit with a hit record, for a ray of direction d: Emissive
// (emissive.go:24-32) emits from the front face; the disc spot light's
// emitter (disc_spot_light.go:26-48) also needs d against its spot direction
// (cosine at most -0.3, d as given).
__device__ __forceinline__ float3 emitted(const DevMaterial& m, bool front, float3 d) {
  if (!front) return f3(0.f, 0.f, 0.f);
  if (m.kind == kMatEmissive) return m.emission;
  if (m.kind == kMatSpotEmissive && dot(d, m.albedo) <= -0.3f) return m.emission;
  return f3(0.f, 0.f, 0.f);
}

// ----------------------------------------------------------------- lights
struct LightSample {
  float3 point, normal, dir;
  float dist;
  float3 emission;
  float pdf;
};

__device__ __forceinline__ float3 gradient_emission(const DevLight& L, float3 dnorm) {
  float t = 0.5f * (dnorm.y + 1.0f);
  return L.b * (1.0f - t) + L.a * t;
}

// Spot falloff (point_spot_light.go:140-158, disc_spot_light.go:150-168)
__device__ __forceinline__ float spot_falloff(const DevLight& L, float c) {
  if (c < L.cos_total) return 0.f;
  if (c >= L.cos_falloff) return 1.f;
  float x = (c - L.cos_total) / (L.cos_falloff - L.cos_total);
  x = x * x;
  return x * x;
}

// Disc.SampleUniform (disc.go:120-134) on a disc record (centre + radius,
// normal, right, up)
__device__ __forceinline__ float3 disc_point(const float4* Q, float2 u) {
  float4 g0 = __ldg(Q);
  float r = sqrtf(u.x) * g0.w;
  float s_, c_;
  sincosf(2.f * kPi * u.y, &s_, &c_);
  return f3(g0) + f3(__ldg(Q + 2)) * (r * c_) + f3(__ldg(Q + 3)) * (r * s_);
}

// Light.Sample (quad_light.go:36-86, sphere_light.go:29-141,
// uniform_infinite_light.go:66-80, gradient_infinite_light.go:77-91,
// disc_light.go, disc_spot_light.go, point_spot_light.go)
__device__ __forceinline__ LightSample light_sample(const DevScene& sc, const DevLight& L, float3 p, float3 n,
                                                    float2 u) {
  LightSample ls;
  if (L.kind == kLightQuad) {
    const float4* Q = sc.quads + (size_t)L.prim * 5;
    float3 c = f3(__ldg(Q)), U = f3(__ldg(Q + 1)), V = f3(__ldg(Q + 2)), N = f3(__ldg(Q + 3));
    float3 sp = c + U * u.x + V * u.y;
    float3 to = sp - p;
    float dist = length(to);
    float3 dir = to * (1.0f / dist);
    float ct = fabsf(dot(N, -dir));
    ls.point = sp;
    ls.normal = N;
    ls.dir = dir;
    ls.dist = dist;
    if (ct < 1e-8f) {
      ls.emission = f3(0.f, 0.f, 0.f);
      ls.pdf = 0.f;
      return ls;
    }
    ls.pdf = (1.0f / L.area) * dist * dist / ct;
    ls.emission = dot(dir, N) < 0.f ? L.a : f3(0.f, 0.f, 0.f);
    return ls;
  }
  if (L.kind == kLightSphere) {
    float4 S = make_float4(L.pos.x, L.pos.y, L.pos.z, L.radius);
    float3 c = f3(S);
    float r = S.w;
    float3 tc = c - p;
    float dc = length(tc);
    bool uniform = dc <= r;
    if (!uniform) {
      // sampleVisible (sphere_light.go:81-141)
      float3 w = normalize(tc);
      float3 uu = fabsf(w.x) > 0.1f ? f3(0.f, 1.f, 0.f) : f3(1.f, 0.f, 0.f);
      uu = normalize(cross(uu, w));
      float3 vv = cross(w, uu);
      float sinMax = r / dc;
      float cosMax = sqrtf(fmaxf(0.f, 1.f - sinMax * sinMax));
      float ct = 1.f - u.x * (1.f - cosMax);
      float st = sqrtf(fmaxf(0.f, 1.f - ct * ct));
      float sp2, cp2;
      sincosf(2.f * kPi * u.y, &sp2, &cp2);
      float3 dir = uu * (st * cp2) + vv * (st * sp2) + w * ct;
      float t;
      if (hit_sphere(p, dir, S, 0.001f, kInfF, t)) {
        float3 hp = p + dir * t;
        float3 on = (hp - c) * (1.0f / r);
        ls.point = hp;
        ls.normal = dot(dir, on) < 0.f ? on : -on;
        ls.dir = dir;
        ls.dist = t;
        ls.emission = L.a;
        ls.pdf = 1.0f / (2.f * kPi * (1.f - cosMax));
        return ls;
      }
      uniform = true;  // the reference falls back to uniform sampling
    }
    // sampleUniform (sphere_light.go:44-78)
    float z = 1.f - 2.f * u.x;
    float rr = sqrtf(fmaxf(0.f, 1.f - z * z));
    float sp3, cp3;
    sincosf(2.f * kPi * u.y, &sp3, &cp3);
    float3 ld = f3(rr * cp3, rr * sp3, z);
    float3 sp = c + ld * r;
    float3 dd = sp - p;
    ls.point = sp;
    ls.normal = ld;
    ls.dir = normalize(dd);
    ls.dist = length(dd);
    ls.emission = L.a;
    ls.pdf = 1.0f / (4.f * kPi * r * r);
    return ls;
  }
  if (L.kind == kLightDisc || L.kind == kLightDiscSpot) {
    // DiscLight.Sample (disc_light.go:28-75); the spot variant scales the
    // emission by the falloff seen from the sampled point (disc_spot_light.go:115-130)
    const float4* Q = sc.quadrics + (size_t)L.prim * 5;
    float3 N = f3(__ldg(Q + 1));
    float3 sp = disc_point(Q, u);
    float3 to = sp - p;
    float dist = length(to);
    ls.point = sp;
    ls.normal = N;
    if (dist == 0.f) {
      ls.dir = f3(0.f, 1.f, 0.f);
      ls.dist = 0.f;
      ls.emission = f3(0.f, 0.f, 0.f);
      ls.pdf = 1.f;
      return ls;
    }
    float3 dir = to * (1.0f / dist);
    float ct = fabsf(dot(N, -dir));
    ls.pdf = ct < 1e-6f ? 0.f : (1.0f / L.area) * dist * dist / ct;
    ls.dir = dir;
    ls.dist = dist;
    ls.emission = L.a;  // Emit(ray, nil) of the emissive material
    if (L.kind == kLightDiscSpot) {
      if (dot(dir, L.b) > -0.3f) ls.emission = f3(0.f, 0.f, 0.f);
      ls.emission = ls.emission * spot_falloff(L, dot(L.b, normalize(p - sp)));
    }
    return ls;
  }
  if (L.kind == kLightPointSpot) {
    // PointSpotLight.Sample (point_spot_light.go:46-97)
    float3 to = L.pos - p;
    float dist = length(to);
    ls.point = L.pos;
    ls.pdf = 1.f;
    if (dist == 0.f) {
      ls.normal = ls.dir = f3(0.f, 1.f, 0.f);
      ls.dist = 0.f;
      ls.emission = f3(0.f, 0.f, 0.f);
      return ls;
    }
    float3 tl = to * (1.0f / dist);
    ls.emission = L.a * (spot_falloff(L, dot(L.b, -tl)) / (dist * dist));
    ls.normal = -tl;
    ls.dir = tl;
    ls.dist = dist;
    return ls;
  }
  // infinite lights: cosine-weighted hemisphere about the shading normal
  float3 dir = sample_cosine_hemisphere(n, u);
  ls.point = p + dir * 1e10f;
  ls.normal = -dir;
  ls.dir = dir;
  ls.dist = kInfF;
  ls.emission = L.kind == kLightUniformInfinite ? L.a : gradient_emission(L, dir);
  ls.pdf = dot(dir, n) / kPi;
  return ls;
}

// Light.PDF (quad_light.go:90-109, sphere_light.go:144-166,
// uniform_infinite_light.go:83-91, gradient_infinite_light.go:94-102,
// disc_light.go:78-100 (also the disc spot light), point_spot_light.go:101-118)
__device__ __forceinline__ float light_pdf(const DevScene& sc, const DevLight& L, float3 p, float3 n, float3 dir) {
  if (L.kind == kLightQuad) {
    const float4* Q = sc.quads + (size_t)L.prim * 5;
    float4 qq[5] = {__ldg(Q), __ldg(Q + 1), __ldg(Q + 2), __ldg(Q + 3), __ldg(Q + 4)};
    float t, a, b;
    if (!hit_quad(p, dir, qq, 0.001f, kInfF, t, a, b)) return 0.f;
    float ct = fabsf(dot(f3(qq[3]), -dir));
    if (ct < 1e-8f) return 0.f;
    return (1.0f / L.area) * t * t / ct;
  }
  if (L.kind == kLightSphere) {
    float4 S = make_float4(L.pos.x, L.pos.y, L.pos.z, L.radius);
    float t;
    if (!hit_sphere(p, dir, S, 0.001f, kInfF, t)) return 0.f;
    float dc = length(f3(S) - p);
    if (dc <= S.w) return 1.0f / (4.f * kPi * S.w * S.w);
    float sinMax = S.w / dc;
    float cosMax = sqrtf(fmaxf(0.f, 1.f - sinMax * sinMax));
    return 1.0f / (2.f * kPi * (1.f - cosMax));
  }
  if (L.kind == kLightDisc || L.kind == kLightDiscSpot) {  // disc_light.go:78-100
    const float4* Q = sc.quadrics + (size_t)L.prim * 5;
    float t, part;
    if (!hit_quadric(p, dir, Q, [](const float4* x) { return __ldg(x); }, 0.001f, kInfF, t, part)) return 0.f;
    float ct = fabsf(dot(f3(__ldg(Q + 1)), -dir));
    if (ct < 1e-6f) return 0.f;
    return (1.0f / L.area) * t * t / ct;
  }
  if (L.kind == kLightPointSpot) {  // point_spot_light.go:101-118
    float3 to = L.pos - p;
    float len = length(to);
    if (len == 0.f) return 0.f;
    return dot(dir, to * (1.0f / len)) > 0.999f ? 1.f : 0.f;
  }
  float c = dot(dir, n);
  return c <= 0.f ? 0.f : c / kPi;
}

// CalculateLightPDF (pkg/lights/light_sampling.go:11-26): sum over ALL lights
__device__ __forceinline__ float total_light_pdf(const DevScene& sc, float3 p, float3 n, float3 dir) {
  float total = 0.f;
  for (int i = 0; i < sc.n_lights; i++) {
    DevLight L = sc.lights[i];
    total += light_pdf(sc, L, p, n, dir) * L.prob;
  }
  return total;
}

// WeightedLightSampler.SampleLight (weighted_light_sampler.go:82-100)
__device__ __forceinline__ int pick_light(const DevScene& sc, float u) {
  float cum = 0.f;
  for (int i = 0; i < sc.n_lights; i++) {
    cum += sc.lights[i].prob;
    if (u <= cum) return i;
  }
  return sc.n_lights - 1;
}

// Sum of Light.Emit over the infinite lights for a missed ray
// (path_tracing.go:51-59, bdpt.go:214-229)
__device__ __forceinline__ float3 background(const DevScene& sc, float3 d) {
  float3 e = f3(0.f, 0.f, 0.f);
  if (!sc.has_infinite) return e;
  float3 dn = normalize_xy(d);
  for (int i = 0; i < sc.n_lights; i++) {
    DevLight L = sc.lights[i];
    if (L.kind == kLightUniformInfinite) e += L.a;
    else if (L.kind == kLightGradientInfinite) e += gradient_emission(L, dn);
  }
  return e;
}

// powerHeuristic (path_tracing.go:225-235)
__device__ __forceinline__ float power_heuristic(float f, float g) {
  if (f == 0.f) return 0.f;
  const float ff = __fmul_rn(f, f);  // roundings spelled out, as normalize_xy
  return __fdiv_rn(ff, __fmaf_rn(g, g, ff));
}

// ----------------------------------------------------------------- camera
// Camera.GetRay (pkg/geometry/camera.go:173-190)
// `yx` as in surface_at.
__device__ __forceinline__ void camera_ray(const DevCamera& c, int i, int j, float2 lens, float2 jit, float3& o,
                                           float3& d, bool yx) {
  float3 ps = c.pixel00 + c.du * ((float)i + (jit.x - 0.5f)) + c.dv * ((float)j + (jit.y - 0.5f));
  o = c.center;
  if (c.has_lens) {
    float2 p = sample_unit_disk(lens);
    o = c.center + c.disk_u * p.x + c.disk_v * p.y;
  }
  d = yx ? normalize_yx(ps - o) : normalize_xy(ps - o);
}

}  // namespace gprt
