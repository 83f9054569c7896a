// Record producer: the reference's path tracer (shader/src/path_tracer.comp)
// over a BVH built on the GPU. Host code (build, launch) and kernels.
//
// This file is compiled with -fmad=false: every multiply and add below is a
// separate IEEE operation unless written as fmaf, so the CPU oracle
// (oracle/nrc_trace_oracle.c), which repeats each expression in the same order
// with contraction off, produces the same floats. For the same reason the
// transcendental functions are this file's own (their methods are named where
// they are defined) rather than CUDA's, and a hit at equal distance from two
// triangles goes to the lower triangle index.
#include <cub/device/device_radix_sort.cuh>

#include <cmath>
#include <new>
#include <utility>
#include <vector>

#include "nrc_common.cuh"
#include "nrc_kernels.h"

// A four-wide node: for each axis the low and the high planes of its four slots,
// so that a ray loads its near and far planes as two 16-byte words chosen by the
// sign of its direction. 128 bytes, one cache line.
struct __align__(128) WideNode {
  float4 plane[6];  // low x, high x, low y, high y, low z, high z; an empty slot's low planes above its high ones
  uint32_t node0;   // first child node
  uint32_t tri0;    // first triangle (in the leaf array)
  // bit 24 + s: slot s holds a node; bits 3s .. 3s+2: the triangles (at most
  // three) of slot s. Nodes and triangles are stored in the order of those bits.
  uint32_t contents;
  uint32_t unused[5];
};
static_assert(sizeof(WideNode) == 128, "one cache line");

struct nrc_bvh {
  int device = 0;
  uint32_t tris = 0, nodes = 0;
  void* block = nullptr;          // the four arrays below
  const uint2* id = nullptr;      // primitive and instance per triangle
  const float4* guard = nullptr;  // 2 x float4 per triangle: lo.xyz, hi.xyz of its guard box
  const float4* leaf = nullptr;   // 3 x float4 per triangle in tree order: v0.xyz triangle, (v1 - v0).xyz, (v2 - v0).xyz
  const WideNode* wide = nullptr;
};

namespace nrc {
namespace {

constexpr float kPi = 3.14159265358979323846f;
constexpr int kMaxBounce = 8;            // path_tracer.comp:11
constexpr float kTMin = 1e-6f, kTMax = 4.0f;  // path_tracer.comp:12-13
constexpr float kC = 0.01f;                   // path_tracer.comp:14
constexpr float kConstLight = 10.0f;          // path_tracer.comp:145

// ------------------------------------------------------------------ math --
struct V3 {
  float x, y, z;
};
__device__ __forceinline__ V3 v3(float x, float y, float z) { return V3{x, y, z}; }
__device__ __forceinline__ V3 add(V3 a, V3 b) { return v3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ V3 sub(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ V3 mul(V3 a, V3 b) { return v3(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ V3 scale(V3 a, float s) { return v3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ V3 divs(V3 a, float s) { return v3(a.x / s, a.y / s, a.z / s); }
__device__ __forceinline__ V3 neg(V3 a) { return v3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross(V3 a, V3 b) {
  return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ V3 normalize(V3 a) { return scale(a, 1.0f / sqrtf(dot(a, a))); }

// Natural logarithm: x = m 2^e with m in [1/sqrt(2), sqrt(2)), log m = 2 atanh(s),
// s = (m - 1) / (m + 1), by the odd series of atanh to s^15; e ln 2 in two parts.
__device__ float t_log(float x) {
  if (x != x || x < 0.0f) return __int_as_float(0x7FC00000);
  if (x == 0.0f) return -__int_as_float(0x7F800000);
  if (x == __int_as_float(0x7F800000)) return x;
  int bits = __float_as_int(x);
  int e = ((bits >> 23) & 0xFF) - 127;
  float m = __int_as_float((bits & 0x007FFFFF) | 0x3F800000);  // [1, 2)
  if (m > 1.41421356f) {
    m = m * 0.5f;
    e = e + 1;
  }
  const float s = (m - 1.0f) / (m + 1.0f), s2 = s * s;
  float p = 1.0f / 15.0f;
  p = fmaf(p, s2, 1.0f / 13.0f);
  p = fmaf(p, s2, 1.0f / 11.0f);
  p = fmaf(p, s2, 1.0f / 9.0f);
  p = fmaf(p, s2, 1.0f / 7.0f);
  p = fmaf(p, s2, 1.0f / 5.0f);
  p = fmaf(p, s2, 1.0f / 3.0f);
  p = fmaf(p, s2, 1.0f);
  const float ef = static_cast<float>(e);
  return fmaf(ef, 0.693145751953125f, fmaf(ef, 1.42860677e-06f, 2.0f * s * p));
}

// sin and cos of 2 pi u: t = 4u = k + f with k = rint(t) (exact) and |f| <= 1/2,
// theta = f pi/2 in [-pi/4, pi/4]; Taylor series of sin to theta^9 and cos to
// theta^10, then the quadrant k mod 4.
__device__ void t_sincos_turns(float u, float& so, float& co) {
  const float t = 4.0f * u;
  const float k = rintf(t);
  const float th = (t - k) * 1.57079637f;
  const float t2 = th * th;
  float sp = 1.0f / 362880.0f;
  sp = fmaf(sp, t2, -1.0f / 5040.0f);
  sp = fmaf(sp, t2, 1.0f / 120.0f);
  sp = fmaf(sp, t2, -1.0f / 6.0f);
  sp = fmaf(sp, t2, 1.0f);
  const float sn = th * sp;
  float cp = -1.0f / 3628800.0f;
  cp = fmaf(cp, t2, 1.0f / 40320.0f);
  cp = fmaf(cp, t2, -1.0f / 720.0f);
  cp = fmaf(cp, t2, 1.0f / 24.0f);
  cp = fmaf(cp, t2, -0.5f);
  const float cs = fmaf(cp, t2, 1.0f);
  const int q = static_cast<int>(k) & 3;
  so = q == 0 ? sn : q == 1 ? cs : q == 2 ? -sn : -cs;
  co = q == 0 ? cs : q == 1 ? -sn : q == 2 ? -cs : sn;
}

// atan on [0, 1]: atan z = pi/6 + atan((z sqrt3 - 1) / (z + sqrt3)) above tan(pi/12),
// then the odd Taylor series to z^13.
__device__ float t_atan_unit(float z) {
  const bool shift = z > 0.267949194f;
  if (shift) z = (z * 1.73205081f - 1.0f) / (z + 1.73205081f);
  const float z2 = z * z;
  float p = 1.0f / 13.0f;
  p = fmaf(p, z2, -1.0f / 11.0f);
  p = fmaf(p, z2, 1.0f / 9.0f);
  p = fmaf(p, z2, -1.0f / 7.0f);
  p = fmaf(p, z2, 1.0f / 5.0f);
  p = fmaf(p, z2, -1.0f / 3.0f);
  p = fmaf(p, z2, 1.0f);
  const float a = z * p;
  return shift ? a + 0.523598790f : a;
}

__device__ float t_atan2(float y, float x) {
  const float ax = fabsf(x), ay = fabsf(y);
  if (ax == 0.0f && ay == 0.0f) return 0.0f;
  const bool low = ay <= ax;
  float a = t_atan_unit((low ? ay : ax) / (low ? ax : ay));
  if (!low) a = 1.57079637f - a;
  if (x < 0.0f) a = kPi - a;
  return y < 0.0f ? -a : a;
}

__device__ float t_acos(float x) { return t_atan2(sqrtf((1.0f - x) * (1.0f + x)), x); }

// e^x: Cody-Waite reduction and the degree-7 Taylor polynomial (as the encoding's)
__device__ float t_exp(float x) {
  x = fminf(fmaxf(x, -87.0f), 88.0f);
  const float k = rintf(x * 1.44269504f);
  float r = fmaf(k, -0.693145751953125f, x);
  r = fmaf(k, -1.42860677e-06f, r);
  float p = 1.98412698e-04f;
  p = fmaf(p, r, 1.38888889e-03f);
  p = fmaf(p, r, 8.33333333e-03f);
  p = fmaf(p, r, 4.16666667e-02f);
  p = fmaf(p, r, 1.66666667e-01f);
  p = fmaf(p, r, 0.5f);
  p = fmaf(p, r, 1.0f);
  p = fmaf(p, r, 1.0f);
  return p * __int_as_float((static_cast<int>(k) + 127) << 23);
}

// ------------------------------------------------------------------- rng --
// RNG.glsl:6-13: a condensed PCG (rxs-m-xs) step, then word / (2^32 - 1).
struct Rng {
  uint32_t s;
  __device__ float next() {
    s = s * 747796405u + 1u;
    uint32_t w = ((s >> ((s >> 28) + 4u)) ^ s) * 277803737u;
    w = (w >> 22) ^ w;
    return static_cast<float>(w) / 4294967295.0f;
  }
};

// ------------------------------------------------------------------ brdf --
// CookTorranceBRDF.glsl: Beckmann distribution, Walter's G1 approximation,
// Schlick's Fresnel, specular/diffuse lobe choice by luminance.
struct Brdf {
  V3 diffuse, specular;
  float roughness, ior;
};

__device__ __forceinline__ float ct_lum(V3 c) { return 0.212671f * c.x + 0.715160f * c.y + 0.072169f * c.z; }
__device__ __forceinline__ float ct_spec_prob(const Brdf& b) {
  const float dl = ct_lum(b.diffuse), sl = ct_lum(b.specular);
  return sl / (dl + sl);
}
__device__ float walter_g1(float v_dot_h, float v_dot_n, float ab2) {
  const float vn2 = v_dot_n * v_dot_n;
  const float a2 = 1.0f / (ab2 * (1.0f - vn2) / vn2), a = sqrtf(a2);
  return fmaxf(v_dot_h / v_dot_n, 0.0f) *
         (a >= 1.6f ? 1.0f : (3.535f * a + 2.181f * a2) / (1.0f + 2.276f * a + 2.577f * a2));
}
__device__ float beckmann_d(float n_dot_h, float a2) {
  const float nh2 = n_dot_h * n_dot_h, nh4 = nh2 * nh2;
  return t_exp((nh2 - 1.0f) / (a2 * nh2)) / (kPi * a2 * nh4);
}
__device__ float schlick(float v_dot_h, float ior) {
  float f0 = (ior - 1.0f) / (ior + 1.0f);
  f0 = f0 * f0;
  const float x = 1.0f - v_dot_h, x2 = x * x;
  return f0 + (1.0f - f0) * (x2 * x2 * x);
}
// AlignDir (Sample.glsl:7-11)
__device__ V3 align_dir(V3 n, V3 d) {
  const V3 u = normalize(cross(fabsf(n.x) > 0.01f ? v3(0.f, 1.f, 0.f) : v3(1.f, 0.f, 0.f), n));
  const V3 v = cross(n, u);
  return add(add(scale(u, d.x), scale(v, d.y)), scale(n, d.z));
}
// The BRDF's value and the sampling density of l (CookTorranceEval and
// CookTorrancePdf), which share the half vector, its cosines and, unless n.h is
// clamped, the distribution. `w` is ct_spec_prob(b).
__device__ V3 ct_eval_pdf(const Brdf& b, V3 l, V3 v, V3 n, float w, float& pdf) {
  const V3 h = normalize(add(l, v));
  const float nl = dot(n, l), nh = dot(n, h), vh = dot(v, h);
  const float n_dot_h = fmaxf(nh, 1e-8f);
  const float v_dot_h = fmaxf(vh, 1e-8f), l_dot_h = v_dot_h;
  const float n_dot_l = fminf(fmaxf(nl, 1e-8f), 1.0f - 1e-8f);
  const float n_dot_v = fminf(fmaxf(dot(n, v), 1e-8f), 1.0f - 1e-8f);
  const float a = b.roughness, a2 = a * a;
  const float G = walter_g1(v_dot_h, n_dot_v, a2) * walter_g1(l_dot_h, n_dot_l, a2);
  const float D = beckmann_d(n_dot_h, a2);
  const float F = schlick(v_dot_h, b.ior);
  pdf = 0.0f;
  if (!(nl < 0.0f)) {
    const float p_h = (nh == n_dot_h ? D : beckmann_d(nh, a2)) * nh;
    const float p_ct = p_h / (4.0f * vh);
    const float p_l = nl / kPi;
    pdf = p_l * (1.0f - w) + p_ct * w;  // mix(p_lambert, p_cook_torrance, w)
  }
  // specular * D * G * F / (4 n.l n.v), left to right per channel; diffuse / pi
  const V3 spec = divs(scale(scale(scale(b.specular, D), G), F), 4.0f * n_dot_l * n_dot_v);
  return add(divs(b.diffuse, kPi), spec);
}
// CookTorranceSample: returns the incident direction; pdf via ct_eval_pdf. The half
// vector of the specular lobe and the cosine-weighted direction of the diffuse one
// (Sample.glsl:13-20) are the same steps from a radius, an angle and a height, so
// the lanes of either lobe take them together.
__device__ V3 ct_sample(const Brdf& b, V3 v, V3 n, float w, Rng& rng) {
  const float u1 = rng.next(), u2 = rng.next();
  const bool diffuse = rng.next() > w;
  float r, z, turn;
  if (diffuse) {
    const float c1 = rng.next();
    turn = rng.next();
    r = sqrtf(c1);
    z = sqrtf(1.0f - c1);
  } else {
    const float a = b.roughness, a2 = a * a;
    float tan2 = -a2 * t_log(1.0f - u1);
    if (tan2 != tan2) tan2 = 0.0f;
    z = sqrtf(1.0f / (1.0f + tan2));
    r = sqrtf(1.0f - z * z);
    turn = u2;
  }
  float s, c;
  t_sincos_turns(turn, s, c);
  const V3 d = align_dir(n, v3(r * c, r * s, z));
  if (diffuse) return d;
  const V3 h = dot(v, d) < 0.0f ? neg(d) : d;
  // reflect(-v, h) = -v - 2 dot(h, -v) h
  const V3 iv = neg(v);
  return sub(iv, scale(h, 2.0f * dot(h, iv)));
}

__device__ __forceinline__ V3 normalize_rgb(V3 c) {  // NormalizeRGB, path_tracer.comp:147
  const bool bad = c.x != c.x || c.y != c.y || c.z != c.z || fabsf(c.x) == __int_as_float(0x7F800000) ||
                   fabsf(c.y) == __int_as_float(0x7F800000) || fabsf(c.z) == __int_as_float(0x7F800000);
  return bad ? v3(0.f, 0.f, 0.f) : v3(fmaxf(c.x, 0.f), fmaxf(c.y, 0.f), fmaxf(c.z, 0.f));
}

// ----------------------------------------------------------------- scene --
struct TraceScene {
  nrc_scene s;
  float lut[256];  // sRGB -> linear (texels decoded before filtering)
};

__device__ V3 xform(const float* T, V3 p) {  // vec4(p, 1) * mat3x4
  return v3(p.x * T[0] + p.y * T[1] + p.z * T[2] + T[3], p.x * T[4] + p.y * T[5] + p.z * T[6] + T[7],
            p.x * T[8] + p.y * T[9] + p.z * T[10] + T[11]);
}

__device__ V3 scene_vertex(const nrc_scene& S, uint32_t inst, uint32_t prim, int k) {
  const float* p = S.vertices + size_t(S.vertex_indices[size_t(prim) * 3 + k]) * 3;
  return xform(S.transforms + size_t(inst) * 12, v3(p[0], p[1], p[2]));
}

__device__ float lerpf(float a, float b, float t) { return a + (b - a) * t; }

__device__ uint32_t wrap_idx(float f, uint32_t n) {
  if ((n & (n - 1u)) == 0u) return static_cast<uint32_t>(static_cast<int>(f)) & (n - 1u);  // the same, f being integral
  const float nf = static_cast<float>(n);
  int r = static_cast<int>(f - nf * floorf(f / nf));
  if (r < 0) r += static_cast<int>(n);
  if (r >= static_cast<int>(n)) r -= static_cast<int>(n);
  return static_cast<uint32_t>(r);
}

__device__ V3 tex_sample(const nrc_texture& t, float tu, float tv, const float* lut) {
  const uint32_t w = t.width, h = t.height;
  if (w == 0 || h == 0 || t.texels == nullptr) return v3(0.f, 0.f, 0.f);
  float u = tu * static_cast<float>(w) - 0.5f, v = tv * static_cast<float>(h) - 0.5f;
  if (!(fabsf(u) < 8388608.0f)) u = 0.0f;
  if (!(fabsf(v) < 8388608.0f)) v = 0.0f;
  const float fu = floorf(u), fv = floorf(v), a = u - fu, b = v - fv;
  const uint32_t i0 = wrap_idx(fu, w), j0 = wrap_idx(fv, h);
  const uint32_t i1 = i0 + 1 == w ? 0 : i0 + 1, j1 = j0 + 1 == h ? 0 : j0 + 1;
  const uchar4* px = reinterpret_cast<const uchar4*>(t.texels);
  const uchar4 t00 = px[size_t(j0) * w + i0], t10 = px[size_t(j0) * w + i1];
  const uchar4 t01 = px[size_t(j1) * w + i0], t11 = px[size_t(j1) * w + i1];
  auto ch = [&](unsigned char c00, unsigned char c10, unsigned char c01, unsigned char c11) {
    return lerpf(lerpf(lut[c00], lut[c10], a), lerpf(lut[c01], lut[c11], a), b);
  };
  return v3(ch(t00.x, t10.x, t01.x, t11.x), ch(t00.y, t10.y, t01.y, t11.y), ch(t00.z, t10.z, t01.z, t11.z));
}

__device__ V3 mat_color(const nrc_scene& S, const float* konst, uint32_t id, float tu, float tv, const float* lut) {
  if (id != 0xFFFFFFFFu && id < S.texture_count) return tex_sample(S.textures[id], tu, tv, lut);
  return v3(konst[0], konst[1], konst[2]);
}

struct Hit {
  V3 position, normal, diffuse, specular, emission;
  float bu, bv;  // barycentrics of vertices 1 and 2
  float roughness, ior;
  uint32_t prim, inst;
  bool flip;
};

struct Ray {
  V3 o, d;
};

// The hit record of (prim, inst) with barycentrics (bu, bv): GetRayQueryHit /
// GetVBufferHit (path_tracer.comp:66-131) after their barycentrics.
__device__ Hit make_hit(const nrc_scene& S, const float* lut, uint32_t prim, uint32_t inst, float bu, float bv,
                        V3 v0, V3 v1, V3 v2, V3 n_unnorm, Ray ray) {
  Hit h;
  const V3 n = normalize(n_unnorm);
  h.flip = dot(n, ray.d) >= 0.0f;
  h.normal = h.flip ? neg(n) : n;
  h.prim = prim;
  h.inst = inst;
  h.bu = bu;
  h.bv = bv;
  const float b0 = 1.0f - bu - bv;
  h.position = add(add(scale(v0, b0), scale(v1, bu)), scale(v2, bv));
  const float* t0 = S.texcoords + size_t(S.texcoord_indices[size_t(prim) * 3 + 0]) * 2;
  const float* t1 = S.texcoords + size_t(S.texcoord_indices[size_t(prim) * 3 + 1]) * 2;
  const float* t2 = S.texcoords + size_t(S.texcoord_indices[size_t(prim) * 3 + 2]) * 2;
  const float tu = t0[0] * b0 + t1[0] * bu + t2[0] * bv, tv = t0[1] * b0 + t1[1] * bu + t2[1] * bv;
  const nrc_material& m = S.materials[S.material_ids[prim]];
  h.diffuse = mat_color(S, m.diffuse, m.diffuse_texture_id, tu, tv, lut);
  h.specular = mat_color(S, m.specular, m.specular_texture_id, tu, tv, lut);
  h.emission = mat_color(S, m.emission, m.emission_texture_id, tu, tv, lut);
  h.roughness = m.roughness;
  h.ior = m.ior;
  return h;
}

// ------------------------------------------------------------- bvh trace --
struct TriView {
  const uint2* id;
  const float4* guard;
  const float4* leaf;
  const WideNode* wide;
  uint32_t tris;
};

// A traversal stacks at most one entry per level of the wide tree, which has at
// most as many as the binary tree under it is high: kMaxHeight, and the passes that
// halve what is left of fewer than 2^30 clusters, at most 30 (see cluster_kernel).
constexpr uint32_t kMaxHeight = 48;
constexpr int kStack = kMaxHeight + 32;

// Moller-Trumbore: t and barycentrics (u: vertex 1, v: vertex 2) when the ray
// meets the triangle with t in [tmin, tmax].
__device__ __forceinline__ bool intersect(float4 a, float4 b, float4 c, Ray r, float tmin, float tmax, float& t, float& u,
                                          float& v) {
  const V3 v0 = v3(a.x, a.y, a.z), e1 = v3(b.x, b.y, b.z), e2 = v3(c.x, c.y, c.z);
  const V3 p = cross(r.d, e2);
  const float det = dot(e1, p);
  if (det == 0.0f || det != det) return false;
  const float inv = 1.0f / det;
  const V3 s = sub(r.o, v0);
  u = dot(s, p) * inv;
  if (!(u >= 0.0f && u <= 1.0f)) return false;
  const V3 q = cross(s, e1);
  v = dot(r.d, q) * inv;
  if (!(v >= 0.0f && u + v <= 1.0f)) return false;
  t = dot(e2, q) * inv;
  return t >= tmin && t <= tmax;
}

// Slab test of a triangle's guard box, which depends on the triangle alone. The
// triangle test's rounding can accept a point off the triangle; a hit counts only if
// the ray meets this box. The boxes of the wide tree contain the guard boxes of what
// is below them, and their slab test allows for more rounding than this one, so which
// triangles a ray can hit does not depend on how the tree groups them. (What a tree's
// order can still decide, as in any tree: a distance that rounding makes shorter than
// the way to the guard box by over 1e-4 of it, slivers only, is passed by once a
// nearer hit is known.)
__device__ __forceinline__ bool guard_hit(float4 lo, float4 hi, V3 o, float ix, float iy, float iz, float tmin,
                                          float tmax) {
  const float x0 = (lo.x - o.x) * ix, x1 = (hi.x - o.x) * ix;
  const float y0 = (lo.y - o.y) * iy, y1 = (hi.y - o.y) * iy;
  const float z0 = (lo.z - o.z) * iz, z1 = (hi.z - o.z) * iz;
  const float tn = fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fmaxf(fminf(z0, z1), tmin));
  const float tf = fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fminf(fmaxf(z0, z1), tmax));
  return tn <= tf * 1.00001f + 1e-7f;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// A ray's offset in the slab test of an axis, coordinate p being met at p * i + o. Where
// it overflows it is NaN, which max3 and min3 pass over: the axis then excludes no box.
__device__ __forceinline__ float slab_offset(float origin, float i) {
  const float o = -origin * i;
  return fabsf(o) < __int_as_float(0x7F800000) ? o : __int_as_float(0x7FC00000);
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Closest triangle along the ray in [tmin, tmax]; equal distances go to the lower
// triangle index. Returns the triangle index or -1. Kept out of line, which
// keeps its registers apart from the shading's (inlined: 1.73 against 1.68 ms).
// The lanes that call together step together: each iteration is one node for
// every lane with a node to visit, or one triangle test for every lane with
// triangles pending, chosen so that steps run with many lanes. A lane goes on
// visiting nodes until the triangles of two nodes are pending.
// Bound by instruction issue at the warp's lane count (ncu, 587,534 triangles,
// 8-bounce paths at 960 x 540: issue slots 62%, ALU pipe 62%, 12.4 of 32 lanes; L1
// wavefronts 48%): 12 nodes and 4.7 triangles a ray. That launch takes 1.67 ms; the
// binary radix tree with freely diverging lanes took 3.18 ms (6 lanes), this loop
// over eight-wide nodes of 8-bit planes 2.25, over four-wide ones 1.88 (unpacking
// the bytes loads the half-rate ALU pipe more than fp32 planes load L1). Lanes that
// finish early and shade while the others go on walking made it slower (1.95 ms):
// the shading, a third of the instructions, then runs more often with fewer lanes.
__device__ __noinline__ int trace_closest(const TriView B, Ray r, float tmin, float tmax, float& bt_out, float& bu,
                                          float& bv) {
  if (B.tris == 0) return -1;
  const float ix = fabsf(r.d.x) > 1e-20f ? 1.0f / r.d.x : copysignf(1e20f, r.d.x);
  const float iy = fabsf(r.d.y) > 1e-20f ? 1.0f / r.d.y : copysignf(1e20f, r.d.y);
  const float iz = fabsf(r.d.z) > 1e-20f ? 1.0f / r.d.z : copysignf(1e20f, r.d.z);
  const float ox = slab_offset(r.o.x, ix), oy = slab_offset(r.o.y, iy), oz = slab_offset(r.o.z, iz);
  const int sx = ix >= 0.0f ? 0 : 1, sy = iy >= 0.0f ? 0 : 1, sz = iz >= 0.0f ? 0 : 1;  // which of the planes is near
  // A ray with a NaN or an infinity meets nothing (every comparison of the triangle test fails).
  const float sum = (r.o.x + r.o.y + r.o.z) + (r.d.x + r.d.y + r.d.z);
  const float most = fmaxf(max3(fabsf(r.o.x), fabsf(r.o.y), fabsf(r.o.z)), max3(fabsf(r.d.x), fabsf(r.d.y), fabsf(r.d.z)));
  const bool finite = sum == sum && most < __int_as_float(0x7F800000);
  constexpr uint32_t kRoot = (1u << 24) | 1u;
  int best = -1;
  float bt = tmax;
  // A group of sibling nodes: the first one, and a word with the slots still to
  // visit (bits 24..27), the nearest of them when the group was met (bits 8, 9)
  // and the slots holding nodes (bits 0..3). The root is slot 0 of its own group.
  uint2 stack[kStack];
  int sp = 0;
  uint32_t base = 0, group = finite ? kRoot : 0u;
  uint32_t tri0 = 0, tset = 0, tri1 = 0, tset1 = 0;  // pending triangles of two nodes: first, present << 12 | hit
  bool strict = false;  // test the guard box of every hit, not only of the closest
  const uint32_t lanes = __activemask();
  while (true) {
    const bool has_tri = tset != 0u, has_node = group >= (1u << 24) && tset1 == 0u;
    const uint32_t want_tri = __ballot_sync(lanes, has_tri), want_node = __ballot_sync(lanes, has_node);
    if ((want_tri | want_node) == 0u) {
      // the closest hit counts if it meets its guard box; if not (a grazing
      // ray, rarely), the lane starts again, testing every hit's
      const bool again = best >= 0 && !strict &&
                         !guard_hit(__ldg(B.guard + size_t(best) * 2), __ldg(B.guard + size_t(best) * 2 + 1), r.o, ix, iy,
                                    iz, tmin, tmax);
      if (__ballot_sync(lanes, again) == 0u) break;
      if (again) {
        strict = true;
        best = -1;
        bt = tmax;
        base = 0u;
        group = kRoot;
      }
      continue;
    }
    if (want_node == 0u || 3 * __popc(want_tri) >= 2 * __popc(want_tri | want_node)) {
      if (has_tri) {
        const uint32_t bit = tset & (0u - tset);
        const float4* T = B.leaf + size_t(tri0 + __popc((tset >> 12) & (bit - 1u))) * 3;
        const float4 a = __ldg(T), b = __ldg(T + 1), c = __ldg(T + 2);
        tset ^= bit;
        if ((tset & 0xFFFu) == 0u) {
          tri0 = tri1;
          tset = tset1;
          tset1 = 0u;
        }
        const int ti = __float_as_int(a.w);
        float t, u, v;
        if (intersect(a, b, c, r, tmin, bt, t, u, v) && (t < bt || best < 0 || ti < best) &&
            (!strict || guard_hit(__ldg(B.guard + size_t(ti) * 2), __ldg(B.guard + size_t(ti) * 2 + 1), r.o, ix, iy, iz, tmin,
                                  tmax))) {
          best = ti;
          bt = t;
          bu = u;
          bv = v;
        }
      }
    } else if (has_node) {
      uint32_t bit = group & (1u << (24u + ((group >> 8) & 3u)));
      const uint32_t left = group & 0x0F000000u;
      bit = bit != 0u ? bit : left & (0u - left);
      group ^= bit;
      const WideNode* N = B.wide + (base + __popc(group & ((bit >> 24) - 1u)));
      const float4 nx = __ldg(N->plane + sx), fx = __ldg(N->plane + (1 - sx)), ny = __ldg(N->plane + 2 + sy),
                   fy = __ldg(N->plane + (3 - sy)), nz = __ldg(N->plane + 4 + sz), fz = __ldg(N->plane + (5 - sz));
      const uint4 m = __ldg(reinterpret_cast<const uint4*>(&N->node0));
      uint32_t hit = 0, near = 0xFFFFFFFFu;
      auto slot = [&](float x0, float y0, float z0, float x1, float y1, float z1, uint32_t s) {
        const float tn = fmaxf(max3(fmaf(x0, ix, ox), fmaf(y0, iy, oy), fmaf(z0, iz, oz)), tmin);
        const float tf = fminf(min3(fmaf(x1, ix, ox), fmaf(y1, iy, oy), fmaf(z1, iz, oz)), bt);
        const bool in = tn <= fmaf(tf, 1.0001f, 1e-6f);
        hit |= in ? (7u << (3 * s)) | (1u << (24 + s)) : 0u;
        near = min(near, in ? (__float_as_uint(tn) & ~3u) | s : 0xFFFFFFFFu);  // tn >= 0: its bits are ordered
      };
      slot(nx.x, ny.x, nz.x, fx.x, fy.x, fz.x, 0);
      slot(nx.y, ny.y, nz.y, fx.y, fy.y, fz.y, 1);
      slot(nx.z, ny.z, nz.z, fx.z, fy.z, fz.z, 2);
      slot(nx.w, ny.w, nz.w, fx.w, fy.w, fz.w, 3);
      hit &= m.z;
      const uint32_t set = (hit & 0xFFFu) != 0u ? ((m.z & 0xFFFu) << 12) | (hit & 0xFFFu) : 0u;
      const bool first = tset == 0u;
      tri1 = first ? tri1 : m.y;
      tset1 = first ? 0u : set;
      tri0 = first ? m.y : tri0;
      tset = first ? set : tset;
      // down into the children met; else on to the siblings left, else to the last group stacked
      const uint32_t below = (hit & 0x0F000000u) | (m.z >> 24) | ((near & 3u) << 8);
      const bool down = below >= (1u << 24), rest = group >= (1u << 24);
      if (down && rest) stack[sp++] = make_uint2(base, group);
      if (!down && !rest && sp > 0) {
        const uint2 e = stack[--sp];
        base = e.x;
        group = e.y;
      }
      base = down ? m.x : base;
      group = down ? below : group;
    }
  }
  bt_out = bt;
  return best;
}

// --------------------------------------------------------------- records --
__device__ uint32_t pack_unorm2x16(float a, float b) {
  const float ca = fminf(fmaxf(a, 0.0f), 1.0f), cb = fminf(fmaxf(b, 0.0f), 1.0f);
  return static_cast<uint32_t>(rintf(ca * 65535.0f)) | (static_cast<uint32_t>(rintf(cb * 65535.0f)) << 16);
}

__device__ void sph_encode(V3 d, float& u, float& v) {  // NRCSphEncode with this file's atan2 / acos
  u = (d.x == 0.0f && d.y == 0.0f) ? 0.5f : 0.5f + t_atan2(d.y, d.x) / (2.0f * kPi);
  v = t_acos(fminf(fmaxf(d.z, -1.0f), 1.0f)) / kPi;
}

__device__ nrc_packed_input make_input(const Hit& h, V3 d) {  // MakeNRCInput, path_tracer.comp:158-165
  nrc_packed_input i;
  i.primitive_id = h.prim;
  i.flip_bit_instance_id = h.inst | (h.flip ? 0x80000000u : 0u);
  i.barycentric_2x16u = pack_unorm2x16(h.bu, h.bv);
  float su, sv;
  sph_encode(d, su, sv);
  i.scattered_dir_2x16u = pack_unorm2x16(su, sv);
  return i;
}

struct Step {  // BRDFStepInfo
  V3 color;
  float cosine, pdf, dist2;
  Ray ray;
};

__device__ Step brdf_step(const Hit& h, Ray ray, Rng& rng) {  // BRDFStep, path_tracer.comp:167-186
  Brdf b{h.diffuse, h.specular, fmaxf(h.roughness, 0.001f), fmaxf(h.ior, 1.5f)};
  const V3 v = neg(ray.d);
  const float w = ct_spec_prob(b);
  const V3 dir = ct_sample(b, v, h.normal, w, rng);
  float pdf;
  const V3 f = ct_eval_pdf(b, dir, v, h.normal, w, pdf);
  const float cosine = fabsf(dot(h.normal, dir));
  Step s;
  s.color = normalize_rgb(divs(scale(f, cosine), pdf));  // brdf * cosine / pdf
  s.ray = Ray{h.position, dir};
  s.cosine = cosine;
  s.pdf = pdf;
  const V3 dd = sub(ray.o, h.position);
  s.dist2 = dot(dd, dd);
  return s;
}

struct TraceArgs {
  TraceScene sc;
  TriView bvh;
  nrc_trace_params p;
  nrc_trace_targets t;
};

__device__ void push_eval(const TraceArgs& A, uint32_t dst, const nrc_packed_input& in) {
  const uint32_t id = atomicAdd(A.t.eval_count, 1u);
  if (id >= A.t.eval_capacity) return;
  uint32_t* w = reinterpret_cast<uint32_t*>(A.t.eval_records + id);
  w[0] = dst;
  w[1] = in.primitive_id;
  w[2] = in.flip_bit_instance_id;
  w[3] = in.barycentric_2x16u;
  w[4] = in.scattered_dir_2x16u;
}

__device__ __forceinline__ uint32_t dst_screen(uint32_t x, uint32_t y) { return (x | (y << 15)) << 1; }
__device__ __forceinline__ uint32_t dst_train(uint32_t b, uint32_t l, uint32_t r) {
  return ((b | (l << 2) | (r << 16)) << 1) | 1u;
}

struct Result {
  V3 bias, factor;
};

// The path of one pixel from its camera ray: PathTrace (path_tracer.comp:208-250)
// or, for training pixels, ExtendedPathTrace (:252-375), which follows the path
// past the point where the screen's part of it ends (`suffix`) and writes train
// records. Both walk the same loop, so the kernel holds one copy of the hit
// record and the BRDF step: with a copy per call site its hot code did not fit
// the instruction cache. The method and `train` are warp-uniform.
__device__ __forceinline__ Result trace_path(const TraceArgs& A, const float* lut, Ray ray, uint32_t method, bool train, Rng& rng,
                             uint32_t x, uint32_t y) {
  V3 lights[kMaxBounce], colors[kMaxBounce];  // training: of the vertex after vertex i
  nrc_packed_input inputs[kMaxBounce];
  V3 radiance = v3(0.f, 0.f, 0.f), acc = v3(1.f, 1.f, 1.f);
  Result result;
  const nrc_scene& S = A.sc.s;
  float c_a0 = 0.0f, sqrt_a_sum = 0.0f;
  bool suffix = false, light_terminate = false;
  int bounce = 0;  // vertices so far
  Hit hit;
  while (true) {
    float t, u, v;
    const int ti = trace_closest(A.bvh, ray, bounce == 0 ? 0.0f : kTMin, bounce == 0 ? __int_as_float(0x7F800000) : kTMax,
                                 t, u, v);
    if (ti < 0) {
      if (bounce == 0) return Result{v3(kConstLight, kConstLight, kConstLight), v3(0.f, 0.f, 0.f)};
      if (!suffix) radiance = add(radiance, scale(acc, kConstLight));
      if (!train) return Result{radiance, acc};
      lights[bounce - 1] = v3(kConstLight, kConstLight, kConstLight);
      light_terminate = true;
    } else {
      const uint2 id = A.bvh.id[ti];
      const uint32_t prim = id.x, inst = id.y;
      const V3 v0 = scene_vertex(S, inst, prim, 0), v1 = scene_vertex(S, inst, prim, 1),
               v2 = scene_vertex(S, inst, prim, 2);
      const V3 v01 = sub(v1, v0), v02 = sub(v2, v0), n = cross(v01, v02);
      if (bounce == 0) {  // GetVBufferHit's barycentrics: the ray against the triangle's plane
        const V3 q = cross(sub(ray.o, v0), ray.d);
        const float d = 1.0f / dot(ray.d, n);
        u = d * dot(neg(q), v02);
        v = d * dot(q, v01);
      }
      hit = make_hit(S, lut, prim, inst, u, v, v0, v1, v2, n, ray);
      const Step info = brdf_step(hit, ray, rng);
      if (!suffix) {
        radiance = add(radiance, mul(acc, hit.emission));
        acc = mul(acc, info.color);
      }
      ray = info.ray;
      if (bounce == 0)
        c_a0 = method == NRC_METHOD_NONE ? __int_as_float(0x7F800000) : kC * info.dist2 / (4.0f * kPi * info.cosine);
      else
        sqrt_a_sum = sqrt_a_sum + sqrtf(info.dist2 / (info.pdf * info.cosine));
      if (train) {
        inputs[bounce] = make_input(hit, ray.d);
        lights[bounce] = v3(0.f, 0.f, 0.f);
        colors[bounce] = v3(1.f, 1.f, 1.f);
        if (bounce > 0) {
          lights[bounce - 1] = hit.emission;
          colors[bounce - 1] = info.color;
        }
      }
      if (bounce == 0) result = Result{radiance, acc};
      ++bounce;
    }
    // does the path go on? (a cache query ends the screen's part at the first vertex)
    const bool grow = !light_terminate && bounce < kMaxBounce && sqrt_a_sum * sqrt_a_sum <= c_a0;
    if (!train) {
      if (grow && method != NRC_METHOD_CACHE) continue;
      if (method != NRC_METHOD_NONE) push_eval(A, dst_screen(x, y), make_input(hit, ray.d));
      return Result{radiance, acc};
    }
    if (grow) continue;
    if (!suffix) {  // the screen's record; then the training suffix, its spread measured anew
      if (method == NRC_METHOD_CACHE) {
        push_eval(A, dst_screen(x, y), inputs[0]);
      } else {
        result = Result{radiance, acc};
        if (!light_terminate) push_eval(A, dst_screen(x, y), inputs[bounce - 1]);
      }
      suffix = true;
      sqrt_a_sum = 0.0f;
      if (!light_terminate && bounce < kMaxBounce && 0.0f <= c_a0) continue;
    }
    break;
  }
  // clamp(uint(u * 4), 0, 3) with u in [0, 1]
  uint32_t batch = static_cast<uint32_t>(rng.next() * static_cast<float>(NRC_TRAIN_BATCH_COUNT));
  batch = batch < NRC_TRAIN_BATCH_COUNT - 1 ? batch : NRC_TRAIN_BATCH_COUNT - 1;
  const uint32_t train_id = atomicAdd(A.t.train_counts[batch], static_cast<uint32_t>(bounce));
  if (train_id < NRC_TRAIN_BATCH_SIZE) {
    for (int i = bounce - 2; i >= 0; --i) {
      lights[i] = add(lights[i], mul(colors[i], lights[i + 1]));
      colors[i] = mul(colors[i], colors[i + 1]);
    }
    const uint32_t count = min(static_cast<uint32_t>(bounce), NRC_TRAIN_BATCH_SIZE - train_id);
    nrc_packed_train_record* rec = A.t.train_records[batch];
    for (uint32_t i = 0; i < count; ++i) {
      float* w = reinterpret_cast<float*>(rec + train_id + i);
      w[0] = lights[i].x;
      w[1] = lights[i].y;
      w[2] = lights[i].z;
      w[3] = colors[i].x;
      w[4] = colors[i].y;
      w[5] = colors[i].z;
      uint32_t* u = reinterpret_cast<uint32_t*>(w + 6);
      u[0] = inputs[i].primitive_id;
      u[1] = inputs[i].flip_bit_instance_id;
      u[2] = inputs[i].barycentric_2x16u;
      u[3] = inputs[i].scattered_dir_2x16u;
    }
    if (!light_terminate) push_eval(A, dst_train(batch, train_id, train_id + count - 1), inputs[bounce - 1]);
  }
  return result;
}

// main(), path_tracer.comp:377-420: 8 x 8 threads per block, warps of 32
// consecutive threads (4 rows), the warp standing in for the subgroup.
// 16 blocks of 64 threads per SM (64 registers): 12 blocks without spills and
// with the traversal inlined measured slower (1.85 against 1.68 ms for 8-bounce
// paths at 960 x 540, 1.83 against 1.70 ms for cache paths at 1920 x 1080; 2.72 ms
// over the binary tree). The shading's length counts twice, in issue slots and in
// instruction cache misses: one atan for either octant, one half vector and
// distribution for the BRDF's value and density and one direction for both lobes
// took the same launches from 1.66 and 1.70 to 1.60 and 1.55 ms.
__global__ void __launch_bounds__(64, 16) path_trace_kernel(const __grid_constant__ TraceArgs A) {
  extern __shared__ float lut_s[];
  for (int i = threadIdx.y * 8 + threadIdx.x; i < 256; i += 64) lut_s[i] = A.sc.lut[i];
  __syncthreads();
  const uint32_t x = blockIdx.x * 8 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
  Rng rng{(((y & 0xFFu) << 8) | (x & 0xFFu)) + A.p.seed};
  const bool inside = x < A.p.width && y < A.p.height;
  const uint32_t active = __ballot_sync(0xffffffffu, inside);
  if (!inside) return;
  const int lane = (threadIdx.y * 8 + threadIdx.x) & 31;
  const bool left_all = __all_sync(active, x <= A.p.width / 2);
  const uint32_t method = left_all ? A.p.left_method : A.p.right_method;
  bool train = false;
  if (method != NRC_METHOD_NONE) {
    const int first = __ffs(active) - 1;  // subgroupElect: the lowest active lane
    if (lane == first) train = rng.next() < A.p.train_probability;
    train = __shfl_sync(active, train ? 1 : 0, first) != 0;
  }
  // the camera ray (the primary hit replaces the V-buffer's primitive and instance)
  const float cx = (static_cast<float>(x) + 0.5f) / static_cast<float>(A.p.width) * 2.0f - 1.0f;
  const float cy = (static_cast<float>(y) + 0.5f) / static_cast<float>(A.p.height) * 2.0f - 1.0f;
  const V3 look = v3(A.p.look[0], A.p.look[1], A.p.look[2]), side = v3(A.p.side[0], A.p.side[1], A.p.side[2]),
           up = v3(A.p.up[0], A.p.up[1], A.p.up[2]);
  Ray ray{v3(A.p.origin[0], A.p.origin[1], A.p.origin[2]), normalize(add(add(look, scale(side, cx)), scale(up, cy)))};
  Result res = trace_path(A, lut_s, ray, method, train, rng, x, y);
  res.bias = normalize_rgb(res.bias);
  res.factor = normalize_rgb(res.factor);
  const size_t px = size_t(y) * A.p.width + x;
  reinterpret_cast<float4*>(A.t.bias_factor_r)[px] = make_float4(res.bias.x, res.bias.y, res.bias.z, res.factor.x);
  reinterpret_cast<float2*>(A.t.factor_gb)[px] = make_float2(res.factor.y, res.factor.z);
}

// ------------------------------------------------------------- bvh build --
struct BuildArgs {
  nrc_scene s;
  const nrc_instance_range* ranges;
  const uint32_t* first_tri;  // prefix sums of the ranges' counts (instances + 1)
  uint32_t instances, tris;
};

// World-space triangles, their scene ids and their centroids.
__global__ void tri_kernel(BuildArgs A, float4* tri, uint2* id, float* cent, uint32_t* bad) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A.tris) return;
  uint32_t lo = 0, hi = A.instances;  // instance i holds triangles [first_tri[i], first_tri[i+1])
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (A.first_tri[mid] <= t) lo = mid; else hi = mid;
  }
  const uint32_t inst = lo, prim = A.ranges[inst].first_primitive + (t - A.first_tri[inst]);
  const nrc_scene& S = A.s;
  V3 v[3] = {v3(0.f, 0.f, 0.f), v3(0.f, 0.f, 0.f), v3(0.f, 0.f, 0.f)};
  bool ok = prim < S.primitive_count;
  for (int k = 0; k < 3 && ok; ++k) {
    const uint32_t vi = S.vertex_indices[size_t(prim) * 3 + k];
    if (vi >= S.vertex_count) { ok = false; break; }
    v[k] = scene_vertex(S, inst, prim, k);
  }
  if (!ok) atomicOr(bad, 1u);
  id[t] = make_uint2(prim, inst);
  for (int k = 0; k < 3; ++k) tri[size_t(t) * 3 + k] = make_float4(v[k].x, v[k].y, v[k].z, 0.0f);
  cent[size_t(t) * 3 + 0] = (v[0].x + v[1].x + v[2].x) * (1.0f / 3.0f);
  cent[size_t(t) * 3 + 1] = (v[0].y + v[1].y + v[2].y) * (1.0f / 3.0f);
  cent[size_t(t) * 3 + 2] = (v[0].z + v[1].z + v[2].z) * (1.0f / 3.0f);
}

__device__ __forceinline__ uint32_t ordered(float f) {  // float -> uint32 preserving order
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

__global__ void bounds_kernel(const float* cent, uint32_t n, uint32_t* box) {  // box: min xyz, max xyz (ordered)
  uint32_t mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int k = 0; k < 3; ++k) {
      const uint32_t o = ordered(cent[size_t(i) * 3 + k]);
      mn[k] = min(mn[k], o);
      mx[k] = max(mx[k], o);
    }
  for (int k = 0; k < 3; ++k) {
    atomicMin(&box[k], mn[k]);
    atomicMax(&box[3 + k], mx[k]);
  }
}

__device__ __forceinline__ uint32_t spread10(uint32_t v) {  // 10 bits -> every third bit
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

__global__ void morton_kernel(const float* cent, uint32_t n, const uint32_t* box, uint32_t* keys, uint32_t* vals) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t code = 0;
  for (int k = 0; k < 3; ++k) {
    const float lo = unordered(box[k]), hi = unordered(box[3 + k]);
    const float ext = hi - lo;
    float f = ext > 0.0f ? (cent[size_t(i) * 3 + k] - lo) / ext : 0.5f;
    f = fminf(fmaxf(f, 0.0f), 1.0f);
    const uint32_t q = min(static_cast<uint32_t>(f * 1024.0f), 1023u);
    code |= spread10(q) << (2 - k);
  }
  keys[i] = code;
  vals[i] = i;
}

// Parallel locally-ordered clustering (Meister and Bittner 2018) over the
// triangles in Morton order: each cluster looks kSearch places to either side for
// the one whose union with it has the least area; pairs that choose each other
// merge; the survivors keep their order. Unlike a radix tree's, a triangle much
// larger than its neighbours (a wall beside a tessellated floor) joins late,
// near the root, instead of stretching the boxes of everything above a small one.
// It runs in stages, each one launch: a block takes kChunk places in a row through
// the passes (three or four) that leave kKeep clusters, the next stage's blocks take
// the survivors of kFan blocks each, and the last stage's one block goes on to a single
// cluster. No pair forms across a chunk's edge in a stage, which hardly matters: over 22
// scenes the traced frames take 0.99 of the time with passes over all places, a single
// one 0.9 to 1.1 either way (where a room's few large triangles land), and chunks of 256
// to 1,024 places with a half to a sixteenth kept 0.99 to 1.03. Nothing is read back.
// Passes over all places, three launches each and a read-back every eight, took the
// build of 7,950 triangles 0.99 ms and of 522,254 1.77; these stages, with the widening
// below, 0.48 and 0.82.
// Ids: a triangle in Morton order at [0, n), merged clusters from n on. A cluster is
// represented by its first triangle's place in that order; merging i with a higher
// place j gives up j's, so the merged cluster's id is n + that one.
constexpr uint32_t kSearch = 16, kBatch = 8;
constexpr uint32_t kChunk = 512, kKeep = 256, kFan = kChunk / kKeep;
constexpr uint32_t kLeafTris = 3;
constexpr uint32_t kNoPlace = 0xFFFFFFFFu;
constexpr float kFarthest = 1e15f;

struct Clusters {
  float4 *lo, *hi;  // box per id; lo.w triangles below, hi.w height (as bits)
  uint2* child;     // of id n + i
  uint32_t n;
};
// The build's counters: a vertex index was out of range; wide nodes and leaf
// triangles so far; clusters left (one); the widening's nodes for its second launch
// (first, count); the bounds of the centroids.
constexpr int kBad = 0, kWide = 1, kLeafs = 2, kLeft = 3, kFrontier = 4, kBox = 6, kCounters = 12;

__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
  const float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
  return x * y + y * z + z * x;
}

// A triangle's guard box: its bounds widened by a margin, so that only hits off the
// triangle fall outside. Of the hits that the triangle test accepts, slivers of
// aspect 0.01 to 1e-5 seen from up to 400 lengths away, one in 29,000 does; from 40,000
// lengths, 0.4 to 10%, whatever the margin between 1e-5 and 1/64 of the length. Wider
// boxes cost the traversal: 1/64 and 1e-4 of the coordinates 1,709 us for a rendered
// 1080p frame, 1/256 and 1e-5 1,629, 1/1024 1,581. The triangle's cluster starts from
// that box, kept within +-kFarthest: half_area stays finite, and so do the traversal's
// slab terms, at most 1e20 times a coordinate (see widen for what lies beyond).
__device__ __forceinline__ void triangle_boxes(const float4* tri, uint32_t t, float4* guard, float4& clo, float4& chi) {
  const float4 v0 = tri[size_t(t) * 3], v1 = tri[size_t(t) * 3 + 1], v2 = tri[size_t(t) * 3 + 2];
  float lo[3] = {fminf(fminf(v0.x, v1.x), v2.x), fminf(fminf(v0.y, v1.y), v2.y), fminf(fminf(v0.z, v1.z), v2.z)};
  float hi[3] = {fmaxf(fmaxf(v0.x, v1.x), v2.x), fmaxf(fmaxf(v0.y, v1.y), v2.y), fmaxf(fmaxf(v0.z, v1.z), v2.z)};
  float margin = 0.0f;
  for (int k = 0; k < 3; ++k)
    margin = fmaxf(margin, (hi[k] - lo[k]) * 0.0009765625f + (fabsf(lo[k]) + fabsf(hi[k])) * 1e-5f + 1e-6f);
  for (int k = 0; k < 3; ++k) {
    lo[k] = lo[k] - margin;
    hi[k] = hi[k] + margin;
  }
  guard[size_t(t) * 2] = make_float4(lo[0], lo[1], lo[2], 0.0f);
  guard[size_t(t) * 2 + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
  for (int k = 0; k < 3; ++k) {
    if (!(lo[k] <= hi[k])) lo[k] = hi[k] = 0.0f;  // no finite vertex: the triangle is never hit
    lo[k] = fminf(fmaxf(lo[k], -kFarthest), kFarthest);
    hi[k] = fminf(fmaxf(hi[k], -kFarthest), kFarthest);
  }
  clo = make_float4(lo[0], lo[1], lo[2], __uint_as_float(1u));
  chi = make_float4(hi[0], hi[1], hi[2], __uint_as_float(0u));
}

// A stage of the clustering: `in` holds the survivors (id, representative) of the
// previous stage's `chunks` blocks, kKeep places each, in_count[b] of them used; the
// first stage (in null) takes the triangles and makes their boxes. Leaves at most
// `keep` clusters of the block in out, their number in out_count.
// Equal areas choose the nearer place, then the pair that starts at an even place,
// then the lower place, so that runs of equal boxes pair up and some pair always
// chooses each other: of the pairs with the least area, distance and parity, the
// lowest does. Two rules keep height and passes bounded for every scene. Once a cluster
// is kMaxHeight high, all later passes of its block pair the clusters by place (even
// with odd), which halves them: one such pass in each of up to 21 stages and nine in the
// last. And when a batch of kBatch passes leaves more than half of the clusters, the
// next pass pairs by place: boxes that grow along the order choose their lower
// neighbour one and all, and only one pair of such a run is mutual. (4,000 triangles
// nested in one another: 56 high after 56 passes, by the search alone 129 and 3,919.)
// A full pass is bound by the minima and maxima of the areas, each pair's computed once
// and read by both places (twice, for either place: 7,700 cycles a pass, and 1.04 ms for
// the build of 522,254 triangles); with few clusters left, several lanes share one's
// pairs, and a pass is its barriers and shared-memory latency.
__global__ void __launch_bounds__(kChunk) cluster_kernel(Clusters C, const uint32_t* order, const float4* tri, float4* guard,
                                                         const uint2* in, const uint32_t* in_count, uint32_t chunks,
                                                         uint32_t keep, uint2* out, uint32_t* out_count) {
  extern __shared__ float4 cluster_smem[];
  float4 *const slo = cluster_smem, *const shi = slo + kChunk;
  float* const pair_area = reinterpret_cast<float*>(shi + kChunk);  // [kSearch][kChunk]
  __shared__ uint32_t sid[kChunk], srep[kChunk], snn[kChunk], warps[kChunk / 32];
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  uint32_t count = 0;
  bool tall = false;
  if (in == nullptr) {
    const uint32_t first = blockIdx.x * kChunk;
    count = min(C.n - first, kChunk);
    if (t < count) {
      float4 lo, hi;
      triangle_boxes(tri, order[first + t], guard, lo, hi);
      C.lo[first + t] = slo[t] = lo;
      C.hi[first + t] = shi[t] = hi;
      sid[t] = srep[t] = first + t;
    }
  } else {
    const uint32_t first = blockIdx.x * kFan, mine = first + t / kKeep;
    uint32_t at = t % kKeep, n = 0;
    for (uint32_t b = first; b < min(first + kFan, chunks); ++b) {
      const uint32_t c = in_count[b];
      if (b < mine) at += c;
      if (b == mine) n = c;
      count += c;
    }
    if (t % kKeep < n) {
      const uint2 v = in[size_t(mine) * kKeep + t % kKeep];
      sid[at] = v.x;
      srep[at] = v.y;
      slo[at] = C.lo[v.x];
      const float4 hi = C.hi[v.x];
      shi[at] = hi;
      tall = __float_as_uint(hi.w) >= kMaxHeight;
    }
  }
  tall = __syncthreads_or(tall) != 0;
  uint32_t batch_count = count;
  bool by_place = false;
  for (uint32_t pass = 1; count > keep && pass < kChunk; ++pass) {  // every pass merges a pair
    if (tall || by_place) {
      if (t < count) snn[t] = (t ^ 1u) < count ? t ^ 1u : kNoPlace;
    } else {
      const uint32_t share = min(__clz(count - 1u) - __clz(kChunk - 1u), 4), lanes = 1u << share;  // lanes a place: count << share <= kChunk
      const uint32_t i = t >> share, sub = t & (lanes - 1u);
      const float inf = __int_as_float(0x7F800000);
      if (i < count) {
        const float4 l = slo[i], h = shi[i];
#pragma unroll 4
        for (uint32_t o = sub; o < kSearch; o += lanes) {  // the pair of places i and i + o + 1
          float d = inf;
          if (i + o + 1 < count) {
            const float4 a = slo[i + o + 1], b = shi[i + o + 1];
            d = half_area(make_float4(fminf(l.x, a.x), fminf(l.y, a.y), fminf(l.z, a.z), 0.0f),
                          make_float4(fmaxf(h.x, b.x), fmaxf(h.y, b.y), fmaxf(h.z, b.z), 0.0f));
          }
          pair_area[o * kChunk + i] = d;
        }
      }
      __syncthreads();
      float best_d = inf;
      int best_o = 0;
      if (i < count) {
#pragma unroll 4
        for (uint32_t o = sub; o < kSearch; o += lanes) {
          const float above = pair_area[o * kChunk + i], below = i > o ? pair_area[o * kChunk + i - o - 1] : inf;
          const bool up = above < below || (above == below && ((i | o) & 1u) == 0u);  // an odd distance from an even place
          const float d = up ? above : below;
          if (d < best_d) {
            best_d = d;
            best_o = up ? static_cast<int>(o) + 1 : -static_cast<int>(o) - 1;
          }
        }
      }
      for (uint32_t off = 1; off < lanes; off <<= 1) {
        const float d = __shfl_xor_sync(0xffffffffu, best_d, off);
        const int o = __shfl_xor_sync(0xffffffffu, best_o, off);
        if (d < best_d || (d == best_d && abs(o) < abs(best_o))) {
          best_d = d;
          best_o = o;
        }
      }
      if (i < count && sub == 0u) snn[i] = i + best_o;
    }
    __syncthreads();
    const uint32_t j = t < count ? snn[t] : kNoPlace;
    const bool mutual = j != kNoPlace && snn[j] == t, kept = t < count && !(mutual && j < t);
    float4 lo = {}, hi = {};
    uint32_t id = 0, rep = 0;
    if (kept) {
      id = sid[t];
      rep = srep[t];
      lo = slo[t];
      hi = shi[t];
      if (mutual) {
        const float4 a = slo[j], b = shi[j];
        const uint32_t merged = srep[j];
        C.child[merged] = make_uint2(id, sid[j]);
        id = C.n + merged;
        lo = make_float4(fminf(lo.x, a.x), fminf(lo.y, a.y), fminf(lo.z, a.z),
                         __uint_as_float(__float_as_uint(lo.w) + __float_as_uint(a.w)));
        hi = make_float4(fmaxf(hi.x, b.x), fmaxf(hi.y, b.y), fmaxf(hi.z, b.z),
                         __uint_as_float(max(__float_as_uint(hi.w), __float_as_uint(b.w)) + 1u));
        C.lo[id] = lo;
        C.hi[id] = hi;
      }
    }
    const uint32_t m = __ballot_sync(0xffffffffu, kept);
    if (lane == 0) warps[warp] = __popc(m);
    tall = __syncthreads_or(tall || (kept && __float_as_uint(hi.w) >= kMaxHeight)) != 0;
    const uint32_t of_warp = lane < kChunk / 32 ? warps[lane] : 0u;
    const uint32_t at = __popc(m & ((1u << lane) - 1u)) + __reduce_add_sync(0xffffffffu, lane < warp ? of_warp : 0u);
    const uint32_t total = __reduce_add_sync(0xffffffffu, of_warp);
    if (kept) {
      sid[at] = id;
      srep[at] = rep;
      slo[at] = lo;
      shi[at] = hi;
    }
    count = total;
    by_place = false;
    if (pass % kBatch == 0) {
      by_place = count > batch_count / 2;
      batch_count = count;
    }
    __syncthreads();
  }
  if (t < min(count, keep)) out[size_t(blockIdx.x) * kKeep + t] = make_uint2(sid[t], srep[t]);
  if (t == 0) out_count[blockIdx.x] = count;
}

// The wide tree's nodes first .. first + count (at most T), each over the binary
// cluster cluster_of[w]. A node starts from its cluster and opens the largest until it
// has four (clusters of more than three triangles before smaller ones); what is left
// of up to three triangles becomes a leaf, whose triangles (in Morton order) go to
// leaf_of. The nodes' children are appended to the tree as one range, which is
// returned. Boxes are widened by 1e-6 of their coordinates: the traversal's p * i + o
// rounds by less. A box that reaches +-kFarthest has no plane on that side.
template <uint32_t T>
__device__ __forceinline__ uint2 widen(const Clusters& C, uint32_t* cluster_of, uint32_t* counters, uint32_t first,
                                       uint32_t count, WideNode* wide, uint32_t* leaf_of) {
  __shared__ uint32_t sums[T / 32], base[2];
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const bool in = t < count;
  float4 lo[4], hi[4];
  uint32_t c[4] = {0u, 0u, 0u, 0u};
  int k = 0;
  if (in) {
    c[0] = cluster_of[first + t];
    lo[0] = C.lo[c[0]];
    hi[0] = C.hi[c[0]];
    k = 1;
#pragma unroll
    for (int s = 1; s < 4; ++s) {
      int pick = -1;
      bool pick_large = false;
      float pick_area = 0.0f;
      uint32_t id = 0;
#pragma unroll
      for (int x = 0; x < s; ++x) {
        const uint32_t tris = __float_as_uint(lo[x].w);
        const bool large = tris > kLeafTris;
        const float area = half_area(lo[x], hi[x]);
        if (tris >= 2 && (pick < 0 || (large && !pick_large) || (large == pick_large && area > pick_area))) {
          pick = x;
          pick_large = large;
          pick_area = area;
          id = c[x];
        }
      }
      if (pick < 0) break;
      const uint2 ch = C.child[id - C.n];
      const float4 al = C.lo[ch.x], ah = C.hi[ch.x];
#pragma unroll
      for (int x = 0; x < s; ++x)
        if (x == pick) {
          c[x] = ch.x;
          lo[x] = al;
          hi[x] = ah;
        }
      c[s] = ch.y;
      lo[s] = C.lo[ch.y];
      hi[s] = C.hi[ch.y];
      k = s + 1;
    }
  }
  uint32_t nodes = 0, tris = 0;
#pragma unroll
  for (int s = 0; s < 4; ++s)
    if (s < k) {
      const uint32_t below = __float_as_uint(lo[s].w);
      if (below > kLeafTris) ++nodes; else tris += below;
    }
  // the block's ranges of nodes and leaf triangles, this thread's places in them (counts of both in one word)
  const uint32_t own = nodes | tris << 16;
  uint32_t upto = own;
#pragma unroll
  for (uint32_t off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, upto, off);
    if (lane >= off) upto += v;
  }
  if (lane == 31) sums[warp] = upto;
  __syncthreads();
  uint32_t before = upto - own, total = 0;
#pragma unroll
  for (uint32_t w = 0; w < T / 32; ++w) {
    if (w < warp) before += sums[w];
    total += sums[w];
  }
  if (t < 2) base[t] = atomicAdd(&counters[kWide + t], t == 0 ? total & 0xFFFFu : total >> 16);
  __syncthreads();
  const uint2 next = make_uint2(base[0], total & 0xFFFFu);
  if (in) {
    WideNode N = {};
    N.node0 = base[0] + (before & 0xFFFFu);
    N.tri0 = base[1] + (before >> 16);
    uint32_t node_at = N.node0, tri_at = N.tri0;
    float* plane = reinterpret_cast<float*>(N.plane);  // [6][4]
    const float inf = __int_as_float(0x7F800000);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if (s >= k) {
        for (int a = 0; a < 3; ++a) {
          plane[8 * a + s] = inf;
          plane[8 * a + 4 + s] = -inf;
        }
        continue;
      }
      const float l3[3] = {lo[s].x, lo[s].y, lo[s].z}, h3[3] = {hi[s].x, hi[s].y, hi[s].z};
      for (int a = 0; a < 3; ++a) {
        const float pad = fmaxf(fabsf(l3[a]), fabsf(h3[a])) * 1e-6f;
        plane[8 * a + s] = l3[a] > -kFarthest ? l3[a] - pad : -inf;
        plane[8 * a + 4 + s] = h3[a] < kFarthest ? h3[a] + pad : inf;
      }
      const uint32_t below = __float_as_uint(lo[s].w);
      if (below > kLeafTris) {
        N.contents |= 1u << (24 + s);
        cluster_of[node_at++] = c[s];
        continue;
      }
      N.contents |= ((1u << below) - 1u) << (3 * s);
      uint32_t x = c[s];  // three triangles or two are pairs over the triangles: each step takes one off
      for (uint32_t r = below; r > 1; --r) {
        const uint2 ch = C.child[x - C.n];
        const bool inner = ch.x >= C.n;
        leaf_of[tri_at++] = inner ? ch.y : ch.x;
        x = inner ? ch.x : ch.y;
      }
      leaf_of[tri_at++] = x;
    }
    wide[first + t] = N;
  }
  __syncthreads();  // the children's clusters are written, base and sums free
  return next;
}

// The wide tree from its root, node 0, level by level in two launches: one block until
// a level has kFrontierNodes nodes, then a block for each node of that level with
// everything below it. (A launch a level and a read-back every four took 129 us for
// 462 triangles and 360 for 522,254.)
constexpr uint32_t kFrontierNodes = 512, kMaxFrontier = 4 * kFrontierNodes, kWidenThreads = 64;
__global__ void __launch_bounds__(kFrontierNodes)
    widen_top_kernel(Clusters C, const uint2* root, uint32_t* cluster_of, uint32_t* counters, WideNode* wide, uint32_t* leaf_of) {
  if (threadIdx.x == 0) cluster_of[0] = root->x;
  __syncthreads();
  uint2 range = make_uint2(0u, 1u);
  while (range.y > 0 && range.y < kFrontierNodes)
    range = widen<kFrontierNodes>(C, cluster_of, counters, range.x, range.y, wide, leaf_of);
  if (threadIdx.x == 0) {
    counters[kFrontier] = range.x;
    counters[kFrontier + 1] = range.y;
  }
}
__global__ void __launch_bounds__(kWidenThreads)
    widen_kernel(Clusters C, uint32_t* cluster_of, uint32_t* counters, WideNode* wide, uint32_t* leaf_of) {
  __shared__ uint2 todo[kStack + 2];  // ranges of nodes; at most one a level
  if (blockIdx.x >= counters[kFrontier + 1]) return;
  int sp = 0;
  uint2 range = make_uint2(counters[kFrontier] + blockIdx.x, 1u);
  while (true) {
    const uint32_t part = min(range.y, kWidenThreads);
    const uint2 next = widen<kWidenThreads>(C, cluster_of, counters, range.x, part, wide, leaf_of);
    if (range.y > part) {
      if (threadIdx.x == 0) todo[sp] = make_uint2(range.x + part, range.y - part);
      ++sp;
      __syncthreads();
    }
    if (next.y > 0) {
      range = next;
    } else {
      if (sp == 0) break;
      range = todo[--sp];
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(256) leaf_kernel(uint32_t n, const uint32_t* leaf_of, const uint32_t* order, const float4* tri,
                                                   float4* leaf) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= n) return;
  const uint32_t t = order[leaf_of[i]];
  const float4 v0 = tri[size_t(t) * 3], v1 = tri[size_t(t) * 3 + 1], v2 = tri[size_t(t) * 3 + 2];
  float4* out = leaf + size_t(i) * 3;
  out[0] = make_float4(v0.x, v0.y, v0.z, __uint_as_float(t));
  out[1] = make_float4(v1.x - v0.x, v1.y - v0.y, v1.z - v0.z, 0.0f);
  out[2] = make_float4(v2.x - v0.x, v2.y - v0.y, v2.z - v0.z, 0.0f);
}

float srgb_to_linear(int i) {
  const double c = i / 255.0;
  return static_cast<float>(c <= 0.04045 ? c / 12.92 : std::pow((c + 0.055) / 1.055, 2.4));
}

}  // namespace
}  // namespace nrc

namespace {
int st(cudaError_t e) { return e == cudaSuccess ? NRC_OK : (e == cudaErrorMemoryAllocation ? NRC_ERROR_OUT_OF_MEMORY : NRC_ERROR_CUDA); }
}  // namespace

extern "C" {

int nrc_bvh_build(const nrc_scene* scene, const nrc_instance_range* d_ranges, nrc_bvh** out) {
  using namespace nrc;
  if (scene == nullptr || out == nullptr || (scene->instance_count > 0 && d_ranges == nullptr))
    return NRC_ERROR_INVALID_ARGUMENT;
  *out = nullptr;
  const uint32_t ni = scene->instance_count;
  std::vector<nrc_instance_range> ranges(ni);
  cudaError_t e = cudaSuccess;
  if (ni > 0) e = cudaMemcpy(ranges.data(), d_ranges, ni * sizeof(nrc_instance_range), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return st(e);
  std::vector<uint32_t> first(ni + 1, 0);
  uint64_t total = 0;
  for (uint32_t i = 0; i < ni; ++i) {
    if (uint64_t(ranges[i].first_primitive) + ranges[i].primitive_count > scene->primitive_count)
      return NRC_ERROR_INVALID_ARGUMENT;
    first[i] = static_cast<uint32_t>(total);
    total += ranges[i].primitive_count;
  }
  first[ni] = static_cast<uint32_t>(total);
  if (total >= (1u << 30)) return NRC_ERROR_TOO_LARGE;
  const uint32_t n = static_cast<uint32_t>(total);
  nrc_bvh* B = new (std::nothrow) nrc_bvh();
  if (B == nullptr) return NRC_ERROR_OUT_OF_MEMORY;
  cudaGetDevice(&B->device);
  B->tris = n;
  B->nodes = n > 1 ? n - 1 : 0;
  // Each wide node but the root is over more than kLeafTris triangles and so has
  // more than kLeafTris children (or four): with c children a node, N nodes and
  // at most n leaves, c N <= N - 1 + n.
  static_assert(kLeafTris >= 1 && kLeafTris <= 3, "at most three triangles a slot, four slots");
  const size_t nn = n, max_wide = nn / kLeafTris + 2;
  if ((e = cudaMalloc(&B->block, max_wide * sizeof(WideNode) + nn * (5 * sizeof(float4) + sizeof(uint2)) + 256)) !=
      cudaSuccess) {
    delete B;
    return st(e);
  }
  WideNode* wide = static_cast<WideNode*>(B->block);
  float4* guard = reinterpret_cast<float4*>(wide + max_wide);
  float4* leaf = guard + 2 * nn;
  uint2* id = reinterpret_cast<uint2*>(leaf + 3 * nn);
  B->id = id;
  B->guard = guard;
  B->leaf = leaf;
  B->wide = wide;
  if (n > 0) {
    // scratch for the build: one allocation, carved below
    size_t tmp_bytes = 0, at = 0;
    uint32_t* const none = nullptr;
    e = cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, none, none, none, none, static_cast<int>(n));
    auto carve = [&](size_t bytes) {
      const size_t o = at;
      at += (bytes + 255) & ~size_t(255);
      return o;
    };
    const size_t chunks = (nn + kChunk - 1) / kChunk;
    const size_t o_hi = carve(2 * nn * 16), o_tri = carve(nn * 48), o_keys = carve(nn * 4), o_vals = carve(nn * 4),
                 o_keys2 = carve(nn * 4), o_vals2 = carve(nn * 4), o_kept = carve(chunks * kKeep * 8),
                 o_kept2 = carve((chunks + kFan - 1) / kFan * kKeep * 8), o_count = carve(chunks * 4),
                 o_count2 = carve(chunks * 4), o_words = carve((kCounters + ni + 1) * 4),
                 o_tmp = carve(tmp_bytes ? tmp_bytes : 16);
    uint8_t* m = nullptr;
    if (e == cudaSuccess) e = cudaMalloc(&m, at);
    auto u32 = [&](size_t o) { return reinterpret_cast<uint32_t*>(m + o); };
    uint32_t *keys = u32(o_keys), *vals = u32(o_vals), *keys2 = u32(o_keys2), *vals2 = u32(o_vals2), *counters = u32(o_words);
    float4* tri = reinterpret_cast<float4*>(m + o_tri);
    // The leaf array, written last, holds the clusters' low corners and children until
    // then, and their upper half the centroids until the first merge.
    float4* lo = leaf;
    uint2* child = reinterpret_cast<uint2*>(leaf + 2 * nn);
    float* cent = reinterpret_cast<float*>(leaf + nn);
    // the counters, then each instance's first triangle
    std::vector<uint32_t> words = {0u, 1u, 0u, 0u, 0u, 0u, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
    words.insert(words.end(), first.begin(), first.end());
    if (e == cudaSuccess) e = cudaMemcpy(counters, words.data(), words.size() * 4, cudaMemcpyHostToDevice);
    BuildArgs A{*scene, d_ranges, counters + kCounters, ni, n};
    const uint32_t blocks = (n + 255) / 256;
    if (e == cudaSuccess) {
      tri_kernel<<<blocks, 256>>>(A, tri, id, cent, counters + kBad);
      bounds_kernel<<<blocks < 1024 ? blocks : 1024, 256>>>(cent, n, counters + kBox);
      morton_kernel<<<blocks, 256>>>(cent, n, counters + kBox, keys, vals);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess)
      e = cub::DeviceRadixSort::SortPairs(m + o_tmp, tmp_bytes, keys, keys2, vals, vals2, static_cast<int>(n), 0, 30);
    constexpr int kClusterSmem = kChunk * (2 * sizeof(float4) + kSearch * sizeof(float));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterSmem);
    if (e == cudaSuccess) {
      // the clustering, from the triangles in Morton order (vals2) to one cluster
      const Clusters C{lo, reinterpret_cast<float4*>(m + o_hi), child, n};
      const uint2* in = nullptr;
      const uint32_t* in_count = nullptr;
      uint2 *kept = reinterpret_cast<uint2*>(m + o_kept), *kept2 = reinterpret_cast<uint2*>(m + o_kept2);
      uint32_t *count = u32(o_count), *count2 = u32(o_count2);
      for (uint32_t of = 0, grid = static_cast<uint32_t>(chunks); of != 1; of = grid, grid = (grid + kFan - 1) / kFan) {
        cluster_kernel<<<grid, kChunk, kClusterSmem>>>(C, vals2, tri, guard, in, in_count, of, grid == 1 ? 1u : kKeep, kept,
                                         grid == 1 ? counters + kLeft : count);
        in = kept;
        in_count = count;
        std::swap(kept, kept2);
        std::swap(count, count2);
      }
      // the wide tree; node 0 is over the last cluster
      widen_top_kernel<<<1, kFrontierNodes>>>(C, in, keys2, counters, wide, keys);
      widen_kernel<<<kMaxFrontier, kWidenThreads>>>(C, keys2, counters, wide, keys);
      leaf_kernel<<<blocks, 256>>>(n, keys, vals2, tri, leaf);
      e = cudaGetLastError();
    }
    uint32_t done[kLeft + 1] = {0u, 0u, 0u, 0u};
    if (e == cudaSuccess) e = cudaMemcpy(done, counters, sizeof(done), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && !done[kBad] && (done[kLeft] != 1 || done[kLeafs] != n)) e = cudaErrorUnknown;  // not for any scene
    cudaFree(m);
    if (e == cudaSuccess && done[kBad]) {
      cudaFree(B->block);
      delete B;
      return NRC_ERROR_INVALID_ARGUMENT;  // an index past the scene's buffers
    }
  }
  if (e != cudaSuccess) {
    cudaFree(B->block);
    delete B;
    return st(e);
  }
  *out = B;
  return NRC_OK;
}

int nrc_bvh_destroy(nrc_bvh* B) {
  if (B == nullptr) return NRC_ERROR_INVALID_ARGUMENT;
  cudaDeviceSynchronize();
  cudaFree(B->block);
  delete B;
  return NRC_OK;
}

int nrc_bvh_info(const nrc_bvh* B, uint32_t* tris, uint32_t* nodes) {
  if (B == nullptr) return NRC_ERROR_INVALID_ARGUMENT;
  if (tris) *tris = B->tris;
  if (nodes) *nodes = B->nodes;
  return NRC_OK;
}

int nrc_path_trace(const nrc_scene* scene, const nrc_bvh* bvh, const nrc_trace_params* p, const nrc_trace_targets* t,
                   void* stream) {
  using namespace nrc;
  if (scene == nullptr || bvh == nullptr || p == nullptr || t == nullptr) return NRC_ERROR_INVALID_ARGUMENT;
  if (p->width == 0 || p->height == 0) return NRC_OK;
  if (p->width > 0x8000u || p->height > 0x10000u) return NRC_ERROR_INVALID_ARGUMENT;  // dst word's 15 / 16 bits
  if (p->left_method > 2 || p->right_method > 2) return NRC_ERROR_INVALID_ARGUMENT;
  if (t->eval_count == nullptr || (t->eval_capacity > 0 && t->eval_records == nullptr) ||
      t->bias_factor_r == nullptr || t->factor_gb == nullptr)
    return NRC_ERROR_INVALID_ARGUMENT;
  for (int b = 0; b < NRC_TRAIN_BATCH_COUNT; ++b)
    if (t->train_counts[b] == nullptr || t->train_records[b] == nullptr) return NRC_ERROR_INVALID_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(t->bias_factor_r) & 15u) || (reinterpret_cast<uintptr_t>(t->factor_gb) & 7u))
    return NRC_ERROR_MISALIGNED;
  TraceArgs A;
  A.sc.s = *scene;
  for (int i = 0; i < 256; ++i) A.sc.lut[i] = srgb_to_linear(i);
  A.bvh = TriView{bvh->id, bvh->guard, bvh->leaf, bvh->wide, bvh->tris};
  A.p = *p;
  A.t = *t;
  dim3 grid((p->width + 7) / 8, (p->height + 7) / 8);
  path_trace_kernel<<<grid, dim3(8, 8), 256 * sizeof(float), static_cast<cudaStream_t>(stream)>>>(A);
  return st(cudaGetLastError());
}

}  // extern "C"
