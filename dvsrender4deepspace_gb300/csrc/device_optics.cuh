// Device-side optics of the GB300 DVS path: float3 algebra, Hapke, pose
// interpolation, the 8-wide warp-packet BVH traversal and the pixel sample.
// Included by the CUDA translation units that trace rays; everything has
// internal linkage.  Compiled with -fmad=false (see kernels.cu).
#pragma once
#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "device_math.cuh"
#include "kernels.h"

namespace dvsgb {
namespace {
constexpr unsigned kFull = 0xffffffffu;
constexpr float kRayEps = 1e-6f;          // include/helper_math.hpp:12
constexpr float kPi = 3.14159265358979323846f;  // include/dvs/math_types.hpp:37
__device__ __forceinline__ float kInf() { return __int_as_float(0x7f800000); }

// ---- float3 algebra (include/helper_math.hpp:18-77) -------------------------
__device__ __forceinline__ float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator-(float3 a) { return f3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 operator*(float s, float3 a) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 operator/(float3 a, float s) { return f3(a.x / s, a.y / s, a.z / s); }
__device__ __forceinline__ float dot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross(float3 a, float3 b) {
  return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float3 normalize(float3 v) {
  float len = sqrtf(dot(v, v));
  if (len > 0.0f) return v / len;
  return f3(0.0f, 0.0f, 0.0f);
}
// normalize in the forms of device_math.cuh (a zero vector stays zero).  Not for vectors shorter than 2^-63, whose
// squares are denormal: rays and lights are near 1, a scene's normals are stored long enough (normal_scaling).
__device__ __forceinline__ float3 unit(float3 v) {
  const float len = sqrt_rn(dot(v, v));
  if (!(len > 0.0f)) return f3(0.0f, 0.0f, 0.0f);
  const float y = rcp_rn(len);
  return f3(div_by(v.x, len, y), div_by(v.y, len, y), div_by(v.z, len, y));
}
__device__ __forceinline__ float clampf(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }

// ---- Hapke (include/dvs/hapke.hpp:14-157), FP32 --------------------------------
// The reference's formulas evaluated through trigonometric identities
// ("identity form"): every transcendental of the phase and azimuth angles
// except acos(cos psi) becomes a square root of a ratio, which the CUDA
// compiler turns into far fewer instructions than tanf/sinf/cosf/powf:
//   tan(acos(c) / 2) = sqrt((1 - c) / (1 + c))      (hapke.hpp:135, :82-84)
//   sin(psi / 2)     = sqrt((1 - cos psi) / 2)       (hapke.hpp:92)
//   cos(psi)         = cos psi (the clamped argument of acos, hapke.hpp:96,123)
//   y^1.5            = y * sqrt(y)                   (hapke.hpp:22-29)
//   e1(y) = exp(-2/pi * q), e2(y) = exp(-1/pi * q^2) with the one quotient
//   q = cot(thetap) cos(y) / sin(y)                  (hapke.hpp:64-73)
// Each is exact in real arithmetic; in FP32 the result stays within a few
// ulp of the reference's own order (bounded against the FP64 oracle in
// tests/test_oracle_golden.py).  The clamps and the one non-finite case keep
// the reference's values: tan(phase/2) is capped at tan(pi/2 - 1e-6)
// (safe_tan, hapke.hpp:14-16), and psi == acos(-1) keeps the reference's
// tan(pi_f / 2) < 0, whose exp overflows and makes the sample NaN (dropped by
// the caller's fmaxf) -- here tan(psi/2) = -inf there.
__device__ __forceinline__ float pow15(float y) { return y * sqrt_rn(y); }
__device__ __forceinline__ float hg_double_lobe(float cosg, const HapkeConst &h) {
  const float den1 = pow15(1.0f - 2.0f * h.b * cosg + h.b * h.b);
  const float den2 = pow15(1.0f + 2.0f * h.b * cosg + h.b * h.b);
  const float lobes = div_rn(h.lobe_pos, den1) + div_rn(h.lobe_neg, den2);
  // a lobe so narrow that its denominator rounds to 0: the quotient by 0 that div_rn does not give
  return fminf(den1, den2) == 0.0f ? h.lobe_zero : lobes;
}
__device__ __forceinline__ float b_s(float tg, float h, float inv_h) {
  if (h <= 0.0f) return tg <= 0.0f ? 1.0f : 0.0f;
  return rcp_rn(1.0f + div_by(tg, h, inv_h));
}
__device__ __forceinline__ float b_c(float tg, float h) {
  if (h <= 0.0f) return tg <= 0.0f ? 1.0f : 0.0f;
  const float T = tg / h;
  if (T < 1e-8f) return 1.0f;
  return (1.0f + (1.0f - expf(-T)) / T) / (2.0f * (1.0f + T) * (1.0f + T));
}
__device__ __forceinline__ float hfunc(float x, float w, float r0) {
  if (x <= 1e-8f) return 1.0f;
  const float term = r0 + (1.0f - 2.0f * r0 * x) * 0.5f * logf(1.0f + rcp_rn(x));
  return rcp_rn(1.0f - w * x * term);
}
__device__ __forceinline__ float hfunc_r0(float w) {
  const float root = sqrtf(fmaxf(0.0f, 1.0f - w));
  return (1.0f - root) / (1.0f + root);
}
__device__ __forceinline__ float porosity_k(float phi) {
  if (phi <= 1e-8f) return 1.0f;
  const float p = 1.209f * powf(phi, 2.0f / 3.0f);
  return -logf(1.0f - p) / p;
}

// A material as the kernels read it.  The parts of hapke.hpp that depend on the
// material only are each the value hapke.hpp recomputes inside every call (same
// operations, same rounding; divisors brought into div_by's range): evaluated on
// the device once per scene (hapke_const_kernel) and read from the view as constants.  Evaluated per pixel sample loop, two tanf, a powf and a
// logf were a sixth of a one-ray loop.
__device__ __forceinline__ HapkeConst hapke_const(const dvs_hapke &p) {
  HapkeConst h;
  h.w = p.w;
  h.hC = p.hC;
  h.B_S0 = p.B_S0;
  h.B_C0 = p.B_C0;
  h.K = porosity_k(p.phi);
  h.K_div = isinf(h.K) ? 1e30f : h.K;  // the H-functions' argument is as good as 0 either way
  h.inv_K = 1.0f / h.K_div;
  h.rough = !(p.thetap <= 1e-8f);
  h.tan_t = tanf(p.thetap);
  h.cot_t = 1.0f / h.tan_t;
  h.chi = 1.0f / sqrtf(1.0f + kPi * h.tan_t * h.tan_t);
  h.r0_w = hfunc_r0(p.w);
  h.tg_max = tanf(kPi / 2.0f - 1e-6f);
  // beyond |b| = 1e12, where the denominators leave the float range, the lobes are as good as 0
  const bool lobes = !(fabsf(p.b) > 1e12f);
  h.b = lobes ? p.b : 0.0f;
  const float one_minus_bb = 1.0f - p.b * p.b;
  h.lobe_pos = lobes ? ((1.0f + p.c) * 0.5f) * one_minus_bb : 0.0f;
  h.lobe_neg = lobes ? ((1.0f - p.c) * 0.5f) * one_minus_bb : 0.0f;
  h.lobe_zero = (p.b > 0.0f ? h.lobe_pos : h.lobe_neg) * kInf();
  // narrower than 1e-30 the surge is below 1e-26 off the exact opposition and 1 at it, as here
  h.hS = p.hS > 0.0f && p.hS < 1e-30f ? 1e-30f : p.hS;
  h.inv_hS = 1.0f / h.hS;
  return h;
}
// The quotient q = cot(thetap) cos(y) / max(sin(y), 1e-6) shared by e1 and e2.
__device__ __forceinline__ float e_quot(float cot_t, float cosy, float siny) {
  return div_rn(cot_t * cosy, fmaxf(siny, 1e-6f));
}

// Inlining policy of the large shading and traversal bodies (instruction-cache pressure).
#ifdef DVS_OUTLINE_SHADING
#define DVS_SHADE_INLINE __noinline__
#else
#define DVS_SHADE_INLINE
#endif
// hapke_reflectance (hapke.hpp:131-152) in the identity form above; r0 is
// hfunc's r0 for this albedo.  Quotients with a divisor in common share its
// reciprocal, and constant divisors have theirs beforehand.  The divisors are
// normal: 2 - e1 >= 1, the shadowing denominators and sines at least 1e-6, the
// material's own brought into range (hapke_const), the lobes' checked
// (hg_double_lobe); 1 + cos g and 1 + cos psi are 0 or at least 6e-8, with the
// 0 noted at its use.  A NaN sample (the azimuth's above) is dropped by the
// caller's fmaxf; an infinite one is not, and makes the call report it.
DVS_SHADE_INLINE __device__ float hapke_reflectance(float cosi, float cose, float cosg, float albedo, float r0,
                                                    const HapkeConst &h) {
  if (cosi <= 0 || cose <= 0) return 0;
  cosi = clampf(cosi, 0, 1);
  cose = clampf(cose, 0, 1);
  cosg = clampf(cosg, -1, 1);
  const float sini = sqrt_rn(fmaxf(0, 1 - cosi * cosi)), sine = sqrt_rn(fmaxf(0, 1 - cose * cose));
  const float tg = fminf(sqrt_rn(div_rn(1.0f - cosg, 1.0f + cosg)), h.tg_max);  // cos g = -1: NaN, and fminf takes tg_max
  const float cpsi = clampf(div_rn(cosg - cosi * cose, sini * sine + 1e-6f), -1.0f, 1.0f);
  const float psi = acosf(cpsi);
  const float p_g = hg_double_lobe(cosg, h);
  const float BS = b_s(tg, h.hS, h.inv_hS);
  // b_c is finite, so with B_C0 == 0 the factor (1 + BC * B_C0) is exactly 1
  // whatever BC is: skip its evaluation.
  const float BC = h.B_C0 != 0.0f ? b_c(tg, h.hC) : 0.0f;
  const float K = h.K;
  float mu0, mue, S;
  if (!h.rough) {
    mu0 = cosi; mue = cose; S = 1.0f;
  } else {
    const float ch = h.chi;
    const float tan_thetap = h.tan_t;
    const float s2 = (1.0f - cpsi) * 0.5f;              // sin^2(psi / 2)
    const float qe = e_quot(h.cot_t, cose, sine), qi = e_quot(h.cot_t, cosi, sini);
    const float e2e = expf((-1.0f / kPi) * qe * qe), e2i = expf((-1.0f / kPi) * qi * qi);
    const float e1e = expf((-2.0f / kPi) * qe), e1i = expf((-2.0f / kPi) * qi);
    // eta(y) = chi * (cos y + sin y * tan(thetap) * e2(y) / (2 - e1(y)))
    const float eta_e = ch * (cose + div_rn(sine * tan_thetap * e2e, 2.0f - e1e));
    const float eta_i = ch * (cosi + div_rn(sini * tan_thetap * e2i, 2.0f - e1i));
    const float tpsi = cpsi > -1.0f ? sqrt_rn(div_rn(1.0f - cpsi, 1.0f + cpsi)) : -kInf();  // tan(psi / 2)
    const float fp = expf(-2.0f * tpsi);
    const float psi_pi = div_by(psi, kPi, 1.0f / kPi);
    // the two branches of hapke.hpp with incidence and emission exchanged
    const bool low = cosi >= cose;
    const float e1a = low ? e1e : e1i, e1b = low ? e1i : e1e;
    const float e2a = low ? e2e : e2i, e2b = low ? e2i : e2e;
    const float cosa = low ? cosi : cose, sina = low ? sini : sine;  // the angle nearer the normal
    const float cosb = low ? cose : cosi, sinb = low ? sine : sini;
    const float den = 2.0f - e1a - psi_pi * e1b, yden = rcp_rn(den);
    const float mua = ch * (cosa + div_by(sina * tan_thetap * (cpsi * e2a + s2 * e2b), den, yden));
    const float mub = ch * (cosb + div_by(sinb * tan_thetap * (e2a - s2 * e2b), den, yden));
    mu0 = low ? mua : mub;
    mue = low ? mub : mua;
    const float yi = rcp_rn(eta_i);
    const float f = div_by(div_rn(mue, eta_e) * cosi, eta_i, yi) * ch;  // mue / eta_e * cosi / eta_i * ch
    const float shadowed = low ? div_by(cosi, eta_i, yi) : div_rn(cose, eta_e);
    S = div_rn(f, 1.0f - fp + fp * ch * shadowed);
  }
  const float M = hfunc(div_by(mu0, h.K_div, h.inv_K), albedo, r0) * hfunc(div_by(mue, h.K_div, h.inv_K), albedo, r0) - 1.0f;
  const float LS = div_rn(mu0, mu0 + mue + 1e-6f);
  return div_by(albedo, 4.0f * kPi, 1.0f / (4.0f * kPi)) * LS * K * (p_g * (1.0f + BS * h.B_S0) + M) *
         (1.0f + BC * h.B_C0) * S;
}

// ---- pose interpolation (include/dvs/device_optics.cuh:6-29) ---------------------
__device__ __forceinline__ float hermite(float a, float va, float b, float vb, float u, float dt) {
  float u2 = u * u, u3 = u2 * u;
  return a + (-2 * u3 + 3 * u2) * (b - a) + (u3 - 2 * u2 + u) * dt * va + (u3 - u2) * dt * vb;
}
__device__ __forceinline__ float3 ld3(const dvs_float3 &v) { return f3(v.x, v.y, v.z); }
__device__ __forceinline__ float3 hermite3(const dvs_float3 &a, const dvs_float3 &va, const dvs_float3 &b,
                                           const dvs_float3 &vb, float u, float dt) {
  return f3(hermite(a.x, va.x, b.x, vb.x, u, dt), hermite(a.y, va.y, b.y, vb.y, u, dt),
            hermite(a.z, va.z, b.z, vb.z, u, dt));
}
// optical_state_at reduced to what the ray generator needs.  The quaternion
// is renormalized with a correctly rounded 1/sqrt (the reference's rsqrtf is
// an approximation the CPU oracle cannot reproduce).
__device__ CellPose pose_at(const dvs_optical_interval &iv, double t) {
  float dt = iv.t1 - iv.t0, u = dt > 0 ? fmin(1.0, fmax(0.0, (t - iv.t0) / dt)) : 0;
  float3 pos = hermite3(iv.start.position, iv.start.velocity, iv.end.position, iv.end.velocity, u, dt);
  float3 light = hermite3(iv.start.light, iv.start.light_rate, iv.end.light, iv.end.light_rate, u, dt);
  float intensity = fmaxf(0, hermite(iv.start.intensity, iv.start.intensity_rate, iv.end.intensity,
                                     iv.end.intensity_rate, u, dt));
  float4 a = make_float4(iv.start.rotation.x, iv.start.rotation.y, iv.start.rotation.z, iv.start.rotation.w);
  float4 b = make_float4(iv.end.rotation.x, iv.end.rotation.y, iv.end.rotation.z, iv.end.rotation.w);
  float d = a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w;
  if (d < 0) { b = make_float4(-b.x, -b.y, -b.z, -b.w); d = -d; }
  float wa = 1 - u, wb = u;
  if (d < .9995f) {
    float angle = acosf(fminf(1, d)), inv = 1 / sinf(angle);
    wa = sinf((1 - u) * angle) * inv;
    wb = sinf(u * angle) * inv;
  }
  float4 q = make_float4(wa * a.x + wb * b.x, wa * a.y + wb * b.y, wa * a.z + wb * b.z, wa * a.w + wb * b.w);
  float norm = 1.0f / sqrtf(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
  float3 ln = normalize(light);  // sample_pixel normalizes pose.light (device_optics.cuh:75)
  CellPose out;
  out.px = pos.x; out.py = pos.y; out.pz = pos.z; out.intensity = intensity;
  out.qx = q.x * norm; out.qy = q.y * norm; out.qz = q.z * norm; out.qw = q.w * norm;
  out.lx = ln.x; out.ly = ln.y; out.lz = ln.z; out.pad = 0;
  return out;
}
__device__ __forceinline__ float3 rotate_ray(const CellPose &q, float3 v) {
  float3 qv = f3(q.qx, q.qy, q.qz);
  float3 c = 2 * cross(qv, v);
  return v + q.qw * c + cross(qv, c);
}

// ---- traversal -------------------------------------------------------------------
__device__ __forceinline__ float3 inverse_direction(float3 d) {  // device_ray.hpp:6-12
  float3 inv;
  inv.x = rcp_rn(fabsf(d.x) > 1e-20f ? d.x : copysignf(1e-20f, d.x));
  inv.y = rcp_rn(fabsf(d.y) > 1e-20f ? d.y : copysignf(1e-20f, d.y));
  inv.z = rcp_rn(fabsf(d.z) > 1e-20f ? d.z : copysignf(1e-20f, d.z));
  return inv;
}

// Scene geometry formats, as bit flags: the reference's (FP32 child bounds,
// Moller-Trumbore on stored edges), kGeoHalfBounds (FP16 child bounds
// quantised outward against a per-node FP32 origin) and kGeoWatertight (the
// watertight FP32 triangle test on stored vertices), alone or together.
enum GeometryKind : int { kGeoReference = 0, kGeoHalfBounds = 1, kGeoWatertight = 2 };

// Moller-Trumbore with precomputed edges (device_ray.hpp:54-80).
__device__ __forceinline__ bool intersect_tri(float3 ray, float3 o, float3 v0, float3 e1, float3 e2, float &t,
                                              float &u, float &v) {
  const float3 pvec = cross(ray, e2);
  const float det = dot(e1, pvec);
  if (fabsf(det) < kRayEps) return false;
  const float inv_det = rcp_rn(det);
  const float3 tvec = o - v0;
  u = dot(tvec, pvec) * inv_det;
  if (u < 0.0f || u > 1.0f) return false;
  const float3 qvec = cross(tvec, e1);
  v = dot(ray, qvec) * inv_det;
  if (v < 0.0f || (u + v) > 1.0f) return false;
  t = dot(e2, qvec) * inv_det;
  if (t <= kRayEps) return false;
  return true;
}

// Watertight ray/triangle test (Woop, Benthin and Wald, "Watertight
// Ray/Triangle Intersection", JCGT 2(1), 2013) for precision scenes.  The ray
// is sheared onto +z through its origin (kz = the dominant axis of the
// direction, kx/ky swapped when it is negative), the vertices are projected,
// and the signs of the 2-D edge functions U, V, W decide the hit: a ray
// through a shared edge or vertex hits at least one of the triangles.  An edge
// function that rounds to exactly zero is recomputed in FP64 (the products of
// two floats are exact there), as the paper prescribes.  U, V, W weight v0,
// v1, v2, so the reference's barycentrics (u on v1, v on v2) are V/det, W/det.
//
// GB300 layout: a watertight scene stores each triangle three times, its
// vertices in the cyclic axis orders (y,z,x), (z,x,y) and (x,y,z) -- copy kz
// lists axis kz last -- and a ray reads the copy of its dominant axis, so the
// test runs on vertices already in the ray's (kx, ky, kz) order without a
// select per component.  The paper's swap of kx and ky for a negative
// direction only preserves the winding: it negates U, V, W, det and T
// exactly, so t, u and v are the same bits with or without it, and the
// kernels leave it out.
struct WtRay {
  int kz;
  float sx, sy, sz;
};
__device__ __forceinline__ float comp3(float3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }
// A vector in the cyclic order whose last axis is kz.
__device__ __forceinline__ float3 wt_perm(float3 v, int kz) {
  return kz == 2 ? v : (kz == 0 ? f3(v.y, v.z, v.x) : f3(v.z, v.x, v.y));
}
__device__ __forceinline__ WtRay wt_setup(float3 d) {
  const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  WtRay w;
  w.kz = ax > ay ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
  const float3 p = wt_perm(d, w.kz);
  w.sz = rcp_rn(p.z);  // the dominant axis: at least 0.57 of the length
  w.sx = div_by(p.x, p.z, w.sz);
  w.sy = div_by(p.y, p.z, w.sz);
  return w;
}
// o, v0, v1, v2 in the ray's cyclic order (wt_perm).
__device__ __forceinline__ bool intersect_wt(const WtRay &w, float3 o, float3 v0, float3 v1, float3 v2, float &t,
                                             float &u, float &v) {
  const float3 A = v0 - o, B = v1 - o, C = v2 - o;
  const float az = A.z, bz = B.z, cz = C.z;
  const float ax = A.x - w.sx * az, ay = A.y - w.sy * az;
  const float bx = B.x - w.sx * bz, by = B.y - w.sy * bz;
  const float cx = C.x - w.sx * cz, cy = C.y - w.sy * cz;
  float U = cx * by - cy * bx, V = ax * cy - ay * cx;
  // A nonzero float edge function has the sign of the exact one (rounding
  // keeps the order of the two products), and so does its FP64 recomputation:
  // opposite nonzero signs of U and V are a miss whatever W is, decided
  // before W is formed.
  if ((U < 0.0f && V > 0.0f) || (U > 0.0f && V < 0.0f)) return false;
  float W = bx * ay - by * ax;
  if (U == 0.0f || V == 0.0f || W == 0.0f) {
    U = (float)((double)cx * (double)by - (double)cy * (double)bx);
    V = (float)((double)ax * (double)cy - (double)ay * (double)cx);
    W = (float)((double)bx * (double)ay - (double)by * (double)ax);
  }
  if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
  const float det = U + V + W;
  if (det == 0.0f) return false;
  const float T = U * (w.sz * az) + V * (w.sz * bz) + W * (w.sz * cz);
  const float rcp = rcp_small(det);  // the smallest triangles' is denormal; beyond the float range: a miss
  t = T * rcp;
  if (!(t > kRayEps)) return false;
  u = V * rcp;
  v = W * rcp;
  return true;
}
// One leaf-order triangle record against one ray.  Records hold (v0, e1, e2),
// or in watertight scenes (v0, v1, v2) in the ray's cyclic order; o is the
// ray origin, op the origin in that order (watertight scenes).
template <int kGeo>
__device__ __forceinline__ bool tri_hit(const WtRay &w, float3 d, float3 o, float3 op, float4 a, float4 b, float4 q,
                                        float &t, float &u, float &v) {
  if constexpr (!(kGeo & kGeoWatertight))
    return intersect_tri(d, o, f3(a.x, a.y, a.z), f3(a.w, b.x, b.y), f3(b.z, b.w, q.x), t, u, v);
  else
    return intersect_wt(w, op, f3(a.x, a.y, a.z), f3(a.w, b.x, b.y), f3(b.z, b.w, q.x), t, u, v);
}
template <int kGeo>
__device__ __forceinline__ WtRay wt_ray(float3 d) {
  if constexpr (!(kGeo & kGeoWatertight)) return WtRay{2, 0.f, 0.f, 0.f};
  else return wt_setup(d);
}
template <int kGeo>
__device__ __forceinline__ float3 wt_origin(const WtRay &w, float3 o) {
  if constexpr (!(kGeo & kGeoWatertight)) return o;
  else return wt_perm(o, w.kz);
}
// The record of leaf-order triangle `tri` a ray with dominant axis kz reads:
// the single record, or in watertight scenes its copy kz (copy 2 holds the
// vertices in world order).
template <int kGeo>
__device__ __forceinline__ const float4 *tri_record(const SceneView &S, int tri, int kz) {
  if constexpr (!(kGeo & kGeoWatertight)) return reinterpret_cast<const float4 *>(S.tris + tri);
  else return reinterpret_cast<const float4 *>(S.tris + 3 * (size_t)tri + kz);
}

// ---- 8-wide packet traversal ------------------------------------------------------
// Float min/max across a warp through order-preserving unsigned keys.
__device__ __forceinline__ unsigned ford(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float funord(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ float wmin(float x) { return funord(__reduce_min_sync(kFull, ford(x))); }
__device__ __forceinline__ float wmax(float x) { return funord(__reduce_max_sync(kFull, ford(x))); }

struct ChildRec {
  float3 lo, hi;
  int child, count;
};
__device__ __forceinline__ float half_bits_to_float(unsigned bits) {
  return __half2float(__ushort_as_half((unsigned short)(bits & 0xffffu)));
}
// Child record `slot` of node `node`.  Precision nodes decode each bound as
// origin + offset with the addition rounded toward -inf (lower bounds) or +inf
// (upper bounds); the builder rounded the offsets the same way, so a decoded
// box always contains the exact FP32 box and no ray misses a child it would
// enter (the leaf's triangles are then tested in FP32).
template <int kGeo>
__device__ __forceinline__ ChildRec load_child(const SceneView &S, int node, int slot) {
  ChildRec r;
  if constexpr (!(kGeo & kGeoHalfBounds)) {
    const float4 *p = reinterpret_cast<const float4 *>(&S.nodes[node].c[slot]);
    const float4 a = __ldg(p), b = __ldg(p + 1);
    r.lo = f3(a.x, a.y, a.z);
    r.hi = f3(a.w, b.x, b.y);
    r.child = __float_as_int(b.z);
    r.count = __float_as_int(b.w);
  } else {
    const float4 org = __ldg(reinterpret_cast<const float4 *>(S.qnodes + node));
    const uint4 c = __ldg(reinterpret_cast<const uint4 *>(&S.qnodes[node].c[slot]));
    r.lo = f3(__fadd_rd(org.x, half_bits_to_float(c.x)), __fadd_rd(org.y, half_bits_to_float(c.x >> 16)),
              __fadd_rd(org.z, half_bits_to_float(c.y)));
    r.hi = f3(__fadd_ru(org.x, half_bits_to_float(c.y >> 16)), __fadd_ru(org.y, half_bits_to_float(c.z)),
              __fadd_ru(org.z, half_bits_to_float(c.z >> 16)));
    const unsigned link = c.w;
    if (link == kQLinkEmpty) {
      r.child = 0;
      r.count = -1;
    } else if (link & kQLinkLeaf) {
      r.child = (int)(link & kQLinkFirstMask);
      r.count = (int)((link >> kQLinkCountShift) & 15u) + 1;
    } else {
      r.child = (int)link;
      r.count = 0;
    }
  }
  return r;
}

// Slab test of one ray (device_ray.hpp:21-29 form).
__device__ __forceinline__ bool slab(float3 lo, float3 hi, float3 o, float3 idir, float t_min, float t_max,
                                     float &tnear) {
  float tx0 = (lo.x - o.x) * idir.x, tx1 = (hi.x - o.x) * idir.x;
  float ty0 = (lo.y - o.y) * idir.y, ty1 = (hi.y - o.y) * idir.y;
  float tz0 = (lo.z - o.z) * idir.z, tz1 = (hi.z - o.z) * idir.z;
  float tmin = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fminf(tz0, tz1));
  float tmax = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fmaxf(tz0, tz1));
  tmin = fmaxf(t_min, tmin);
  tmax = fminf(t_max, tmax);
  tnear = tmin;
  return tmax >= tmin;
}

// The rays of a warp as intervals of origin and inverse direction.  A child
// is entered when some ray of the box could hit it: every bound is an
// extreme of the same rounded operations each ray performs, so the packet
// never culls a node that one of its rays would enter.
//
// Packets use interval tests only when each axis' inverse direction keeps
// one sign across the packet.  Where a direction component changes sign
// inside the packet (near-axial rays, e.g. the image centre of a nadir
// camera) its inverse spans -1e20..1e20 and that axis culls nothing, so such
// packets take the per-ray path.
// A packet whose directions spread further per axis takes the per-ray tests: its interval bounds reach too many nodes.
// (346x260 frames at 60 degrees, 8 x 4 pixels a packet, 0.027: 0.263 ms with 0.02 here, 0.235 with 0.05 or 0.1; 64x48
// jobs lose from 0.1 on.)
constexpr float kCoherentSpread = 0.05f;
struct Packet {
  float3 olo, ohi, ilo, ihi;
  // per axis: the origin bound that gives the earliest entry (o_near) and
  // the latest exit (o_far), and whether the direction is negative
  float3 o_near, o_far;
  bool nx, ny, nz;
  bool coherent;
};
// Interval slab bounds of one axis for a packet whose inverse direction has
// one sign: the entry plane is the near one for every ray, and the extreme
// of the four corner products (lo/hi plane offset x ilo/ihi) is the one
// picked by the sign of the plane offset.  Rounded subtraction and
// multiplication are monotone, so L and U equal the four-product interval
// bounds (up to the sign of a zero) with a third of the arithmetic.
__device__ __forceinline__ void axis_bounds_fixed(float lo, float hi, bool neg, float on, float of, float ilo,
                                                  float ihi, float &L, float &U) {
  const float aN = (neg ? hi : lo) - on;
  const float aF = (neg ? lo : hi) - of;
  L = aN * (aN >= 0.0f ? ilo : ihi);
  U = aF * (aF >= 0.0f ? ihi : ilo);
}
__device__ __forceinline__ bool packet_slab(const ChildRec &c, const Packet &P, float t_min, float t_max,
                                            float &tnear) {
  float Lx, Ux, Ly, Uy, Lz, Uz;
  axis_bounds_fixed(c.lo.x, c.hi.x, P.nx, P.o_near.x, P.o_far.x, P.ilo.x, P.ihi.x, Lx, Ux);
  axis_bounds_fixed(c.lo.y, c.hi.y, P.ny, P.o_near.y, P.o_far.y, P.ilo.y, P.ihi.y, Ly, Uy);
  axis_bounds_fixed(c.lo.z, c.hi.z, P.nz, P.o_near.z, P.o_far.z, P.ilo.z, P.ihi.z, Lz, Uz);
  const float lb = fmaxf(fmaxf(fmaxf(Lx, Ly), Lz), t_min);
  const float ub = fminf(fminf(fminf(Ux, Uy), Uz), t_max);
  tnear = lb;
  return ub >= lb;
}
// Warp-uniform traversal stack in shared memory: node codes and the packet's
// entry distance.  Inner node: index >= 0; leaf: -(node * 8 + slot) - 1.
struct Stack {
  int *code;
  float *t;
  int sp;
};
__device__ __forceinline__ int leaf_code(int node, int slot) { return -(node * kBvhWidth + slot) - 1; }

struct HitRecord {
  int hit;  // 1 hit, 0 miss, -1 stack overflow (device_ray.hpp:152)
  int tri;
  float t, u, v;
};

// The float after a finite x in the direction of the sign of `to` (nextafterf toward +-infinity); x when `to` is zero.
__device__ __forceinline__ float next_toward(float x, float to) {
  const int b = __float_as_int(x);
  const int step = (b >= 0) == (to > 0) ? 1 : -1;
  const float y = x == 0.0f ? copysignf(__int_as_float(1), to) : __int_as_float(b + step);
  return to != 0 ? y : x;
}

// shadow_origin (device_optics.cuh:37-51) from the leaf-order triangle and shading records (normal: ShadeRecord::ng).
__device__ __forceinline__ float3 shadow_origin(float3 a, float3 e1, float3 e2, float3 normal, float u, float v,
                                                float3 light) {
  float3 point = a + u * e1 + v * e2;
  if (dot(normal, light) < 0) normal = -normal;
  constexpr float epsilon = 5.960464477539063e-8f, gamma = 8 * epsilon / (1 - 8 * epsilon);
  float3 error = f3(gamma * (fabsf(a.x) + fabsf(u * e1.x) + fabsf(v * e2.x)),
                    gamma * (fabsf(a.y) + fabsf(u * e1.y) + fabsf(v * e2.y)),
                    gamma * (fabsf(a.z) + fabsf(u * e1.z) + fabsf(v * e2.z)));
  float distance = fabsf(normal.x) * error.x + fabsf(normal.y) * error.y + fabsf(normal.z) * error.z + 1e-6f;
  float3 offset = normal * distance;
  point = point + offset;
  return f3(next_toward(point.x, offset.x), next_toward(point.y, offset.y), next_toward(point.z, offset.z));
}

// shadow_origin from a record (a, b, c = its three float4s): the edges are
// stored, or v1 - v0, v2 - v0 with the same float subtraction (watertight
// scenes), so both give the reference's edge bits.
template <int kGeo>
__device__ __forceinline__ float3 shadow_origin_rec(float4 a, float4 b, float4 c, float4 ng, float u, float v,
                                                    float3 light) {
  const float3 n = f3(ng.x, ng.y, ng.z);
  const float3 v0 = f3(a.x, a.y, a.z), p = f3(a.w, b.x, b.y), q = f3(b.z, b.w, c.x);
  if constexpr (!(kGeo & kGeoWatertight)) return shadow_origin(v0, p, q, n, u, v, light);
  else return shadow_origin(v0, p - v0, q - v0, n, u, v, light);
}

struct PixelSample {
  double radiance;
  float depth;
  bool valid;
  unsigned primary, shadow;
  bool redo;  // a ray left its item's beam: the sample has to be taken without it (warp-uniform)
};

// What one pixel sample produces.
enum SampleMode : int { kRadiance = 0, kRadianceDepth = 1 };

// cos^4 field falloff (device_optics.cuh:90) in FP64, as the reference.
__device__ __forceinline__ double cos4_of(float px, float py) {
  return 1.0 / ((1.0 + px * px + py * py) * (1.0 + px * px + py * py));
}
// One sub-ray of a pixel: its image-plane coordinates and FP64 cos^4, the
// same values subray_x/subray_y/cos4_of give.  A warp whose lanes all sample
// one pixel forms them once per sub-ray in shared memory instead of once per
// lane and ray (an integer division by the sub-ray count and four IEEE
// divisions per ray).
struct SubraySample {
  double cos4;
  float px, py;
};
__device__ __forceinline__ float subray_x(const SceneView &S, int px_i, int sx) {
  return (px_i + (sx + .5f) / S.samples - .5f - S.cx) / S.fx;
}
__device__ __forceinline__ float subray_y(const SceneView &S, int py_i, int sy) {
  return (py_i + (sy + .5f) / S.samples - .5f - S.cy) / S.fy;
}

// ---- packet walks: R sub-rays per lane ---------------------------------------------
// A packet is 32 x R rays: each lane carries R neighbouring sub-rays of its
// pixel-cell, so the interval node tests, the stack traffic and the packet
// set-up are paid once per 32 x R rays, and a leaf's triangle records are
// loaded once for the lane's R rays.  Per-ray results do not depend on R
// (every interval bound covers all R rays; leaves are tested per ray).

// Warp extremes of per-lane [lo, hi] ranges; inactive lanes count as empty.
__device__ __forceinline__ void wrange(float lo, float hi, bool active, float &wlo, float &whi) {
  wlo = funord(__reduce_min_sync(kFull, active ? ford(lo) : 0xff800000u));
  whi = funord(__reduce_max_sync(kFull, active ? ford(hi) : 0x007fffffu));
}

// The interval bundle of given ranges; coherent means each axis' inverse direction keeps one sign.
__device__ __forceinline__ Packet range_packet(float3 olo, float3 ohi, float3 ilo, float3 ihi) {
  Packet P;
  P.olo = olo; P.ohi = ohi; P.ilo = ilo; P.ihi = ihi;
  P.nx = ihi.x < 0.0f;
  P.ny = ihi.y < 0.0f;
  P.nz = ihi.z < 0.0f;
  P.coherent = (P.nx || ilo.x > 0.0f) && (P.ny || ilo.y > 0.0f) && (P.nz || ilo.z > 0.0f);
  P.o_near = f3(P.nx ? olo.x : ohi.x, P.ny ? olo.y : ohi.y, P.nz ? olo.z : ohi.z);
  P.o_far = f3(P.nx ? ohi.x : olo.x, P.ny ? ohi.y : olo.y, P.nz ? ohi.z : olo.z);
  return P;
}
template <int R>
__device__ Packet make_packet_r(const SceneView &S, const float3 (&o)[R], const float3 (&d)[R],
                                const float3 (&idir)[R], const bool (&active)[R]) {
  float3 olo = f3(kInf(), kInf(), kInf()), ohi = -olo, ilo = olo, ihi = -olo, dlo = olo, dhi = -olo;
  bool any = false;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (active[r]) {
      any = true;
      olo = f3(fminf(olo.x, o[r].x), fminf(olo.y, o[r].y), fminf(olo.z, o[r].z));
      ohi = f3(fmaxf(ohi.x, o[r].x), fmaxf(ohi.y, o[r].y), fmaxf(ohi.z, o[r].z));
      ilo = f3(fminf(ilo.x, idir[r].x), fminf(ilo.y, idir[r].y), fminf(ilo.z, idir[r].z));
      ihi = f3(fmaxf(ihi.x, idir[r].x), fmaxf(ihi.y, idir[r].y), fmaxf(ihi.z, idir[r].z));
      dlo = f3(fminf(dlo.x, d[r].x), fminf(dlo.y, d[r].y), fminf(dlo.z, d[r].z));
      dhi = f3(fmaxf(dhi.x, d[r].x), fmaxf(dhi.y, d[r].y), fmaxf(dhi.z, d[r].z));
    }
  wrange(olo.x, ohi.x, any, olo.x, ohi.x);
  wrange(olo.y, ohi.y, any, olo.y, ohi.y);
  wrange(olo.z, ohi.z, any, olo.z, ohi.z);
  wrange(ilo.x, ihi.x, any, ilo.x, ihi.x);
  wrange(ilo.y, ihi.y, any, ilo.y, ihi.y);
  wrange(ilo.z, ihi.z, any, ilo.z, ihi.z);
  float wl, wh;
  wrange(dlo.x, dhi.x, any, wl, wh);
  const float dx = wh - wl;
  wrange(dlo.y, dhi.y, any, wl, wh);
  const float dy = wh - wl;
  wrange(dlo.z, dhi.z, any, wl, wh);
  const float dz = wh - wl;
  const float ds = fmaxf(fmaxf(dx, dy), dz);
  const float os = fmaxf(fmaxf(ohi.x - olo.x, ohi.y - olo.y), ohi.z - olo.z);
  Packet P = range_packet(olo, ohi, ilo, ihi);
  P.coherent = P.coherent && ds <= kCoherentSpread && os <= S.coherent_span;
  return P;
}

// Expands an inner node: children the packet may hit are ordered near to far;
// all but the nearest go on the stack.  Returns false when none is hit.
// Coherent packets test one child per lane (lanes 0..7) with interval bounds;
// others test every child per ray and take the warp minimum as the key.
template <bool kSorted, int R, int kGeo>
__device__ __forceinline__ bool expand_node_r(const SceneView &S, int node, const Packet &P, const float3 (&o)[R],
                                              const float3 (&idir)[R], const bool (&live)[R], float t_min,
                                              const float (&lane_tmax)[R], float packet_tmax, Stack &st, int &next,
                                              float &next_t, bool &overflow) {
  const int lane = threadIdx.x & 31;
  float key = kInf();
  bool hit = false;
  int code = 0;
  if (P.coherent) {
    if (lane < kBvhWidth) {
      const ChildRec c = load_child<kGeo>(S, node, lane);
      if (c.count >= 0) {
        hit = packet_slab(c, P, t_min, packet_tmax, key);
        code = c.count > 0 ? leaf_code(node, lane) : c.child;
      }
    }
  } else {
    for (int slot = 0; slot < kBvhWidth; ++slot) {
      const ChildRec c = load_child<kGeo>(S, node, slot);
      float near = kInf();
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float tn = kInf();
        if (c.count >= 0 && live[r] && slab(c.lo, c.hi, o[r], idir[r], t_min, lane_tmax[r], tn)) near = fminf(near, tn);
      }
      const float k = wmin(near);
      if (lane == slot) {
        hit = k < kInf();
        key = k;
        code = c.count > 0 ? leaf_code(node, slot) : c.child;
      }
    }
  }
  const unsigned mask = __ballot_sync(kFull, hit && lane < kBvhWidth);
  if (!mask) return false;
  const int n = __popc(mask);
  if (n == 1) {
    const int only = __ffs(mask) - 1;
    next = __shfl_sync(kFull, code, only);
    next_t = __shfl_sync(kFull, key, only);
    return true;
  }
  int rank = 0;
  if (kSorted) {
#pragma unroll
    for (int j = 0; j < kBvhWidth; ++j) {
      const float kj = __shfl_sync(kFull, key, j);
      rank += ((mask >> j) & 1) && (kj < key || (kj == key && j < lane)) ? 1 : 0;
    }
  } else {
    rank = __popc(mask & ((1u << lane) - 1u));
  }
  if (st.sp + n - 1 > kStackSlots) {
    overflow = true;
    return false;
  }
  if (hit && lane < kBvhWidth && rank > 0) {
    const int slot = st.sp + (n - 1 - rank);
    st.code[slot] = code;
    st.t[slot] = key;
  }
  const int first = __ffs(__ballot_sync(kFull, hit && lane < kBvhWidth && rank == 0)) - 1;
  next = __shfl_sync(kFull, code, first);
  next_t = __shfl_sync(kFull, key, first);
  st.sp += n - 1;
  __syncwarp();
  return true;
}

template <int R>
__device__ __forceinline__ float lane_reach(const bool (&active)[R], const float (&closest)[R]) {
  float m = -1.0f;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (active[r]) m = fmaxf(m, closest[r]);
  return m;
}

// Nearest hits of a packet (trace_nearest, device_ray.hpp:136-158).  All 32
// lanes call converged; inactive rays never hit.  Each ray is tested against a
// leaf's triangles only when its own slab test reaches the leaf.
template <int R, int kGeo>
__device__ void trace_nearest_packet_r(const SceneView &S, const float3 (&o)[R], const float3 (&d)[R],
                                       const bool (&active)[R], int *stack_code, float *stack_t, HitRecord (&h)[R]) {
  float3 idir[R], op[R];
  float closest[R];
  WtRay wr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    idir[r] = inverse_direction(d[r]);
    wr[r] = wt_ray<kGeo>(d[r]);
    op[r] = wt_origin<kGeo>(wr[r], o[r]);
    closest[r] = active[r] ? 1e30f : -1.0f;
    h[r] = HitRecord{0, -1, 0.f, 0.f, 0.f};
  }
  const Packet P = make_packet_r<R>(S, o, d, idir, active);
  float packet_tmax = wmax(lane_reach<R>(active, closest));
  Stack st{stack_code, stack_t, 0};
  int entry = 0;
  float entry_t = 0.0f;
  bool overflow = false;
  while (true) {
    if (entry_t <= packet_tmax) {
      if (entry >= 0) {
        int next;
        float next_t;
        if (expand_node_r<true, R, kGeo>(S, entry, P, o, idir, active, kRayEps, closest, packet_tmax, st, next, next_t,
                                   overflow)) {
          entry = next;
          entry_t = next_t;
          continue;
        }
        if (overflow) break;
      } else {
        const int lc = -entry - 1;
        const ChildRec c = load_child<kGeo>(S, lc / kBvhWidth, lc % kBvhWidth);
        bool need[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float tn;
          need[r] = active[r] && slab(c.lo, c.hi, o[r], idir[r], kRayEps, closest[r], tn);
        }
        for (int i = 0; i < c.count; ++i) {
          // one record per lane for all its rays; a ray of another dominant
          // axis (watertight scenes, rare inside a lane) reads its own copy
          const float4 *q4 = tri_record<kGeo>(S, c.child + i, wr[0].kz);
          float4 a = __ldg(q4), b = __ldg(q4 + 1), q = __ldg(q4 + 2);
          int loaded = wr[0].kz;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if constexpr ((kGeo & kGeoWatertight) != 0) {
              if (wr[r].kz != loaded) {
                const float4 *p4 = tri_record<kGeo>(S, c.child + i, wr[r].kz);
                a = __ldg(p4);
                b = __ldg(p4 + 1);
                q = __ldg(p4 + 2);
                loaded = wr[r].kz;
              }
            }
            float t, u, v;
            if (need[r] && tri_hit<kGeo>(wr[r], d[r], o[r], op[r], a, b, q, t, u, v) && t < closest[r]) {
              closest[r] = t;
              h[r].hit = 1; h[r].tri = c.child + i; h[r].t = t; h[r].u = u; h[r].v = v;
            }
          }
        }
        packet_tmax = wmax(lane_reach<R>(active, closest));
      }
    }
    if (st.sp == 0) break;
    --st.sp;
    entry = st.code[st.sp];
    entry_t = st.t[st.sp];
  }
  __syncwarp();
  if (overflow)
#pragma unroll
    for (int r = 0; r < R; ++r) h[r].hit = -1;
}

// The direction terms of a lane's shadow rays (all toward the same light):
// formed once per pixel sample loop, not once per shadow packet.
struct ShadowDir {
  float3 idir;
  WtRay wr;
};
template <int kGeo>
__device__ __forceinline__ ShadowDir shadow_dir(float3 light) {
  return ShadowDir{inverse_direction(light), wt_ray<kGeo>(light)};
}

// Any hit toward the light (trace_shadow_ray_any_hit, device_ray.hpp:81-135):
// skips the camera-hit triangle, t in (kRayEps, 1e30); overflow counts as occluded.
template <int R, int kGeo>
__device__ void trace_shadow_packet_r(const SceneView &S, const float3 (&o)[R], float3 light, const ShadowDir &sd,
                                      const bool (&active)[R], const int (&self)[R], int *stack_code, float *stack_t,
                                      bool (&occluded)[R]) {
  const float3 idir1 = sd.idir;
  const WtRay wr = sd.wr;
  float3 d[R], idir[R], op[R];
  bool alive[R];
  float reach[R];
  const float t_max = 1e30f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    d[r] = light;
    idir[r] = idir1;
    op[r] = wt_origin<kGeo>(wr, o[r]);
    alive[r] = active[r];
    occluded[r] = false;
  }
  const Packet P = make_packet_r<R>(S, o, d, idir, active);
  Stack st{stack_code, stack_t, 0};
  int entry = 0;
  bool overflow = false;
  while (true) {
    bool any = false;
#pragma unroll
    for (int r = 0; r < R; ++r) any = any || alive[r];
    if (!__any_sync(kFull, any)) break;
    if (entry >= 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) reach[r] = alive[r] ? t_max : -1.0f;
      int next;
      float next_t;
      if (expand_node_r<false, R, kGeo>(S, entry, P, o, idir, alive, kRayEps, reach, t_max, st, next, next_t, overflow)) {
        entry = next;
        continue;
      }
      if (overflow) {
#pragma unroll
        for (int r = 0; r < R; ++r) occluded[r] = occluded[r] || alive[r];  // conservative (device_ray.hpp:119)
        break;
      }
    } else {
      const int lc = -entry - 1;
      const ChildRec c = load_child<kGeo>(S, lc / kBvhWidth, lc % kBvhWidth);
      bool need[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float tn;
        need[r] = alive[r] && slab(c.lo, c.hi, o[r], idir[r], kRayEps, t_max, tn);
      }
      for (int i = 0; i < c.count; ++i) {
        const int id = c.child + i;
        const float4 *q4 = tri_record<kGeo>(S, id, wr.kz);
        const float4 a = __ldg(q4), b = __ldg(q4 + 1), q = __ldg(q4 + 2);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float t, u, v;
          if (need[r] && alive[r] && id != self[r] && tri_hit<kGeo>(wr, light, o[r], op[r], a, b, q, t, u, v) &&
              t > kRayEps && t < t_max) {
            occluded[r] = true;
            alive[r] = false;
          }
        }
      }
    }
    if (st.sp == 0) break;
    --st.sp;
    entry = st.code[st.sp];
  }
  __syncwarp();
}

// ---- beams: one walk of the tree for all the packets of a warp's item -------------------
// A warp's item is many packets through nearly the same rays: every sub-ray of
// a pixel (or of a few neighbouring pixels) at many circuit cells.  Walking the
// tree from the root for each packet repeats the same node tests: on the
// 1280x720 workload they were more than half of the trace's instructions, all
// of them in one dependent chain of load, test and vote per level.  So the
// warp walks the tree once for the bundle of all its rays (the beam) and keeps
// the leaves the bundle may reach, decoded and sorted by entry distance, in
// shared memory; each packet then tests only these.  A second list holds the
// leaves between the beam's hit points and the light.
//
// The lists change which leaves are looked at, not what a ray hits: a leaf's
// triangles are tested after the ray's own slab test as before, and a leaf that is
// not in the list is one that the ray's slab test fails (the beam's interval bounds
// are extremes of the same rounded operations).  Only where two triangles are hit
// at exactly the same distance (a common edge, a triangle that lies twice in the
// mesh) may the list's order find the other one first.  What the beam assumes of
// a ray -- its direction, or its shadow origin, inside the beam's ranges -- is
// checked for every ray, and a sample with a ray outside is taken again by walks
// from the root.  An item whose beam reaches more leaves than a list holds has no
// lists and walks the tree for every packet, two sub-rays per lane.
constexpr int kBeamLeaves = 32;  // one per lane
struct Beam {                    // shared memory, one per warp
  float4 leaf[kBeamLeaves][2];   // {lo, hi.x}, {hi.y, hi.z, first triangle, count}, nearest entry first
  float4 shadow[kBeamLeaves][2];
  float3 olo, ohi, dlo, dhi;     // ranges of the rays' origins and directions
  float3 llo, lhi;               // range of the light directions' inverses
  float3 slo, shi;               // range of the shadow origins
};
// What a warp holds of its item's lists: their lengths, and where shadow_in_list starts.
struct BeamLists {
  int leaves, shadow, first;
};
constexpr int kNoList = -1;  // a list's length when there is none

__device__ __forceinline__ float3 min3(float3 a, float3 b) { return f3(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z)); }
__device__ __forceinline__ float3 max3(float3 a, float3 b) { return f3(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z)); }
__device__ __forceinline__ bool within(float3 v, float3 lo, float3 hi) {
  return v.x >= lo.x && v.x <= hi.x && v.y >= lo.y && v.y <= hi.y && v.z >= lo.z && v.z <= hi.z;
}
__device__ __forceinline__ float3 wmin3(float3 v) { return f3(wmin(v.x), wmin(v.y), wmin(v.z)); }
__device__ __forceinline__ float3 wmax3(float3 v) { return f3(wmax(v.x), wmax(v.y), wmax(v.z)); }

// The primary beam's bundle: 1/d of directions of one sign decreases with d, so the ends of the inverse's range are
// the inverses of the ends, rounded outward by more than rcp_rn's last bit.  On an axis whose range holds zero (or
// comes so near it that inverse_direction could clamp: the rows and columns of pixels that look along a coordinate
// plane) the inverse has no range, and leaf boxes are tested there by position: where the rays are on that
// axis between the entry and the exit that the other axes give.
__device__ __forceinline__ float rcp_low(float d) { const float y = 1.0f / d; return y - 2.4e-7f * fabsf(y); }
__device__ __forceinline__ float rcp_high(float d) { const float y = 1.0f / d; return y + 2.4e-7f * fabsf(y); }
__device__ __forceinline__ bool one_sign(float lo, float hi) { return lo > 1e-18f || hi < -1e-18f; }
struct PrimaryBundle {
  Packet P;
  bool tx, ty, tz;  // axes whose inverse direction keeps one sign
};
__device__ __forceinline__ PrimaryBundle primary_bundle(const Beam &B) {
  const float3 dlo = B.dlo, dhi = B.dhi;
  PrimaryBundle b;
  b.P = range_packet(B.olo, B.ohi, f3(rcp_low(dhi.x), rcp_low(dhi.y), rcp_low(dhi.z)),
                     f3(rcp_high(dlo.x), rcp_high(dlo.y), rcp_high(dlo.z)));
  b.tx = one_sign(dlo.x, dhi.x);
  b.ty = one_sign(dlo.y, dhi.y);
  b.tz = one_sign(dlo.z, dhi.z);
  b.P.coherent = b.tx || b.ty || b.tz;
  return b;
}
// Whether rays between entry and exit distance can be inside [lo, hi] on an axis; the margin covers the roundings of a
// ray's own slab test (three of them on a distance, one on a coordinate).
__device__ __forceinline__ bool passes(float lo, float hi, float olo, float ohi, float dlo, float dhi, float entry,
                                       float exit) {
  const float a = olo + fminf(entry * dlo, exit * dlo), b = ohi + fmaxf(entry * dhi, exit * dhi);
  const float m = 2e-6f * (fmaxf(fabsf(a), fabsf(b)) + fmaxf(fabsf(olo), fabsf(ohi)) + fmaxf(fabsf(lo), fabsf(hi)));
  return b + m >= lo && a - m <= hi;
}
// The beam's entry and exit distance at a box, and whether one of its rays may enter it.
__device__ __forceinline__ bool bundle_slab(const ChildRec &c, const PrimaryBundle &b, const Beam &B, float &entry,
                                            float &exit) {
  const Packet &P = b.P;
  float L, U;
  entry = kRayEps;
  exit = 1e30f;
  if (b.tx) {
    axis_bounds_fixed(c.lo.x, c.hi.x, P.nx, P.o_near.x, P.o_far.x, P.ilo.x, P.ihi.x, L, U);
    entry = fmaxf(entry, L);
    exit = fminf(exit, U);
  }
  if (b.ty) {
    axis_bounds_fixed(c.lo.y, c.hi.y, P.ny, P.o_near.y, P.o_far.y, P.ilo.y, P.ihi.y, L, U);
    entry = fmaxf(entry, L);
    exit = fminf(exit, U);
  }
  if (b.tz) {
    axis_bounds_fixed(c.lo.z, c.hi.z, P.nz, P.o_near.z, P.o_far.z, P.ilo.z, P.ihi.z, L, U);
    entry = fmaxf(entry, L);
    exit = fminf(exit, U);
  }
  return exit >= entry && (b.tx || passes(c.lo.x, c.hi.x, P.olo.x, P.ohi.x, B.dlo.x, B.dhi.x, entry, exit)) &&
         (b.ty || passes(c.lo.y, c.hi.y, P.olo.y, P.ohi.y, B.dlo.y, B.dhi.y, entry, exit)) &&
         (b.tz || passes(c.lo.z, c.hi.z, P.olo.z, P.ohi.z, B.dlo.z, B.dhi.z, entry, exit));
}
__device__ __forceinline__ ChildRec list_leaf(const float4 (*list)[2], int i) {
  const float4 a = list[i][0], b = list[i][1];
  return ChildRec{f3(a.x, a.y, a.z), f3(a.w, b.x, b.y), __float_as_int(b.z), __float_as_int(b.w)};
}

// The leaves a bundle may reach, in no order: up to four nodes at a time, one
// child per lane (reaches: whether the bundle may enter its box).  Returns their
// number, kNoList when they are more than the list holds.
template <int kGeo, class Test>
__device__ __forceinline__ int collect_leaves(const SceneView &S, const Test &reaches, int *stack, float4 (*list)[2]) {
  const int lane = threadIdx.x & 31, group = lane >> 3, slot = lane & 7;
  const unsigned below = (1u << lane) - 1u;
  int sp = 1, n = 0;
  if (lane == 0) stack[0] = 0;
  __syncwarp();
  while (sp > 0) {
    const int take = min(sp, 4);
    sp -= take;
    const int node = group < take ? stack[sp + group] : -1;
    ChildRec c{};
    bool hit = false;
    if (node >= 0) {
      c = load_child<kGeo>(S, node, slot);
      hit = c.count >= 0 && reaches(c);
    }
    const unsigned leaves = __ballot_sync(kFull, hit && c.count > 0);
    const unsigned inner = __ballot_sync(kFull, hit && c.count == 0);
    const int nl = __popc(leaves), ni = __popc(inner);
    if (n + nl > kBeamLeaves || sp + ni > kStackSlots) {
      __syncwarp();
      return kNoList;
    }
    if (hit) {
      if (c.count > 0) {
        float4 *q = list[n + __popc(leaves & below)];
        q[0] = make_float4(c.lo.x, c.lo.y, c.lo.z, c.hi.x);
        q[1] = make_float4(c.hi.y, c.hi.z, __int_as_float(c.child), __int_as_float(c.count));
      } else {
        stack[sp + __popc(inner & below)] = c.child;  // the nodes read above are below or in other lanes' registers
      }
    }
    n += nl;
    sp += ni;
    __syncwarp();
  }
  return n;
}

// The primary list: the beam's leaves by entry distance (ties in walk order).
template <int kGeo>
__device__ __forceinline__ int build_primary_list(const SceneView &S, Beam &B, int *stack) {
  const PrimaryBundle bundle = primary_bundle(B);
  if (!bundle.P.coherent) return kNoList;
  const int n = collect_leaves<kGeo>(
      S, [&](const ChildRec &c) { float entry, exit; return bundle_slab(c, bundle, B, entry, exit); }, stack, B.leaf);
  if (n > 1) {
    const int lane = threadIdx.x & 31;
    float4 a, b;
    float key = kInf();
    if (lane < n) {
      a = B.leaf[lane][0];
      b = B.leaf[lane][1];
      float exit;
      bundle_slab(list_leaf(B.leaf, lane), bundle, B, key, exit);
    }
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const float kj = __shfl_sync(kFull, key, j);
      rank += kj < key || (kj == key && j < lane) ? 1 : 0;
    }
    __syncwarp();
    if (lane < n) {
      B.leaf[rank][0] = a;
      B.leaf[rank][1] = b;
    }
    __syncwarp();
  }
  return n;
}

// The shadow list.  The shadow origins lie on the list's triangles inside the
// beam: per leaf the beam's entry and exit distance bound the hit points, cut to
// the leaf's box; the margin covers the float hit point and shadow_origin's offset
// (packets check their origins against the range).
template <int kGeo>
__device__ __forceinline__ int build_shadow_list(const SceneView &S, Beam &B, int n_leaf, int *stack) {
  const int lane = threadIdx.x & 31;
  const PrimaryBundle bundle = primary_bundle(B);
  float3 lo = f3(kInf(), kInf(), kInf()), hi = -lo;
  if (lane < n_leaf) {
    const ChildRec c = list_leaf(B.leaf, lane);
    float t0, t1;
    bundle_slab(c, bundle, B, t0, t1);
    t1 = fmaxf(t0, t1);
    const float3 dlo = B.dlo, dhi = B.dhi;
    lo = max3(c.lo, B.olo + min3(t0 * dlo, t1 * dlo));
    hi = min3(c.hi, B.ohi + max3(t0 * dhi, t1 * dhi));
    const float m = 3e-6f * fmaxf(fmaxf(fmaxf(fabsf(c.lo.x), fabsf(c.hi.x)), fmaxf(fabsf(c.lo.y), fabsf(c.hi.y))),
                                  fmaxf(fabsf(c.lo.z), fabsf(c.hi.z))) + 1e-5f;
    lo = lo - f3(m, m, m);
    hi = hi + f3(m, m, m);
  }
  lo = wmin3(lo);
  hi = wmax3(hi);
  if (lane == 0) {
    B.slo = lo;
    B.shi = hi;
  }
  __syncwarp();
  const Packet L = range_packet(lo, hi, B.llo, B.lhi);
  if (!L.coherent) return kNoList;
  return collect_leaves<kGeo>(
      S, [&](const ChildRec &c) { float key; return packet_slab(c, L, kRayEps, 1e30f, key); }, stack, B.shadow);
}

// A longer list is first cut to the leaves the packet's own interval bundle may reach, one leaf per lane: the bundle's
// extremes and the test cost about as much as five leaves tested by every ray.
constexpr int kListFilter = 5;
__device__ __forceinline__ unsigned list_mask(const float4 (*list)[2], int n, const Packet &P) {
  const int lane = threadIdx.x & 31;
  bool hit = false;
  if (lane < n) {
    float key;
    hit = packet_slab(list_leaf(list, lane), P, kRayEps, 1e30f, key);
  }
  return __ballot_sync(kFull, hit);
}
__device__ __forceinline__ unsigned whole_list(int n) { return n >= 32 ? kFull : (1u << n) - 1u; }
// The extremes of a packet's R vectors per lane, live ones only.
template <int R>
__device__ __forceinline__ void packet_range(const float3 (&v)[R], const bool (&live)[R], float3 &lo, float3 &hi) {
  lo = f3(kInf(), kInf(), kInf());
  hi = -lo;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (live[r]) {
      lo = min3(lo, v[r]);
      hi = max3(hi, v[r]);
    }
  lo = wmin3(lo);
  hi = wmax3(hi);
}

// A wider bundle of directions (the sum of its extents per axis) takes no beam.
constexpr float kBeamSpread = 0.1f;
// A beam and its lists from each lane's ranges of origins, directions and
// inverse light directions; reach: what the rays' origins and light directions may leave the
// ranges by, as a share of their extent.
template <int kGeo>
__device__ __forceinline__ BeamLists close_beam(const SceneView &S, float3 olo, float3 ohi, float3 dlo, float3 dhi,
                                                float3 llo, float3 lhi, float reach, Beam &B, int *stack) {
  olo = wmin3(olo);
  ohi = wmax3(ohi);
  dlo = wmin3(dlo);
  dhi = wmax3(dhi);
  llo = wmin3(llo);
  lhi = wmax3(lhi);
  const float ext = (dhi.x - dlo.x) + (dhi.y - dlo.y) + (dhi.z - dlo.z);
  BeamLists lists{kNoList, kNoList, 0};
  if (!(ext <= kBeamSpread)) return lists;  // a wide bundle reaches too many leaves (or a ray has no direction)
  const float m = ext * ext + 4e-7f;
  if (reach > 0.0f) {
    const float3 a = max3(-olo, ohi), o = reach * (ohi - olo) + 5e-7f * max3(a, -a);
    const float3 b = max3(-llo, lhi), l = reach * (lhi - llo) + 5e-7f * max3(b, -b);
    olo = olo - o;
    ohi = ohi + o;
    llo = llo - l;
    lhi = lhi + l;
  }
  if ((threadIdx.x & 31) == 0) {
    B.olo = olo;
    B.ohi = ohi;
    B.dlo = dlo - f3(m, m, m);
    B.dhi = dhi + f3(m, m, m);
    B.llo = llo;
    B.lhi = lhi;
  }
  __syncwarp();
  lists.leaves = build_primary_list<kGeo>(S, B, stack);
  if (lists.leaves >= 0) lists.shadow = build_shadow_list<kGeo>(S, B, lists.leaves, stack);
  return lists;
}

// The general walks, out of line: they serve the packets no list holds for.
template <int R>
struct PacketRays {
  float3 o[R], d[R];
  bool live[R];
};
template <int R>
struct PacketHits {
  HitRecord h[R];
};
template <int R, int kGeo>
__device__ __noinline__ PacketHits<R> nearest_general(const SceneView &S, PacketRays<R> in, int *stack_code,
                                                      float *stack_t) {
  PacketHits<R> out;
  trace_nearest_packet_r<R, kGeo>(S, in.o, in.d, in.live, stack_code, stack_t, out.h);
  return out;
}
template <int R>
struct ShadowRays {
  float3 o[R], light;
  int self[R];
  bool live[R];
};
template <int R, int kGeo>
__device__ __noinline__ unsigned shadow_general(const SceneView &S, ShadowRays<R> in, int *stack_code,
                                                float *stack_t) {
  bool occ[R];
  trace_shadow_packet_r<R, kGeo>(S, in.o, in.light, shadow_dir<kGeo>(in.light), in.live, in.self, stack_code, stack_t,
                                 occ);
  unsigned m = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) m |= occ[r] ? 1u << r : 0u;
  return m;
}

// Nearest hits of a packet from the beam's list (trace_nearest_packet_r's leaves, nearest first).
template <int R, int kGeo>
__device__ __forceinline__ void nearest_in_list(const SceneView &S, const Beam &B, int n, float3 o,
                                                const float3 (&d)[R], const bool (&live)[R], HitRecord (&h)[R]) {
  float3 idir[R], op[R];
  float closest[R];
  WtRay wr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    idir[r] = inverse_direction(d[r]);
    wr[r] = wt_ray<kGeo>(d[r]);
    op[r] = wt_origin<kGeo>(wr[r], o);
    closest[r] = live[r] ? 1e30f : -1.0f;
    h[r] = HitRecord{0, -1, 0.f, 0.f, 0.f};
  }
  unsigned left = whole_list(n);
  if (n > kListFilter) {
    float3 ilo, ihi;
    packet_range<R>(idir, live, ilo, ihi);
    const Packet P = range_packet(B.olo, B.ohi, ilo, ihi);
    if (P.coherent) left = list_mask(B.leaf, n, P);
  }
  for (; left; left &= left - 1u) {
    const ChildRec c = list_leaf(B.leaf, __ffs(left) - 1);
    bool need[R], any = false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float tn;
      need[r] = live[r] && slab(c.lo, c.hi, o, idir[r], kRayEps, closest[r], tn);
      any = any || need[r];
    }
    if (!__any_sync(kFull, any)) continue;
    for (int k = 0; k < c.count; ++k) {
      const float4 *q4 = tri_record<kGeo>(S, c.child + k, wr[0].kz);
      float4 a = __ldg(q4), b = __ldg(q4 + 1), q = __ldg(q4 + 2);
      int loaded = wr[0].kz;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if constexpr ((kGeo & kGeoWatertight) != 0) {
          if (wr[r].kz != loaded) {
            const float4 *p4 = tri_record<kGeo>(S, c.child + k, wr[r].kz);
            a = __ldg(p4);
            b = __ldg(p4 + 1);
            q = __ldg(p4 + 2);
            loaded = wr[r].kz;
          }
        }
        float t, u, v;
        if (need[r] && tri_hit<kGeo>(wr[r], d[r], o, op[r], a, b, q, t, u, v) && t < closest[r]) {
          closest[r] = t;
          h[r].hit = 1; h[r].tri = c.child + k; h[r].t = t; h[r].u = u; h[r].v = v;
        }
      }
    }
  }
}

// Occlusion of a packet's shadow rays from the shadow list; `first`: where to
// start, the leaf that last occluded a ray of this item (any hit ends a ray,
// so the order decides nothing but the time).
template <int R, int kGeo>
__device__ __forceinline__ unsigned shadow_in_list(const SceneView &S, const Beam &B, int n, const float3 (&o)[R],
                                                   float3 light, const ShadowDir &sd, const bool (&live)[R],
                                                   const int (&self)[R], int &first) {
  const float t_max = 1e30f;
  unsigned occluded = 0;
  float3 op[R];
  bool alive[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    op[r] = wt_origin<kGeo>(sd.wr, o[r]);
    alive[r] = live[r];
  }
  unsigned left = whole_list(n);
  if (n > kListFilter) {
    float3 olo, ohi;
    packet_range<R>(o, live, olo, ohi);
    left = list_mask(B.shadow, n, range_packet(olo, ohi, B.llo, B.lhi));
  }
  left = __funnelshift_r(left, left, first);  // bit j: leaf (first + j) mod 32
  const int start = first;
  for (; left; left &= left - 1u) {
    const int i = (start + __ffs(left) - 1) & 31;
    const ChildRec c = list_leaf(B.shadow, i);
    bool need[R], any = false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float tn;
      need[r] = alive[r] && slab(c.lo, c.hi, o[r], sd.idir, kRayEps, t_max, tn);
      any = any || need[r];
    }
    if (__any_sync(kFull, any)) {
      const unsigned before = occluded;
      for (int k = 0; k < c.count; ++k) {
        const int id = c.child + k;
        const float4 *q4 = tri_record<kGeo>(S, id, sd.wr.kz);
        const float4 a = __ldg(q4), b = __ldg(q4 + 1), q = __ldg(q4 + 2);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float t, u, v;
          if (need[r] && alive[r] && id != self[r] &&
              tri_hit<kGeo>(sd.wr, light, o[r], op[r], a, b, q, t, u, v) && t > kRayEps && t < t_max) {
            occluded |= 1u << r;
            alive[r] = false;
          }
        }
      }
      if (__any_sync(kFull, occluded != before)) {
        first = i;
        bool some = false;
#pragma unroll
        for (int r = 0; r < R; ++r) some = some || alive[r];
        if (!__any_sync(kFull, some)) break;
      }
    }
  }
  return occluded;
}

// sample_pixel (device_optics.cuh:73-94) for one lane of a converged warp, R
// neighbouring sub-rays at a time (ss^2 a multiple of R).  The order of the FP64
// radiance and depth sums and the ray counts do not depend on R.
// subrays: the sub-rays' coordinates and cos^4, formed once per pixel (shared memory), or nullptr.
// kBeam: the item has lists, and the packets' leaves come from them; a ray
// outside the beam ends the sample (redo).  The loop then holds no call, whose
// registers would be spilled around it.
template <int kMode, int R, int kGeo, bool kBeam>
__device__ __forceinline__ PixelSample sample_pixel_group(const SceneView &S, int pixel, bool active,
                                                          const CellPose &pose, int *stack_code, float *stack_t,
                                                          const SubraySample *subrays, const Beam *beam,
                                                          BeamLists *lists) {
  PixelSample out{0.0, -1.0f, true, 0u, 0u, false};
  double depth = 0;
  int valid_depth = 0;
  const float3 light = f3(pose.lx, pose.ly, pose.lz);
  const float3 origin = f3(pose.px, pose.py, pose.pz);
  const int ss = S.samples, n_sub = ss * ss;
  const int px_i = pixel % S.width, py_i = pixel / S.width;
  const HapkeConst &hc = S.hc;
  // hapke_directional_reflectance normalizes the light for every shaded ray
  // (hapke.hpp:153-157); it is the same vector for all of this lane's rays
  const float3 lnorm = unit(light);
  const ShadowDir sdir = shadow_dir<kGeo>(light);
  for (int j = 0; j < n_sub; j += R) {
    float px[R], py[R];
    float3 ray[R];
    bool live[R], inside = true;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (subrays) {
        px[r] = subrays[j + r].px;
        py[r] = subrays[j + r].py;
      } else {
        const int sx = (j + r) % ss, sy = (j + r) / ss;
        px[r] = subray_x(S, px_i, sx);
        py[r] = subray_y(S, py_i, sy);
      }
      ray[r] = unit(rotate_ray(pose, f3(px[r], -py[r], -1)));
      live[r] = active && out.valid;
      if constexpr (kBeam) inside = inside && (!live[r] || within(ray[r], beam->dlo, beam->dhi));
    }
    HitRecord hit[R];
    if constexpr (!kBeam) {
      float3 org[R];
#pragma unroll
      for (int r = 0; r < R; ++r) org[r] = origin;
      trace_nearest_packet_r<R, kGeo>(S, org, ray, live, stack_code, stack_t, hit);
    } else {
      if (!__all_sync(kFull, inside)) {
        out.redo = true;
        return out;
      }
      nearest_in_list<R, kGeo>(S, *beam, lists->leaves, origin, ray, live, hit);
    }
    bool lit[R];
    float3 normal[R], sorigin[R];
    float albedo[R], r0[R];
    int self[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (active && out.valid) ++out.primary;
      if (hit[r].hit < 0) out.valid = false;
      const bool hitp = active && out.valid && hit[r].hit == 1;
      lit[r] = false;
      normal[r] = f3(0, 0, 0);
      sorigin[r] = f3(0, 0, 0);
      albedo[r] = S.hc.w;
      r0[r] = hc.r0_w;
      self[r] = hit[r].tri;
      if (hitp) {
        if (kMode != kRadiance) {
          depth += hit[r].t;
          ++valid_depth;
        }
        const float4 *q = reinterpret_cast<const float4 *>(S.shade + hit[r].tri);
        const float4 s0 = __ldg(q), s1 = __ldg(q + 1), s2 = __ldg(q + 2);
        const float w = 1 - hit[r].u - hit[r].v;
        normal[r] =
            unit(f3(s0.x, s0.y, s0.z) * w + f3(s1.x, s1.y, s1.z) * hit[r].u + f3(s2.x, s2.y, s2.z) * hit[r].v);
        lit[r] = !(dot(normal[r], light) <= 0 || dot(normal[r], -ray[r]) <= 0);
        if (lit[r]) {
          const float4 *t4 = tri_record<kGeo>(S, hit[r].tri, 2);
          const float4 a = __ldg(t4), b = __ldg(t4 + 1), c = __ldg(t4 + 2);
          sorigin[r] = shadow_origin_rec<kGeo>(a, b, c, __ldg(q + 3), hit[r].u, hit[r].v, light);
          if (S.has_albedo) {
            albedo[r] = s0.w * w + s1.w * hit[r].u + s2.w * hit[r].v;
            r0[r] = hfunc_r0(albedo[r]);
          }
        }
      }
    }
    bool any_lit = false;
#pragma unroll
    for (int r = 0; r < R; ++r) any_lit = any_lit || lit[r];
    if (__any_sync(kFull, any_lit)) {
      unsigned occluded = 0;
      bool near = true;
      if constexpr (kBeam) {
#pragma unroll
        for (int r = 0; r < R; ++r) near = near && (!lit[r] || within(sorigin[r], beam->slo, beam->shi));
      }
      if constexpr (!kBeam) {
        bool occ[R];
        trace_shadow_packet_r<R, kGeo>(S, sorigin, light, sdir, lit, self, stack_code, stack_t, occ);
#pragma unroll
        for (int r = 0; r < R; ++r) occluded |= occ[r] ? 1u << r : 0u;
      } else {
        if (!__all_sync(kFull, near)) {
          out.redo = true;
          return out;
        }
        occluded = shadow_in_list<R, kGeo>(S, *beam, lists->shadow, sorigin, light, sdir, lit, self, lists->first);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (lit[r]) ++out.shadow;
        if (lit[r] && !((occluded >> r) & 1u)) {
          const double cos4 = subrays ? subrays[j + r].cos4 : cos4_of(px[r], py[r]);
          const float3 n = unit(normal[r]), l = lnorm, v = unit(-ray[r]);
          const float n_h = hapke_reflectance(dot(n, l), dot(n, v), dot(l, v), albedo[r], r0[r], hc);
          out.radiance += fmaxf(0, n_h * pose.intensity) * cos4;
        }
      }
    }
  }
  out.radiance /= ss * ss;
  out.depth = valid_depth ? float(depth / valid_depth) : -1.0f;
  return out;
}

// One sub-ray per lane, each lane with its own pose and image-plane
// coordinates: the body of sample_pixel_group's loop for packets whose lanes
// are sub-rays, poses or pixels.  term: the ray's addend of the pixel's
// FP64 radiance sum (0 when unlit).  kChecked: the beam's origin and light
// ranges were formed from other poses than these, so each ray's are checked too.
struct RaySample {
  double term;
  float t;  // hit distance
  bool hit, lit, overflow;
};
template <int kGeo, bool kChecked>
__device__ __forceinline__ RaySample sample_ray(const SceneView &S, float px, float py, const CellPose &pose, bool live,
                                                int *stack_code, float *stack_t, Beam &B, BeamLists &lists) {
  RaySample out{0.0, 0.0f, false, false, false};
  const float3 light = f3(pose.lx, pose.ly, pose.lz);
  const float3 origin = f3(pose.px, pose.py, pose.pz);
  const float3 ray[1] = {unit(rotate_ray(pose, f3(px, -py, -1)))};
  const bool lives[1] = {live};
  const ShadowDir sdir = shadow_dir<kGeo>(light);
  HitRecord hit[1];
  bool inside = within(ray[0], B.dlo, B.dhi);
  if (kChecked) inside = inside && within(origin, B.olo, B.ohi) && within(sdir.idir, B.llo, B.lhi);
  const bool listed = lists.shadow >= 0 && __all_sync(kFull, inside || !live);
  if (listed) {
    nearest_in_list<1, kGeo>(S, B, lists.leaves, origin, ray, lives, hit);
  } else {
    const PacketHits<1> got = nearest_general<1, kGeo>(S, PacketRays<1>{{origin}, {ray[0]}, {live}}, stack_code, stack_t);
    hit[0] = got.h[0];
  }
  out.overflow = live && hit[0].hit < 0;
  out.hit = live && hit[0].hit == 1;
  out.t = hit[0].t;
  float3 normal = f3(0, 0, 0), sorigin[1] = {f3(0, 0, 0)};
  float albedo = S.hc.w, r0 = S.hc.r0_w;
  if (out.hit) {
    const float4 *q = reinterpret_cast<const float4 *>(S.shade + hit[0].tri);
    const float4 s0 = __ldg(q), s1 = __ldg(q + 1), s2 = __ldg(q + 2);
    const float w = 1 - hit[0].u - hit[0].v;
    normal = unit(f3(s0.x, s0.y, s0.z) * w + f3(s1.x, s1.y, s1.z) * hit[0].u + f3(s2.x, s2.y, s2.z) * hit[0].v);
    out.lit = !(dot(normal, light) <= 0 || dot(normal, -ray[0]) <= 0);
    if (out.lit) {
      const float4 *r = tri_record<kGeo>(S, hit[0].tri, 2);
      const float4 a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + 2);
      sorigin[0] = shadow_origin_rec<kGeo>(a, b, c, __ldg(q + 3), hit[0].u, hit[0].v, light);
      if (S.has_albedo) {
        albedo = s0.w * w + s1.w * hit[0].u + s2.w * hit[0].v;
        r0 = hfunc_r0(albedo);
      }
    }
  }
  if (!__any_sync(kFull, out.lit)) return out;
  const bool lit[1] = {out.lit};
  const int self[1] = {hit[0].tri};
  unsigned occluded;
  if (listed && __all_sync(kFull, !out.lit || within(sorigin[0], B.slo, B.shi)))
    occluded = shadow_in_list<1, kGeo>(S, B, lists.shadow, sorigin, light, sdir, lit, self, lists.first);
  else
    occluded = shadow_general<1, kGeo>(S, ShadowRays<1>{{sorigin[0]}, light, {self[0]}, {out.lit}}, stack_code, stack_t);
  if (out.lit && !occluded) {
    const float3 n = unit(normal), l = unit(light), v = unit(-ray[0]);
    const float n_h = hapke_reflectance(dot(n, l), dot(n, v), dot(l, v), albedo, r0, S.hc);
    out.term = fmaxf(0, n_h * pose.intensity) * cos4_of(px, py);
  }
  return out;
}

__device__ __forceinline__ unsigned warp_sum(unsigned v) { return __reduce_add_sync(kFull, v); }

}  // namespace
}  // namespace dvsgb
