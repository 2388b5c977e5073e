// Shared device helpers for the tile-centre render path (sm_100a only).
//
// Arithmetic contract: every float operation that feeds an integer decision (tile overlap, sort
// order, hit / no hit) is written with explicit round-to-nearest intrinsics, so the compiler can
// neither fuse nor reorder it, and det_exp() replaces the hardware exponential.  A CPU that issues
// the same IEEE-754 binary32 operations in the same order reproduces those decisions bit for bit.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "../../include/mlpsp.h"

#define MLPSP_SENTINEL_KEY 1e30f
#define MLPSP_TERM 1e-3f

namespace mlpsp {

__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }

// exp(x) from IEEE operations only: Cody-Waite reduction by ln2 (hi/lo), degree-5 polynomial with
// the Cephes expf coefficients, exponent assembled from integer bits.  x < -87 -> 0, x > 88 -> inf.
__device__ __forceinline__ float det_exp(float x) {
  if (!(x >= -87.0f)) return (x != x) ? x : 0.0f;
  if (x > 88.0f) return __int_as_float(0x7f800000);
  const float kf = rintf(fmul(x, 1.44269504088896341f));
  float r = ffma(kf, -0.693359375f, x);
  r = ffma(kf, 2.12194440e-4f, r);
  float p = 1.9875691500e-4f;
  p = ffma(p, r, 1.3981999507e-3f);
  p = ffma(p, r, 8.3334519073e-3f);
  p = ffma(p, r, 4.1665795894e-2f);
  p = ffma(p, r, 1.6666665459e-1f);
  p = ffma(p, r, 5.0000001201e-1f);
  const float r2 = fmul(r, r);
  float y = ffma(p, r2, r);
  y = fadd(y, 1.0f);
  const int k = (int)kf;
  return fmul(y, __int_as_float((k + 127) << 23));
}

struct V3 { float x, y, z; };

// R^T v for unit quaternion (w,x,y,z): v + w t + u x t, t = 2 (u x v), u = -(x,y,z).
// (scannet/cuda/np_tile_kernels.cu:416-435)
__device__ __forceinline__ V3 rot_conj(float qw, float qx, float qy, float qz, V3 v) {
  const float ux = -qx, uy = -qy, uz = -qz;
  const float tx = fmul(2.f, ffma(uy, v.z, -fmul(uz, v.y)));
  const float ty = fmul(2.f, ffma(uz, v.x, -fmul(ux, v.z)));
  const float tz = fmul(2.f, ffma(ux, v.y, -fmul(uy, v.x)));
  V3 r;
  r.x = fadd(ffma(qw, tx, v.x), ffma(uy, tz, -fmul(uz, ty)));
  r.y = fadd(ffma(qw, ty, v.y), ffma(uz, tx, -fmul(ux, tz)));
  r.z = fadd(ffma(qw, tz, v.z), ffma(ux, ty, -fmul(uy, tx)));
  return r;
}

// Packed primitive geometry: 4 x float4 per primitive.
//   g0 = (cx, cy, cz, qw)   g1 = (qx, qy, qz, max_k exp(ls_k))
//   g2 = (m_x, m_y, m_z, 0) with m_k = exp(-2 ls_k)     g3 = (ls_x, ls_y, ls_z, 0)
struct Geom {
  float cx, cy, cz, qw, qx, qy, qz, smax, mx, my, mz;
};

__device__ __forceinline__ Geom load_geom(const float4* __restrict__ geom, int p) {
  const float4 a = __ldg(geom + (size_t)p * 4 + 0);
  const float4 b = __ldg(geom + (size_t)p * 4 + 1);
  const float4 c = __ldg(geom + (size_t)p * 4 + 2);
  Geom g;
  g.cx = a.x; g.cy = a.y; g.cz = a.z; g.qw = a.w;
  g.qx = b.x; g.qy = b.y; g.qz = b.z; g.smax = b.w;
  g.mx = c.x; g.my = c.y; g.mz = c.z;
  return g;
}

__device__ __forceinline__ float ab_terms(const Geom& g, V3 o, V3 d, float& numer) {
  V3 v = { fsub(g.cx, o.x), fsub(g.cy, o.y), fsub(g.cz, o.z) };
  const V3 vl = rot_conj(g.qw, g.qx, g.qy, g.qz, v);
  const V3 dl = rot_conj(g.qw, g.qx, g.qy, g.qz, d);
  const float denom = ffma(fmul(dl.x, dl.x), g.mx, ffma(fmul(dl.y, dl.y), g.my, fmul(fmul(dl.z, dl.z), g.mz)));
  numer = ffma(fmul(dl.x, vl.x), g.mx, ffma(fmul(dl.y, vl.y), g.my, fmul(fmul(dl.z, vl.z), g.mz)));
  return denom;
}

// ab_terms with the local-frame offset vl = R^T (c - o) supplied by the caller: for rays that share one origin it
// is the same three numbers for every ray, bit for bit, whichever thread computes them.
__device__ __forceinline__ float ab_terms_vl(const Geom& g, V3 vl, V3 d, float& numer) {
  const V3 dl = rot_conj(g.qw, g.qx, g.qy, g.qz, d);
  const float denom = ffma(fmul(dl.x, dl.x), g.mx, ffma(fmul(dl.y, dl.y), g.my, fmul(fmul(dl.z, dl.z), g.mz)));
  numer = ffma(fmul(dl.x, vl.x), g.mx, ffma(fmul(dl.y, vl.y), g.my, fmul(fmul(dl.z, vl.z), g.mz)));
  return denom;
}
__device__ __forceinline__ V3 local_offset(const Geom& g, V3 o) {
  V3 v = { fsub(g.cx, o.x), fsub(g.cy, o.y), fsub(g.cz, o.z) };
  return rot_conj(g.qw, g.qx, g.qy, g.qz, v);
}

// Tile-centre ordering key (np_tile_kernels.cu:483-518): t* on the tile-centre ray, 1e30 when the
// ray is degenerate for this primitive or t* <= 0.
__device__ __forceinline__ float tile_key(const Geom& g, V3 o, V3 d) {
  float numer;
  const float denom = ab_terms(g, o, d, numer);
  if (denom <= 1e-20f) return MLPSP_SENTINEL_KEY;
  const float t = fdiv(numer, denom);
  return (t > 0.f) ? t : MLPSP_SENTINEL_KEY;
}

// Euclidean depth of the centre along the tile-centre ray: the ordering key of the reference's
// expected-depth kernel (np_tile_kernels.cu:5538-5543).
__device__ __forceinline__ float tile_key_euclid(const Geom& g, V3 o, V3 d) {
  const float vx = fsub(g.cx, o.x), vy = fsub(g.cy, o.y), vz = fsub(g.cz, o.z);
  const float t = ffma(vx, d.x, ffma(vy, d.y, fmul(vz, d.z)));
  return (t > 0.f) ? t : MLPSP_SENTINEL_KEY;
}

struct Hit { float t, dx, dy, dz, qx, qy, qz, decay; };

// Rotated-ellipsoid closest approach (np_tile_kernels.cu:659-711).  HAVE_VL: vl = local_offset(g, o) comes from
// the caller (same operations, same bits).
template <bool HAVE_VL>
__device__ __forceinline__ bool hit_test_t(const Geom& g, V3 o, V3 d, V3 vl, float thr, Hit& h) {
  float numer;
  const float denom = HAVE_VL ? ab_terms_vl(g, vl, d, numer) : ab_terms(g, o, d, numer);
  if (denom <= 1e-20f) return false;
  const float t = fdiv(numer, denom);
  if (!(t > 0.f)) return false;
  const float px = ffma(t, d.x, o.x), py = ffma(t, d.y, o.y), pz = ffma(t, d.z, o.z);
  V3 dd = { fsub(g.cx, px), fsub(g.cy, py), fsub(g.cz, pz) };
  const V3 q = rot_conj(g.qw, g.qx, g.qy, g.qz, dd);
  float r2 = fmul(fmul(q.x, q.x), g.mx);
  r2 = ffma(fmul(q.y, q.y), g.my, r2);
  r2 = ffma(fmul(q.z, q.z), g.mz, r2);
  r2 = fmaxf(r2, 0.f);
  const float decay = det_exp(fmul(-0.5f, r2));
  h.t = t; h.dx = dd.x; h.dy = dd.y; h.dz = dd.z; h.qx = q.x; h.qy = q.y; h.qz = q.z; h.decay = decay;
  return decay > thr;
}
__device__ __forceinline__ bool hit_test(const Geom& g, V3 o, V3 d, float thr, Hit& h) {
  return hit_test_t<false>(g, o, d, V3{0.f, 0.f, 0.f}, thr, h);
}

// The same geometry for a pair that is already known to hit: t, the offset c - p, its local-frame image
// and decay as plain float values for the evaluator and the compositor.  No decision hangs on them, so
// the compiler may fuse and the hardware reciprocal / exponential are used.
__device__ __forceinline__ V3 rot_conj_fast(float qw, float qx, float qy, float qz, V3 v) {
  const float tx = 2.f * (qz * v.y - qy * v.z), ty = 2.f * (qx * v.z - qz * v.x), tz = 2.f * (qy * v.x - qx * v.y);
  V3 r;
  r.x = v.x + qw * tx + (qz * ty - qy * tz);
  r.y = v.y + qw * ty + (qx * tz - qz * tx);
  r.z = v.z + qw * tz + (qy * tx - qx * ty);
  return r;
}

__device__ __forceinline__ void hit_values_fast(const Geom& g, V3 o, V3 d, Hit& h) {
  const V3 v = {g.cx - o.x, g.cy - o.y, g.cz - o.z};
  const V3 vl = rot_conj_fast(g.qw, g.qx, g.qy, g.qz, v);
  const V3 dl = rot_conj_fast(g.qw, g.qx, g.qy, g.qz, d);
  const float denom = dl.x * dl.x * g.mx + dl.y * dl.y * g.my + dl.z * dl.z * g.mz;
  const float numer = dl.x * vl.x * g.mx + dl.y * vl.y * g.my + dl.z * vl.z * g.mz;
  const float t = __fdividef(numer, denom);
  const V3 dd = {g.cx - (o.x + t * d.x), g.cy - (o.y + t * d.y), g.cz - (o.z + t * d.z)};
  const V3 q = rot_conj_fast(g.qw, g.qx, g.qy, g.qz, dd);
  const float r2 = fmaxf(q.x * q.x * g.mx + q.y * q.y * g.my + q.z * q.z * g.mz, 0.f);
  h.t = t; h.dx = dd.x; h.dy = dd.y; h.dz = dd.z; h.qx = q.x; h.qy = q.y; h.qz = q.z;
  h.decay = __expf(-0.5f * r2);
}

// Cheap necessary condition for a hit: the centre's distance to the ray's line must be below the
// bounding radius.  With r^2 = sum q_k^2 m_k >= |c - p|^2 / smax^2 >= perp^2 / smax^2 for every point p
// of the line, decay > thr needs perp^2 < smax^2 * (-2 ln thr).  bound2 carries a 2 % margin, far
// above any rounding error here, so a rejected pair is one the full test also rejects and the
// decisions stay identical to evaluating hit_test everywhere.  NaNs fall through to the full test.
__device__ __forceinline__ bool surely_misses(const Geom& g, V3 o, V3 d, float bound2) {
  const float vx = g.cx - o.x, vy = g.cy - o.y, vz = g.cz - o.z;
  const float te = vx * d.x + vy * d.y + vz * d.z;
  const float wx = vx - te * d.x, wy = vy - te * d.y, wz = vz - te * d.z;
  return (wx * wx + wy * wy + wz * wz) > bound2 * (g.smax * g.smax);
}

// ---- the reference kernels' own arithmetic (frame.hit_arith = 1) ----
// The decisions above use IEEE-only operations so that a CPU can reproduce them bit for bit.  The reference's
// kernels evaluate the same formulas with the hardware exponential and leave the contraction of a * b + c to the
// compiler (np_tile_kernels.cu:416-435 rotation, 483-518 tile-centre key, 659-711 hit test).  The functions below
// state the formulas in that form -- plain float expressions in the reference's association, fmaf only where the
// reference writes fmaf, __expf where it writes __expf, compiled by the same compiler with the same default
// contraction -- so that on the GPU the keys, the hit decisions and the hit values come out as the reference
// kernels' own do.  No CPU reproduces those bits; CPU checks of this mode need a margin around the threshold.
struct GeomRef { float cx, cy, cz, qw, qx, qy, qz, lsx, lsy, lsz; };

__device__ __forceinline__ GeomRef load_geom_ref(const float4* __restrict__ geom, int p) {
  const float4 a = __ldg(geom + (size_t)p * 4 + 0);
  const float4 b = __ldg(geom + (size_t)p * 4 + 1);
  const float4 c = __ldg(geom + (size_t)p * 4 + 3);
  GeomRef g;
  g.cx = a.x; g.cy = a.y; g.cz = a.z; g.qw = a.w;
  g.qx = b.x; g.qy = b.y; g.qz = b.z;
  g.lsx = c.x; g.lsy = c.y; g.lsz = c.z;
  return g;
}

// v + w t + u x t with t = 2 (u x v), u = (x, y, z); the conjugate rotation passes -u
__device__ __forceinline__ V3 rot_ref(float w, float x, float y, float z, V3 v) {
  const float tx = 2.f * (y * v.z - z * v.y);
  const float ty = 2.f * (z * v.x - x * v.z);
  const float tz = 2.f * (x * v.y - y * v.x);
  V3 r;
  r.x = v.x + w * tx + (y * tz - z * ty);
  r.y = v.y + w * ty + (z * tx - x * tz);
  r.z = v.z + w * tz + (x * ty - y * tx);
  return r;
}

__device__ __forceinline__ float tile_key_ref(const GeomRef& g, V3 o, V3 d) {
  const float vx = g.cx - o.x, vy = g.cy - o.y, vz = g.cz - o.z;
  const float mx = __expf(-2.f * g.lsx), my = __expf(-2.f * g.lsy), mz = __expf(-2.f * g.lsz);
  const V3 vl = rot_ref(g.qw, -g.qx, -g.qy, -g.qz, V3{vx, vy, vz});
  const V3 dl = rot_ref(g.qw, -g.qx, -g.qy, -g.qz, d);
  const float denom = fmaf(dl.x * dl.x, mx, fmaf(dl.y * dl.y, my, (dl.z * dl.z) * mz));
  const float numer = fmaf(dl.x * vl.x, mx, fmaf(dl.y * vl.y, my, (dl.z * vl.z) * mz));
  if (denom <= 1e-20f) return MLPSP_SENTINEL_KEY;
  const float t = numer / denom;
  return (t > 0.f) ? t : MLPSP_SENTINEL_KEY;
}

__device__ __forceinline__ bool hit_test_ref(const GeomRef& g, V3 o, V3 d, float thr, Hit& h) {
  const float vx = g.cx - o.x, vy = g.cy - o.y, vz = g.cz - o.z;
  const float mx = __expf(-2.f * g.lsx), my = __expf(-2.f * g.lsy), mz = __expf(-2.f * g.lsz);
  const V3 vl = rot_ref(g.qw, -g.qx, -g.qy, -g.qz, V3{vx, vy, vz});
  const V3 dl = rot_ref(g.qw, -g.qx, -g.qy, -g.qz, d);
  const float denom = fmaf(dl.x * dl.x, mx, fmaf(dl.y * dl.y, my, (dl.z * dl.z) * mz));
  if (denom <= 1e-20f) return false;
  const float numer = fmaf(dl.x * vl.x, mx, fmaf(dl.y * vl.y, my, (dl.z * vl.z) * mz));
  const float t = numer / denom;
  if (t <= 0.f) return false;
  const float px = o.x + t * d.x, py = o.y + t * d.y, pz = o.z + t * d.z;
  const float dx = g.cx - px, dy = g.cy - py, dz = g.cz - pz;
  const V3 q = rot_ref(g.qw, -g.qx, -g.qy, -g.qz, V3{dx, dy, dz});
  const float r2 = fmaxf(q.x * q.x * mx + q.y * q.y * my + q.z * q.z * mz, 0.f);
  const float decay = __expf(-0.5f * r2);
  h.t = t; h.dx = dx; h.dy = dy; h.dz = dz; h.qx = q.x; h.qy = q.y; h.qz = q.z; h.decay = decay;
  return decay > thr;
}

// ---- the (tile, primitive) pre-test of the fused frame path ----
// The frame's tangent plane: origin o and an orthonormal frame (a, u, v) around the central ray.  A ray direction d from
// that origin is a + alpha u + beta v up to scale (alpha = d.u / d.a, beta = d.v / d.a), and the rays of a tile lie in the
// rectangle [a0, a1] x [b0, b1] of those coordinates (slightly inflated).  A tile whose rays do not all leave o, or lie
// 75 degrees and more off the central ray, has no rectangle (NaN): no candidate of it is ever rejected.
struct __align__(16) FramePlane {
  float ox, oy, oz, pad0, ax, ay, az, pad1, ux, uy, uz, pad2, vx, vy, vz, pad3;
};

// Whitening map of one primitive: x -> diag(1 / exp(ls)) R^T x as a 3x3 matrix (row-major), its centre, the
// largest inverse scale.  Built once per primitive, used for every tile of its rectangle.
struct PrimWhiten { float m[9]; float cx, cy, cz, ismax; };

__device__ __forceinline__ PrimWhiten make_whiten(const Geom& g) {
  PrimWhiten w;
  const float is[3] = {sqrtf(g.mx), sqrtf(g.my), sqrtf(g.mz)};
  const V3 c0 = rot_conj(g.qw, g.qx, g.qy, g.qz, V3{1.f, 0.f, 0.f});
  const V3 c1 = rot_conj(g.qw, g.qx, g.qy, g.qz, V3{0.f, 1.f, 0.f});
  const V3 c2 = rot_conj(g.qw, g.qx, g.qy, g.qz, V3{0.f, 0.f, 1.f});
  w.m[0] = c0.x * is[0]; w.m[1] = c1.x * is[0]; w.m[2] = c2.x * is[0];
  w.m[3] = c0.y * is[1]; w.m[4] = c1.y * is[1]; w.m[5] = c2.y * is[1];
  w.m[6] = c0.z * is[2]; w.m[7] = c1.z * is[2]; w.m[8] = c2.z * is[2];
  w.cx = g.cx; w.cy = g.cy; w.cz = g.cz;
  w.ismax = fmaxf(is[0], fmaxf(is[1], is[2]));
  return w;
}

__device__ __forceinline__ V3 whiten(const PrimWhiten& w, float x, float y, float z) {
  V3 r;
  r.x = fmaf(w.m[0], x, fmaf(w.m[1], y, w.m[2] * z));
  r.y = fmaf(w.m[3], x, fmaf(w.m[4], y, w.m[5] * z));
  r.z = fmaf(w.m[6], x, fmaf(w.m[7], y, w.m[8] * z));
  return r;
}

// What a primitive's threshold ellipsoid r^2 <= K cuts out of the tangent plane: the lines from o that meet it form the
// ellipse (z - z0)^T A (z - z0) <= rho around z0.  In the primitive's whitened frame (rotate by R^T, divide axis k by
// exp(ls_k)) the ellipsoid is a sphere of radius sqrt(K) around the origin, and the line from x with direction e meets it
// iff |x cross e|^2 <= K |e|^2.  The coordinates are taken relative to the direction of the centre, for which the cross
// product vanishes, so nothing cancels.  K carries a margin of 0.4 % plus twice the bound on hit_test's rounding that the
// hit pass derives (hit_form).  never = the ellipse does not exist (centre beside or behind the plane, origin inside,
// anything not finite): such a primitive is never rejected.
struct __align__(16) PlaneEllipse { float zx, zy, a11, a12, a22, r1, r2, rho; };     // r1 = a12 / a22, r2 = a12 / a11

__device__ __forceinline__ PlaneEllipse plane_ellipse(const Geom& g, const FramePlane& f, float K0) {
  PlaneEllipse e;
  e.zx = e.zy = e.a11 = e.a12 = e.a22 = e.r1 = e.r2 = 0.f;
  e.rho = __int_as_float(0x7f800000);                       // no value exceeds it: never rejected
  const PrimWhiten pw = make_whiten(g);
  const float vx = g.cx - f.ox, vy = g.cy - f.oy, vz = g.cz - f.oz;
  const float va = vx * f.ax + vy * f.ay + vz * f.az;
  const float dist = sqrtf(vx * vx + vy * vy + vz * vz);
  if (!(va > 0.1f * dist) || !(dist > 0.f)) return e;
  const float rva = 1.f / va;
  const float ac = (vx * f.ux + vy * f.uy + vz * f.uz) * rva, bc = (vx * f.vx + vy * f.vy + vz * f.vz) * rva;
  const V3 x = whiten(pw, vx, vy, vz);
  const V3 ec = {x.x * rva, x.y * rva, x.z * rva};          // direction of the centre: a + ac u + bc v
  const V3 e1 = whiten(pw, f.ux, f.uy, f.uz), e2 = whiten(pw, f.vx, f.vy, f.vz);
  const V3 w1 = {x.y * e1.z - x.z * e1.y, x.z * e1.x - x.x * e1.z, x.x * e1.y - x.y * e1.x};
  const V3 w2 = {x.y * e2.z - x.z * e2.y, x.z * e2.x - x.x * e2.z, x.x * e2.y - x.y * e2.x};
  const float S = fabsf(vx) + fabsf(vy) + fabsf(vz) + fabsf(f.ox) + fabsf(f.oy) + fabsf(f.oz);
  const float K = K0 * 1.004f + 2e-5f * sqrtf(K0) * S * pw.ismax;
  const float a11 = (w1.x * w1.x + w1.y * w1.y + w1.z * w1.z) - K * (e1.x * e1.x + e1.y * e1.y + e1.z * e1.z);
  const float a22 = (w2.x * w2.x + w2.y * w2.y + w2.z * w2.z) - K * (e2.x * e2.x + e2.y * e2.y + e2.z * e2.z);
  const float a12 = (w1.x * w2.x + w1.y * w2.y + w1.z * w2.z) - K * (e1.x * e2.x + e1.y * e2.y + e1.z * e2.z);
  const float b1 = -K * (ec.x * e1.x + ec.y * e1.y + ec.z * e1.z), b2 = -K * (ec.x * e2.x + ec.y * e2.y + ec.z * e2.z);
  const float c0 = -K * (ec.x * ec.x + ec.y * ec.y + ec.z * ec.z);
  const float det = a11 * a22 - a12 * a12;
  // (the forms lose their digits where the origin comes close to the ellipsoid)
  if (!(a11 > 0.1f * K * (e1.x * e1.x + e1.y * e1.y + e1.z * e1.z)) || !(a22 > 0.1f * K * (e2.x * e2.x + e2.y * e2.y + e2.z * e2.z)) ||
      !(det > 1e-3f * a11 * a22))
    return e;
  const float rdet = 1.f / det;
  const float zx = (a12 * b2 - a22 * b1) * rdet, zy = (a12 * b1 - a11 * b2) * rdet;
  const float rho = -(b1 * zx + b2 * zy) - c0;
  if (!(rho > 0.f) || !(rho < 1e30f) || !(fabsf(zx) + fabsf(zy) < 1e3f)) return e;
  e.zx = ac + zx; e.zy = bc + zy;
  e.a11 = a11; e.a12 = a12; e.a22 = a22;
  e.r1 = a12 / a22; e.r2 = a12 / a11;
  e.rho = rho * 1.001f;
  return e;
}

// The smallest value of the ellipse's form over the rectangle r = (a0, a1, b0, b1), relative to its centre: attained at the
// centre, or on an edge that faces it.  Above rho no ray of the tile can hit (NaNs answer false).  The rectangle is widened
// by the rounding of the centre's coordinates.
__device__ __forceinline__ bool ellipse_misses(const float4 z /* zx zy a11 a12 */, const float4 w /* a22 r1 r2 rho */, const float4 r) {
  const float pad = 1e-6f * (1.f + fabsf(z.x) + fabsf(z.y));
  const float l1 = r.x - z.x - pad, h1 = r.y - z.x + pad, l2 = r.z - z.y - pad, h2 = r.w - z.y + pad;
  const float xs = fminf(fmaxf(0.f, l1), h1), ys = fminf(fmaxf(0.f, l2), h2);
  const float y1 = fminf(fmaxf(-w.y * xs, l2), h2), x2 = fminf(fmaxf(-w.z * ys, l1), h1);
  const float f1 = z.z * xs * xs + (2.f * z.w * xs + w.x * y1) * y1;
  const float f2 = z.z * x2 * x2 + (2.f * z.w * x2 + w.x * ys) * ys;
  return fminf(f1, f2) > w.w && r.x == r.x;
}

__device__ __forceinline__ V3 load3(const float* __restrict__ p, int64_t i) {
  V3 r = { __ldg(p + i * 3), __ldg(p + i * 3 + 1), __ldg(p + i * 3 + 2) };
  return r;
}

// pixel k (row-major inside the 8x8 tile) of a tile: image index and whether it lies inside the image
struct TilePix {
  int pix; bool valid;
};

__device__ __forceinline__ TilePix tile_pixel(int tile, int k, int ntx, int W, int H) {
  const int tx = tile % ntx, ty = tile / ntx;
  const int x = tx * 8 + (k & 7), y = ty * 8 + (k >> 3);
  TilePix r;
  r.valid = (x < W) && (y < H);
  r.pix = r.valid ? y * W + x : 0;
  return r;
}

// The warp's number in its CTA, as a value the compiler knows to be the same in all lanes: what is computed from it (work units,
// descriptors, addresses) then takes one scalar instruction instead of a vector one.  All lanes must call it.
__device__ __forceinline__ int warp_of_cta() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }

// Output activations (np_tile_kernels.cu:75-83); values, not decisions, so hardware exp is fine.
__device__ __forceinline__ float sigmoid_fast(float x) { return __fdividef(1.0f, 1.0f + __expf(-x)); }
__device__ __forceinline__ float softplus_fast(float x) {
  // log(1 + e) on the hardware logarithm: within 1e-7 absolute of log1p over [-20, 20], far below what the
  // compositing weights resolve (selections, not branches: lanes differ)
  const float e = __expf(x), l = __logf(1.0f + e);
  return x > 20.f ? x : (x < -20.f ? e : l);
}

// position of the (k+1)-th set bit of m (k >= 0 and fewer than popc(m)): five halvings by population count, the
// same number of steps for every lane of a warp (the library's __fns walks the set bits one by one)
__device__ __forceinline__ int nth_set_bit(uint32_t m, int k) {
  int pos = 0, c;
  c = __popc(m & 0xffffu); if (k >= c) { k -= c; pos += 16; m >>= 16; }
  c = __popc(m & 0xffu);   if (k >= c) { k -= c; pos += 8;  m >>= 8; }
  c = __popc(m & 0xfu);    if (k >= c) { k -= c; pos += 4;  m >>= 4; }
  c = __popc(m & 0x3u);    if (k >= c) { k -= c; pos += 2;  m >>= 2; }
  c = (int)(m & 1u);       if (k >= c) { pos += 1; }
  return pos;
}

// ---- block-wide exclusive scan of one int per thread (blockDim.x <= 1024, multiple of 32) ----
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums /* [32] shared */, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += n;
  }
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    int w = (lane < nw) ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += n;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  const int base = (warp > 0) ? warp_sums[warp - 1] : 0;
  total = warp_sums[((blockDim.x + 31) >> 5) - 1];
  __syncthreads();
  return base + inc - v;
}

}  // namespace mlpsp
