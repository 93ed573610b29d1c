// The reference's analytic signed-distance scenes on the device
// (src/engine/wgsl.ts:20-76,101-116 primitives and scene switch;
// src/engine/f1.ts:20-320 generic F1, :397-407 heat emission), shared by the
// voxelizer and the renderer.  Every float operation keeps the reference's
// order (units built with -fmad=false); sin, cos and atan are the project's
// functions (wt_fmath.h).  Shape-wide values (rake rotation, rear main-plane
// direction) are computed once on the host by make_scene with the same
// functions, which gives the same bits as evaluating them per point.
#pragma once
#include <cuda_fp16.h>

#include "wt_fmath.h"
#include "wt_internal.h"
#include "wt_vec.cuh"

namespace wt {
namespace {

// The F1's parts as tables of operands, formed from the shape on the host (f1_tables) by
// the operations the reference writes at each part.  One copy of each primitive reads them
// (sd_taper and on): the scene as straight-line code is some 2500 instructions whose
// fetches were the bound (a 1280x720 frame issued in 15 % of its cycles and waited for an
// instruction in 26 of every 30; half of the requests missed the first instruction cache).
// With the parts left out that cannot matter (beyond): frame 3.15 -> 1.81 ms, voxelizing
// 168x50x38 cells 75 -> 48 us.  A loop over the parts as a list of operations fetches
// better still (96 % hits) and issues twice the instructions: 3.4 ms.
// Quads of floats:
//   taper    x0 dx mid half | r0 r1 - - | c0 c1 | s0 s1      capsule  a, r | b - a, |b - a|^2
//   box      centre, r | half - r                           ellipsoid  centre | r | r * r
//   wing     le.x le.y chord ang | thick z0 z1 rise | taper curl - -
//   around   low corner, factor | high corner, addend
enum : uint32_t { T_MID, T_NOSE, T_SCUTTLE, T_COVER, T_KEEL, T_POD, T_TAIL, T_COUNT };
enum : uint32_t { C_HALO = 0, C_SUSF = 4, C_SUSR = 10, C_MIRROR = 15, C_EXHAUST, C_BORE, C_EDGE, C_POST, C_CARVE, C_COUNT = C_CARVE + 2 };
enum : uint32_t {
  B_BODY, B_FLOOR, B_FRONT, B_REAR, B_WHEEL,  // the groups' own boxes (two wheels)
  B_PYLON = B_WHEEL + 2, B_AIRBOX, B_COCKPIT, B_MIRROR, B_FIN, B_LIGHT, B_CARVE, B_FENCE, B_STRAKE = B_FENCE + 2,
  B_FOOT = B_STRAKE + 2, B_POST, B_DUCT, B_COUNT = B_DUCT + 2
};
enum : uint32_t { E_NOSE, E_AIR, E_HELMET, E_COUNT };
enum : uint32_t {  // boxes around parts (beyond)
  K_SCUTTLE, K_NOSE, K_COVER, K_KEEL, K_POD, K_AIRBOX, K_COCKPIT, K_CABIN, K_HELMET, K_HALO, K_MIRROR, K_SUSF, K_SUSR,
  K_TAIL, K_FIN, K_LIGHT, K_FENCE, K_STRAKE, K_EDGE, K_COUNT
};
struct F1Tables {
  float4 taper[T_COUNT][4], cap[C_COUNT][2], box[B_COUNT][2], ell[E_COUNT][3], wing[6][3],
      around[K_COUNT][2];
  float pod_k[3];      // the sidepod's carvings: capsules, then the box
  uint32_t pod_caps, front_wings, pylon;
  float ep[5];         // front endplate: centre x, y, half x, y, radius
};

// Shape plus host-computed shape-wide constants.  The renderer has them as a copy of the
// thread's (scene_of), as the W17's distance likes them, the tables in the kernel's
// parameters (F1 and W17 mesh frames of 1280x720 2.11 -> 2.08 and 0.91 -> 0.89 ms); the
// voxelizer, one distance to a thread, reads both from there (with a copy 48.9 -> 53 us).
struct Scene {
  const F1Tables* f1;         // kind 0; set by scene_of
  wt_shape s;
  CarView car;                // the W17 model (kind 5)
  float rake_c, rake_s;       // cos/sin of the rake angle (f1.ts:37-40)
  float rear_c, rear_s;       // cos/sin of the rear main-plane angle after variant offsets (f1.ts:274)
  float ang_m, ang_f, chord_m, chord_f, rise_m, ep_hx, ep_hy;  // rear-wing variant (f1.ts:260-272)
};
struct SceneParam {
  Scene s;
  F1Tables f1;
};
__host__ __device__ __forceinline__ Scene scene_of(const SceneParam& P) {
  Scene S = P.s;
  S.f1 = &P.f1;
  return S;
}

constexpr float DEG = 0.017453292f, FA = 1.0f, RA = 4.6f, WR = 0.36f, FWZ = 0.84f, FHW = 0.152f, RWZ = 0.80f,
                RHW = 0.20f, RA26 = 4.4f, WR26 = 0.355f, FHW26 = 0.14f, RHW26 = 0.1875f, BODY_X = 0.9444444f,
                BODY_Z = 0.96f, BODY_LIP = 0.96f;

// ---------------------------------------------------------------- primitives
__device__ float sd_box(V3 p, V3 b) {
  const V3 q = v3(ab(p.x) - b.x, ab(p.y) - b.y, ab(p.z) - b.z);
  return len3(v3(mx(q.x, 0.0f), mx(q.y, 0.0f), mx(q.z, 0.0f))) + mn(mx(q.x, mx(q.y, q.z)), 0.0f);
}
__device__ float sd_rbox(V3 p, V3 b, float r) { return sd_box(p, v3(b.x - r, b.y - r, b.z - r)) - r; }
__device__ float sd_capsule(V3 p, V3 a, V3 b, float r) {
  const V3 pa = p - a, ba = b - a;
  const float hh = clmp(dv(dot3(pa, ba), dot3(ba, ba)), 0.0f, 1.0f);
  return len3(pa - ba * hh) - r;
}
__device__ float sd_rrect(V2 p, V2 b, float r) {
  const V2 q = v2(ab(p.x) - b.x + r, ab(p.y) - b.y + r);
  return len2(v2(mx(q.x, 0.0f), mx(q.y, 0.0f))) + mn(mx(q.x, q.y), 0.0f) - r;
}
__device__ float op_extrude(float d2, float dz) {
  return mn(mx(d2, dz), 0.0f) + len2(v2(mx(d2, 0.0f), mx(dz, 0.0f)));
}
__device__ float sd_uneven_capsule(V2 p0, float r1, float r2, float hh) {
  const V2 p = v2(ab(p0.x), p0.y);
  const float b = dv(r1 - r2, hh);
  const float a = __fsqrt_rn(mx(1.0f - b * b, 0.0f));
  const float k = dot2(p, v2(-b, a));
  if (k < 0.0f) return len2(p) - r1;
  if (k > a * hh) return len2(p - v2(0.0f, hh)) - r2;
  return dot2(p, v2(a, b)) - r1;
}
__device__ float sd_wing_cs(V3 p, V2 le, float chord, float c, float s, float thick, float z0, float z1) {
  const V2 q = v2(p.x, p.y) - le;
  const float lx = q.x * c + q.y * s;
  const float ly = -q.x * s + q.y * c;
  const float r1 = thick * 0.5f;
  const float r2 = mx(thick * 0.12f, 0.006f);
  const float d2 = sd_uneven_capsule(v2(ly, lx - r1), r1, r2, mx(chord - r1 - r2, 0.01f));
  return op_extrude(d2, ab(p.z - 0.5f * (z0 + z1)) - 0.5f * (z1 - z0));
}
__device__ float sd_wing(V3 p, V2 le, float chord, float ang, float thick, float z0, float z1) {
  float s, c;
  wtm::sincosf(ang, &s, &c);
  return sd_wing_cs(p, le, chord, c, s, thick, z0, z1);
}
__device__ __forceinline__ V2 op_u(V2 a, V2 b) { return (b.x < a.x) ? b : a; }

// ---------------------------------------------------------------- generic F1
__device__ V3 body_frame(const Scene& S, V3 pw) {
  const float c = S.rake_c, s = S.rake_s;
  const float dx = pw.x - FA, dy = pw.y - S.s.ride_h;
  const V3 p = v3(FA + dx * c + dy * s, S.s.ride_h - dx * s + dy * c, pw.z);
  float x = p.x;
  if (x > FA) {
    const float a = FA + dv(x - FA, BODY_X);
    const float b = x + (RA - RA26);
    x = (x > RA26) ? b : a;
  }
  return v3(x, p.y, dv(p.z, BODY_Z));
}
__device__ __noinline__ float smin(float a, float b, float k) {
  const float h = dv(mx(k - ab(a - b), 0.0f), k);
  return mn(a, b) - h * h * k * 0.25f;
}
__device__ __forceinline__ float smax(float a, float b, float k) { return -smin(-a, -b, k); }
__device__ __noinline__ float sd_taper(const float4* q, V3 p) {
  const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3];
  const float t = clmp(dv(p.x - q0.x, q0.y), 0.0f, 1.0f);
  const V2 c = mix2(v2(q2.x, q2.y), v2(q2.z, q2.w), t);
  const V2 s = mix2(v2(q3.x, q3.y), v2(q3.z, q3.w), t);
  const float r = mn(mixf(q1.x, q1.y, t), mn(s.x, s.y));
  const float d2 = sd_rrect(v2(p.y, p.z) - c, s, r);
  return op_extrude(d2, ab(p.x - q0.z) - q0.w) * 0.8f;
}
__device__ __noinline__ float sd_cap(const float4* q, V3 p) {
  const float4 q0 = q[0], q1 = q[1];
  const V3 pa = p - v3(q0.x, q0.y, q0.z), ba = v3(q1.x, q1.y, q1.z);
  const float hh = clmp(dv(dot3(pa, ba), q1.w), 0.0f, 1.0f);
  return len3(pa - ba * hh) - q0.w;
}
__device__ __noinline__ float sd_rb(const float4* q, V3 p) {
  const float4 q0 = q[0], q1 = q[1];
  return sd_box(p - v3(q0.x, q0.y, q0.z), v3(q1.x, q1.y, q1.z)) - q0.w;
}
__device__ __noinline__ float sd_ellipsoid(const float4* q, V3 pw) {
  const float4 q0 = q[0], q1 = q[1], q2 = q[2];
  const V3 p = pw - v3(q0.x, q0.y, q0.z);
  const float k0 = len3(v3(dv(p.x, q1.x), dv(p.y, q1.y), dv(p.z, q1.z)));
  const float k1 = len3(v3(dv(p.x, q2.x), dv(p.y, q2.y), dv(p.z, q2.z)));
  return dv(k0 * (k0 - 1.0f), mx(k1, 1e-5f));
}
__device__ float sd_cyl_z(V3 p, float r, float hz) {
  const float dx = len2(v2(p.x, p.y)) - r, dz = ab(p.z) - hz;
  return mn(mx(dx, dz), 0.0f) + len2(v2(mx(dx, 0.0f), mx(dz, 0.0f)));
}
__device__ __noinline__ float sd_cyl(V3 p, float r, float hz) { return sd_cyl_z(p, r, hz); }
__device__ __noinline__ float sd_wing_z(const float4* q, V3 p) {
  const float4 q0 = q[0], q1 = q[1], q2 = q[2];
  const float z1 = q1.z, rise = q1.w;
  const float s = sstep(q2.y, z1, p.z);
  return sd_wing(p, v2(q0.x, q0.y) + v2(0.0f, rise * s), q0.z * (1.0f - q2.x * s), q0.w + rise * s * 0.6f, q1.x, q1.y,
                 z1) *
         0.85f;
}
__device__ float tunnel_roof(float x, float b) {
  if (x < 2.5f) return mixf(b + 0.12f, b + 0.05f, sstep(1.55f, 2.5f, x));
  if (x < 3.8f) return b + 0.05f;
  return mixf(b + 0.05f, b + 0.25f, sstep(3.8f, 4.98f, x));
}
__device__ float sd_slab(V3 p, float b, float roof) {
  const float zlim = mixf(0.80f, 0.58f, sstep(3.6f, 4.15f, p.x));
  const float top = (ab(p.z - 0.40f) < 0.28f) ? roof + 0.03f : b + 0.05f;
  const float slab = mx(mx(b - p.y, p.y - top), mx(ab(p.x - 3.265f) - 1.715f, p.z - zlim));
  const float tunnel = mx(p.y - roof, ab(p.z - 0.40f) - 0.255f);
  return mx(slab, -tunnel) * 0.8f;
}
__device__ float sd_tyre(V3 p, V3 c, float hw) {
  const V3 q = p - c;
  return sd_rrect(v2(len2(v2(q.x, q.y)) - 0.2925f, q.z), v2(0.0625f, hw), 0.06f);
}
// A part cannot change a point's result when its distance as computed is at least what it
// joins: mn(d, part) is exactly d when part >= d, smin(d, part, k) exactly d when
// part >= d + k.  The distance as computed is bounded below by a factor (1 for boxes,
// capsules and cylinders, 0.8 for tapers, min/max radius for ellipsoids) times the
// distance to a box around the part; beyond() tests that against r.  Its margin covers
// the roundings (relative 1e-3, and 0.1 mm of a model in metres); points and parts that
// are not finite are never beyond.
// r = factor * (d + addend) is the distance to the box that leaves d as it is.
__device__ __noinline__ bool beyond(const float4* q, V3 p, float d) {
  const float4 lo = q[0], hi = q[1];
  const float x = fmaxf(fmaxf(lo.x - p.x, p.x - hi.x), 0.0f), y = fmaxf(fmaxf(lo.y - p.y, p.y - hi.y), 0.0f),
              z = fmaxf(fmaxf(lo.z - p.z, p.z - hi.z), 0.0f);
  const float r = lo.w * (d + hi.w), m = (fmaxf(r, 0.0f) + 1e-4f) * 1.001f, d2 = fmaf(x, x, fmaf(y, y, z * z));
  return d2 > m * m && d2 < 1e12f && r < 1e6f;
}
// The same with the test along x, where most parts fail, in line.
__device__ __forceinline__ bool beyond_x(const float4* q, V3 p, float lo, float hi, float factor, float addend, float d) {
  const float gap = fmaxf(lo - p.x, p.x - hi), r = fmaxf(factor * (d + addend), 0.0f);
  return (gap > r * 1.001f + 2e-4f && gap < 1e6f) || beyond(q, p, d);
}
// The body's own distance.  The chain is smin(smin(nose, scuttle), cockpit) and on: the
// cockpit's part comes first, and what stands before it only where it can reach it (a
// smin lowers the smaller value by at most k / 4; the nose's ellipsoid has radii 1 : 2).
__device__ float sd_bodywork(const F1Tables& F, V3 p) {
  const float mid = sd_taper(F.taper[T_MID], p);
  float d = mid;
  if (!beyond_x(F.around[K_SCUTTLE], p, 1.20f, 2.24f, 1.25f, 0.08f, mid) ||
      !beyond_x(F.around[K_NOSE], p, -0.06f, 1.26f, 2.0f, 0.09f, mid)) {
    d = sd_taper(F.taper[T_NOSE], p);
    d = smin(d, sd_ellipsoid(F.ell[E_NOSE], p), 0.04f);
    if (F.pylon) d = mn(d, sd_rb(F.box[B_PYLON], p));
    d = smin(d, sd_taper(F.taper[T_SCUTTLE], p), 0.08f);
    d = smin(d, mid, 0.06f);
  }
#pragma unroll 1
  for (uint32_t i = 0; i < 3; i++) {  // engine cover, keel, sidepods; each joins with its box's addend
    if (beyond(F.around[K_COVER + i], p, d)) continue;
    float v = sd_taper(F.taper[T_COVER + i], p);
    if (i == 2) {
#pragma unroll 1
      for (uint32_t j = 0; j <= F.pod_caps; j++) {
        const float c = j < F.pod_caps ? sd_cap(F.cap[C_CARVE + j], p) : sd_rb(F.box[B_CARVE], p);
        v = smax(v, -c, F.pod_k[j < F.pod_caps ? j : 2]);
      }
    }
    d = smin(d, v, F.around[K_COVER + i][1].w);
  }
  if (!beyond(F.around[K_AIRBOX], p, d))
    d = smin(d, smax(sd_rb(F.box[B_AIRBOX], p), -sd_ellipsoid(F.ell[E_AIR], p), 0.015f), 0.10f);
  // smax(d, -x, k) is exactly d when x >= k - d
  if (!beyond(F.around[K_COCKPIT], p, d))
    d = smax(d, -sd_rb(F.box[B_COCKPIT], p), 0.03f);
  return d;
}
__device__ __noinline__ float cap_min(const float4 (*q)[2], uint32_t n, V3 p, float d) {
#pragma unroll 1
  for (uint32_t i = 0; i < n; i++) d = mn(d, sd_cap(q[i], p));
  return d;
}
// near: the point's distance so far; what is not below it need not be exact.
__device__ float sd_carbon(const F1Tables& F, V3 p, float near) {
  float d = 1e30f;
  if (!beyond_x(F.around[K_SUSF], p, 0.84f, 1.44f, 1.0f, 0.0f, near))
    d = cap_min(F.cap + C_SUSF, 6u, p, d);
  if (!beyond_x(F.around[K_SUSR], p, 4.26f, 4.84f, 1.0f, 0.0f, fminf(d, near)))
    d = cap_min(F.cap + C_SUSR, 5u, p, d);
  if (!beyond_x(F.around[K_TAIL], p, 4.78f, 5.42f, 1.25f, 0.0f, fminf(d, near)))
    d = mn(d, sd_taper(F.taper[T_TAIL], p));
  if (!beyond_x(F.around[K_FIN], p, 3.40f, 4.50f, 1.0f, 0.0f, fminf(d, near)))
    d = mn(d, sd_rb(F.box[B_FIN], p));
  return d;
}
__device__ float sd_floor(const F1Tables& F, V3 p, float b, float near) {
  const float roof = tunnel_roof(p.x, b);
  float d = sd_slab(p, b, roof);
  if (!beyond(F.around[K_FENCE], p, fminf(d, near)))
#pragma unroll 1
    for (uint32_t i = 0; i < 2; i++) d = mn(d, mx(sd_rb(F.box[B_FENCE + i], p), p.y - roof - 0.02f));
  if (!beyond(F.around[K_STRAKE], p, fminf(d, near)))
#pragma unroll 1
    for (uint32_t i = 0; i < 2; i++) d = mn(d, mx(sd_rb(F.box[B_STRAKE + i], p), p.y - roof));
  if (!beyond(F.around[K_EDGE], p, fminf(d, near)))
    d = mn(d, sd_cap(F.cap[C_EDGE], p));
  return d;
}
__device__ V2 sd_f1(const Scene& S, const F1Tables& F, V3 pw) {
  const V3 pworld = v3(pw.x, pw.y, ab(pw.z));
  const V3 p = body_frame(S, pworld);
  const float b = S.s.ride_h;
  V2 res = v2(1e3f, 0.0f);
  if (sd_rb(F.box[B_BODY], p) < res.x) {
    res = op_u(res, v2(sd_bodywork(F, p), 0.0f));
    // cockpit: helmet, halo (its smins lower it by at most 0.0225), mirror
    if (!beyond_x(F.around[K_CABIN], p, 2.13f, 3.06f, 1.25f, 0.018f, res.x)) {
      if (!beyond(F.around[K_HELMET], p, res.x))
        res = op_u(res, v2(sd_ellipsoid(F.ell[E_HELMET], p), 3.0f));
      if (!beyond(F.around[K_HALO], p, res.x)) {
        float d = sd_cap(F.cap[C_HALO], p);
#pragma unroll 1
        for (uint32_t i = 1; i < 4; i++) d = smin(d, sd_cap(F.cap[C_HALO + i], p), 0.03f);
        res = op_u(res, v2(d, 4.0f));
      }
      if (!beyond(F.around[K_MIRROR], p, res.x))
        res = op_u(res, v2(mn(sd_rb(F.box[B_MIRROR], p), sd_cap(F.cap[C_MIRROR], p)), 0.0f));
    }
    res = op_u(res, v2(sd_carbon(F, p, res.x), 1.0f));
    if (!beyond_x(F.around[K_LIGHT], p, 4.90f, 5.42f, 1.0f, 0.0f, res.x)) {
      res = op_u(res, v2(sd_rb(F.box[B_LIGHT], p), 11.0f));
      res = op_u(res, v2(mx(sd_cap(F.cap[C_EXHAUST], p), -sd_cap(F.cap[C_BORE], p)), 10.0f));
    }
  }
  if (sd_rb(F.box[B_FLOOR], p) < res.x) res = op_u(res, v2(sd_floor(F, p, b, res.x), 1.0f));
  const float lip = BODY_LIP * BODY_X;
  res.x = res.x * lip;
#pragma unroll 1
  for (uint32_t w = 0; w < 2; w++) {  // front, rear wing
    if (!(sd_rb(F.box[B_FRONT + w], p) < dv(res.x, lip))) continue;
    const uint32_t i0 = w ? 4u : 0u, i1 = w ? 6u : F.front_wings;
    float d = sd_wing_z(F.wing[i0], p);
#pragma unroll 1
    for (uint32_t i = i0 + 1; i < i1; i++) d = mn(d, sd_wing_z(F.wing[i], p));
    const float4 e = w ? make_float4(5.25f, (b + 0.80f) - 0.03f, S.ep_hx, S.ep_hy) : make_float4(F.ep[0], F.ep[1], F.ep[2], F.ep[3]);
    const float ep = sd_rrect(v2(p.x - e.x, p.y - e.y), v2(e.z, e.w), w ? 0.13f : F.ep[4]);
    if (w) d = mn(d, sd_cap(F.cap[C_POST], p));
    d = mn(d, mx(ep, w ? ab(p.z - 0.513f) - 0.012f : ab(p.z - (0.94f + 0.012f)) - 0.010f));
    d = mn(d, sd_rb(F.box[B_FOOT + w], p));
    res = op_u(res, v2(d * BODY_LIP * BODY_X, w ? 8.0f : 7.0f));  // (d * LIP) * X, as written
  }
#pragma unroll 1
  for (uint32_t w = 0; w < 2; w++) {  // wheels, in the world's frame
    if (sd_rb(F.box[B_WHEEL + w], pworld) > res.x) continue;
    const float4 c4 = F.box[B_WHEEL + w][0];
    const V3 c = v3(c4.x, c4.y, c4.z);
    const float hw = w ? RHW26 : FHW26, inboard = w ? 0.08f : 0.10f;
    res = op_u(res, v2(sd_tyre(pworld, c, hw), 2.0f));
    const V3 q = pworld - c;
    const float cover = mn(sd_cyl(q, 0.234f, hw - 0.028f), sd_cyl(q - v3(0.0f, 0.0f, hw - 0.02f), 0.045f, 0.02f));
    res = op_u(res, v2(cover, 9.0f));
    const float duct = sd_cyl(pworld - v3(c.x, c.y, c.z - hw - inboard * 0.5f), 0.17f, inboard * 0.5f);
    res = op_u(res, v2(mn(duct, sd_rb(F.box[B_DUCT + w], pworld)), 10.0f));
  }
  return res;
}
__device__ float f1_emission(const Scene& S, V3 pw) {
  const V3 p = body_frame(S, v3(pw.x, pw.y, ab(pw.z)));
  const float b = S.s.ride_h;
  float e = 0.0f;
  if (len2(v2(p.x - FA, p.y - WR)) < 0.21f && ab(p.z - (FWZ - FHW - 0.03f)) < 0.12f) e = mx(e, S.s.heat_brakes);
  if (len2(v2(p.x - RA, p.y - WR)) < 0.21f && ab(p.z - (RWZ - RHW - 0.03f)) < 0.12f) e = mx(e, S.s.heat_brakes * 0.8f);
  if (p.x > 5.02f && sd_capsule(p, v3(4.95f, b + 0.44f, 0.0f), v3(5.16f, b + 0.45f, 0.0f), 0.09f) < 0.0f) e = mx(e, S.s.heat_engine);
  if (p.x > 3.85f && p.x < 4.5f && p.z > 0.10f && p.y > b + 0.12f && p.y < b + 0.45f) e = mx(e, S.s.heat_rad);
  if (p.x > 3.55f && p.x < 4.25f && p.z < 0.13f && p.y > b + 0.42f) e = mx(e, S.s.heat_rad * 1.4f);
  return e;
}

// ---------------------------------------------------------------- baked W17 model (kind 5)
// src/engine/f1.ts:322-394 and the rig functions of src/engine/car-model.ts:59-136.
constexpr float W17_H = 0.015f, W17_BASE_RIDE = 0.092f;
constexpr int RIG_HINGES = 71, RIG_ANGLES = 72, RIG_EXTRA = 73, RIG_FLY = 74, RIG_GRIDS = 75;

__device__ __forceinline__ float4 rig_at(const float4* R, int i) { return __ldg(R + i); }
__device__ __forceinline__ float half_at(const uint16_t* t, size_t i) {
  return __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short*>(t) + i)));
}
// textureSampleLevel of an r16float texture through the engine's linear,
// clamp-to-edge sampler (engine.ts:270) with f32 weights: c = uvw * size - 0.5,
// i = floor(c), t = c - i, clamped indices, blended along x, then y, then z.
__device__ __forceinline__ int floor_index(float f, int n) { return (int)(f < -1.0f ? -1.0f : (f > (float)n ? (float)n : f)); }
__device__ float sample3(const uint16_t* tex, int w, int h, int d, V3 uvw) {
  const float cx = uvw.x * (float)w - 0.5f, cy = uvw.y * (float)h - 0.5f, cz = uvw.z * (float)d - 0.5f;
  const float fx = floorf(cx), fy = floorf(cy), fz = floorf(cz);
  const float tx = cx - fx, ty = cy - fy, tz = cz - fz;
  const int i = floor_index(fx, w), j = floor_index(fy, h), k = floor_index(fz, d);
  auto at = [&](int x, int y, int z) {
    x = x < 0 ? 0 : (x >= w ? w - 1 : x);
    y = y < 0 ? 0 : (y >= h ? h - 1 : y);
    z = z < 0 ? 0 : (z >= d ? d - 1 : z);
    return half_at(tex, ((size_t)z * (size_t)h + (size_t)y) * (size_t)w + (size_t)x);
  };
  const float c00 = at(i, j, k) * (1.0f - tx) + at(i + 1, j, k) * tx;
  const float c10 = at(i, j + 1, k) * (1.0f - tx) + at(i + 1, j + 1, k) * tx;
  const float c01 = at(i, j, k + 1) * (1.0f - tx) + at(i + 1, j, k + 1) * tx;
  const float c11 = at(i, j + 1, k + 1) * (1.0f - tx) + at(i + 1, j + 1, k + 1) * tx;
  const float c0 = c00 * (1.0f - ty) + c10 * ty, c1 = c01 * (1.0f - ty) + c11 * ty;
  return c0 * (1.0f - tz) + c1 * tz;
}

// rigWeight, rigHinge, rigAngle, rigScale, rigRotate (car-model.ts:70-118); the
// RIG constants (car-model.ts:44-49) as the reference interpolates them
__device__ float rig_weight(uint32_t part, float z) {
  if (part == 1u || part == 2u) {
    const float az = ab(z);
    return sstep(0.16f, 0.22f, az) * (1.0f - sstep(0.5f, 0.56f, az));
  }
  return (part == 3u || part == 4u) ? 1.0f : 0.0f;
}
__device__ V2 rig_hinge(const float4* R, uint32_t part, float z) {
  if (part == 3u) { const float4 g = rig_at(R, RIG_HINGES); return v2(g.z, g.w); }
  if (part == 4u) { const float4 g = rig_at(R, RIG_HINGES); return v2(g.x, g.y); }
  const float f = clmp(ab(z) / 0.01f, 0.0f, 70.0f);
  const uint32_t i = (uint32_t)floorf(f);
  const uint32_t j = (i + 1u) < 70u ? i + 1u : 70u;
  const float4 a = rig_at(R, (int)i), b = rig_at(R, (int)j);
  const float t = f - (float)i;
  return part == 1u ? mix2(v2(a.x, a.y), v2(b.x, b.y), t) : mix2(v2(a.z, a.w), v2(b.z, b.w), t);
}
__device__ float rig_angle(const float4* R, uint32_t part, float z) {
  const float4 an = rig_at(R, RIG_ANGLES);
  float a = 0.0f;
  if (part == 1u) a = an.x;
  else if (part == 2u) a = an.y;
  else if (part == 3u) a = an.z;
  else if (part == 4u) a = an.w;
  if (part == 3u || part == 4u) a = a + rig_at(R, RIG_EXTRA).x * sstep(0.12f, 0.48f, ab(z));
  return a * rig_weight(part, z);
}
__device__ float rig_scale(const float4* R, uint32_t part) {
  const float ey = rig_at(R, RIG_EXTRA).y;
  if (part == 3u) return ey;
  if (part == 1u || part == 2u) return 1.0f - (1.0f - ey) * 0.65f;
  return 1.0f;
}
// rigRotate with dir = -1 (the distance field's direction)
__device__ V3 rig_rotate_back(const Scene& S, V3 p, uint32_t part) {
  if (part == 0u || part > 4u) return p;
  const float a = rig_angle(S.car.rig, part, p.z) * -1.0f;
  const float k = rig_scale(S.car.rig, part);
  const V2 h = rig_hinge(S.car.rig, part, p.z);
  const float c = wtm::cosf(a), s = wtm::sinf(a);
  V2 d = v2(p.x, p.y) - h;
  d = v2(c * d.x - s * d.y, s * d.x + c * d.y);
  d = v2(dv(d.x, k), dv(d.y, k));
  return v3(h.x + d.x, h.y + d.y, p.z);
}
// podWeight, podDeform (car-model.ts:121-135), dir = -1
__device__ float pod_weight(V3 p) {
  return sstep(1.85f, 2.25f, p.x) * (1.0f - sstep(3.55f, 4.05f, p.x)) * sstep(0.12f, 0.2f, p.y) *
         (1.0f - sstep(0.6f, 0.7f, p.y)) * sstep(0.26f, 0.4f, ab(p.z));
}
__device__ V3 pod_deform_back(const Scene& S, V3 p) {
  const float c = rig_at(S.car.rig, RIG_EXTRA).z * pod_weight(p);
  if (c <= 0.0f) return p;
  const float az = ab(p.z);
  const float kz = dv(1.0f, 1.0f - c);
  const float ky = dv(1.0f, 1.0f - 0.45f * c);
  const float nz = az > 0.26f ? 0.26f + (az - 0.26f) * kz : az;
  const float sg = p.z > 0.0f ? 1.0f : (p.z < 0.0f ? -1.0f : 0.0f);
  return v3(p.x, 0.12f + (p.y - 0.12f) * ky, sg * nz);
}
// w17BodyFrame (f1.ts:329-334), with the rake of toBodyFrame
__device__ V3 w17_body_frame(const Scene& S, V3 pw) {
  const float dx = pw.x - FA, dy = pw.y - S.s.ride_h;
  return v3(FA + dx * S.rake_c + dy * S.rake_s, W17_BASE_RIDE - dx * S.rake_s + dy * S.rake_c, pw.z);
}
// sdW17Body (f1.ts:335-341)
__device__ float sd_w17_body(const Scene& S, V3 p) {
  const V3 ext = v3(368.0f * W17_H, 84.0f * W17_H, 67.0f * W17_H);
  const V3 half = ext * 0.5f;
  const float box = sd_box(p - v3(-0.3f + half.x, 0.0f + half.y, 0.0f + half.z), half);
  if (box > 0.0f) return box + 0.07f;
  const V3 uvw = v3(dv(dv(p.x - -0.3f, W17_H) + 0.5f, 368.0f), dv(dv(p.y - 0.0f, W17_H) + 0.5f, 84.0f),
                    dv(dv(p.z - 0.0f, W17_H) + 0.5f, 67.0f));
  return sample3(S.car.body, 368, 84, 67, uvw);
}
// sdW17Part (f1.ts:342-353)
__device__ __noinline__ float sd_w17_part(const Scene& S, V3 pb, uint32_t part) {
  const float4 g0 = rig_at(S.car.rig, RIG_GRIDS + (int)(part - 1u) * 2), g1 = rig_at(S.car.rig, RIG_GRIDS + (int)(part - 1u) * 2 + 1);
  const V3 q = rig_rotate_back(S, pb, part);
  const V3 ext = v3((g1.x - 1.0f) * g0.w, (g1.y - 1.0f) * g0.w, (g1.z - 1.0f) * g0.w);
  const V3 half = ext * 0.5f;
  const float box = sd_box(q - v3(g0.x + half.x, g0.y + half.y, g0.z + half.z), half);
  if (box > 0.0f) return box + 0.03f;
  const V3 cell = v3(dv(q.x - g0.x, g0.w), dv(q.y - g0.y, g0.w), dv(q.z - g0.z, g0.w));
  const float ax = (float)S.car.pdims[0], ay = (float)S.car.pdims[1], az = (float)S.car.pdims[2];
  const V3 uvw = v3(dv(cell.x + 0.5f, ax), dv(cell.y + 0.5f, ay), dv(cell.z + g1.w + 0.5f, az));
  const float sc = rig_scale(S.car.rig, part);
  return sample3(S.car.parts, (int)S.car.pdims[0], (int)S.car.pdims[1], (int)S.car.pdims[2], uvw) * mn(sc, 1.0f);
}
// sdW17 (f1.ts:354-369)
__device__ __noinline__ V2 sd_w17(const Scene& S, V3 pw) {
  const V3 pa = v3(pw.x, pw.y, ab(pw.z));
  const V3 p = w17_body_frame(S, pa);
  const float squeeze = 1.0f - rig_at(S.car.rig, RIG_EXTRA).z * pod_weight(p);
  V2 res = v2(sd_w17_body(S, pod_deform_back(S, p)) * 0.95f * squeeze, 12.0f);
  const float4 fly = rig_at(S.car.rig, RIG_FLY);
  if (fly.z > 0.5f && p.x < 0.85f && p.y < 0.6f)
    res = op_u(res, v2(mn(mn(sd_w17_part(S, p, 1u), sd_w17_part(S, p, 2u)), sd_w17_part(S, p, 5u)) * 0.95f, 7.0f));
  if (fly.w > 0.5f && p.x > 4.4f && p.y > 0.5f)
    res = op_u(res, v2(mn(mn(sd_w17_part(S, p, 3u), sd_w17_part(S, p, 4u)), sd_w17_part(S, p, 6u)) * 0.95f, 8.0f));
  const V3 front = v3(1.0f, 0.36f, 0.779f), rear = v3(4.4f, 0.351f, 0.737f);
  res = op_u(res, v2(mn(sd_tyre(pa, front, 0.175f), sd_cyl_z(pa - front, 0.234f, 0.15f)), 2.0f));
  res = op_u(res, v2(mn(sd_tyre(pa, rear, 0.205f), sd_cyl_z(pa - rear, 0.234f, 0.18f)), 2.0f));
  return res;
}
// w17Duct (f1.ts:374-383)
__device__ float w17_duct(const Scene& S, V3 pw) {
  if (S.s.duct <= 0.0f) return 1e3f;
  const V3 p = pod_deform_back(S, w17_body_frame(S, v3(pw.x, pw.y, ab(pw.z))));
  const float k = S.s.duct;
  const float mouth = sd_capsule(p, v3(2.05f, 0.52f, 0.58f), v3(3.0f, 0.50f, 0.48f), 0.09f * k);
  const float main = sd_capsule(p, v3(2.05f, 0.55f, 0.47f), v3(3.25f, 0.46f, 0.43f), 0.1f * k);
  const float exit = sd_capsule(p, v3(3.25f, 0.46f, 0.43f), v3(4.1f, 0.40f, 0.32f), 0.085f * k);
  return mn(mn(mouth, main), exit);
}
// w17Emission (f1.ts:386-394)
__device__ float w17_emission(const Scene& S, V3 pw) {
  const V3 pa = v3(pw.x, pw.y, ab(pw.z));
  const V3 p = w17_body_frame(S, pa);
  float e = 0.0f;
  if (len2(v2(pa.x - 1.0f, pa.y - 0.36f)) < 0.2f && ab(pa.z - (0.779f - 0.215f)) < 0.1f) e = mx(e, S.s.heat_brakes);
  if (len2(v2(pa.x - 4.4f, pa.y - 0.351f)) < 0.2f && ab(pa.z - (0.737f - 0.245f)) < 0.1f) e = mx(e, S.s.heat_brakes * 0.8f);
  if (len3(p - v3(5.07f, 0.53f, 0.0f)) < 0.1f) e = mx(e, S.s.heat_engine);
  if (p.x > 3.7f && p.x < 4.3f && p.y > 0.2f && p.y < 0.5f && p.z > 0.18f && p.z < 0.48f) e = mx(e, S.s.heat_rad);
  if (p.x > 4.15f && p.x < 4.65f && p.y > 0.5f && p.z < 0.16f) e = mx(e, S.s.heat_rad * 1.4f);
  return e;
}

__device__ V2 scene_sdf(const Scene& S, const F1Tables& F, V3 p) {
  switch (S.s.kind) {
    case WT_KIND_F1: return sd_f1(S, F, p);
    case WT_KIND_SPHERE: return v2(len3(p - v3(2.6f, 1.0f, 0.0f)) - 0.6f, 6.0f);
    case WT_KIND_CUBE: return v2(sd_rbox(p - v3(2.6f, 1.0f, 0.0f), v3(0.5f, 0.5f, 0.5f), 0.03f), 6.0f);
    case WT_KIND_WING: return v2(sd_wing(p, v2(1.6f, 1.2f), 1.8f, -S.s.aoa, 0.24f, -1.25f, 1.25f), 6.0f);
    case WT_KIND_W17: return S.car.body ? sd_w17(S, p) : v2(1e3f, 0.0f);
    case WT_KIND_BOX:
      return v2(sd_box(p - v3(S.s.box_center[0], S.s.box_center[1], S.s.box_center[2]),
                       v3(S.s.box_half[0], S.s.box_half[1], S.s.box_half[2])), 6.0f);
    default: return v2(1e3f, 0.0f);
  }
}

uint32_t host_variant(float v) {  // u32(v + 0.5), saturating
  const float t = v + 0.5f;
  return (t == t && t > 0.0f) ? (t >= 4294967296.0f ? 4294967295u : (uint32_t)t) : 0u;
}
// The parts of f1.ts:42-320.
void f1_tables(const Scene& S, F1Tables& F) {
  const float b = S.s.ride_h, yw = 0.19f + b * 0.45f, yr = b + 0.80f, ff = S.s.front_flap;
  auto f4 = [](float x, float y, float z, float w) { return make_float4(x, y, z, w); };
  auto at = [&](float x, float y, float z) { return v3(x, b + y, z); };
  auto taper = [&](uint32_t i, float x0, float x1, V2 c0, V2 c1, V2 s0, V2 s1, float r0, float r1) {
    float4* q = F.taper[i];
    q[0] = f4(x0, x1 - x0, 0.5f * (x0 + x1), 0.5f * (x1 - x0));
    q[1] = f4(r0, r1, 0.0f, 0.0f);
    q[2] = f4(c0.x, c0.y, c1.x, c1.y);
    q[3] = f4(s0.x, s0.y, s1.x, s1.y);
  };
  auto cap = [&](uint32_t i, V3 a, V3 e, float r) {
    const float x = e.x - a.x, y = e.y - a.y, z = e.z - a.z;
    F.cap[i][0] = f4(a.x, a.y, a.z, r);
    F.cap[i][1] = f4(x, y, z, x * x + y * y + z * z);
  };
  auto box = [&](uint32_t i, V3 c, V3 h, float r) {
    F.box[i][0] = f4(c.x, c.y, c.z, r);
    F.box[i][1] = f4(h.x - r, h.y - r, h.z - r, 0.0f);
  };
  auto ell = [&](uint32_t i, V3 c, V3 r) {
    F.ell[i][0] = f4(c.x, c.y, c.z, 0.0f);
    F.ell[i][1] = f4(r.x, r.y, r.z, 0.0f);
    F.ell[i][2] = f4(r.x * r.x, r.y * r.y, r.z * r.z, 0.0f);
  };
  auto wing = [&](uint32_t i, float lx, float ly, float chord, float ang, float thick, float z0, float z1, float rise,
                  float tap, float curl) {
    F.wing[i][0] = f4(lx, ly, chord, ang);
    F.wing[i][1] = f4(thick, z0, z1, rise);
    F.wing[i][2] = f4(tap, curl, 0.0f, 0.0f);
  };
  auto y0z = [&](float y) { return v2(b + y, 0.0f); };
  auto around = [&](uint32_t i, V3 lo, V3 hi, float factor, float addend) {
    F.around[i][0] = f4(lo.x, lo.y, lo.z, factor);
    F.around[i][1] = f4(hi.x, hi.y, hi.z, addend);
  };
  around(K_SCUTTLE, at(1.20f, 0.17f, -0.29f), at(2.24f, 0.67f, 0.29f), 1.25f, 0.08f);
  around(K_NOSE, v3(-0.06f, fminf(b, yw - 0.02f), -0.17f), v3(1.26f, fmaxf(b + 0.51f, yw + 0.02f), 0.17f), 2.0f, 0.09f);
  around(K_COVER, at(2.96f, 0.28f, -0.31f), at(4.86f, 0.92f, 0.31f), 1.25f, 0.10f);
  around(K_KEEL, at(1.30f, 0.03f, -0.19f), at(4.70f, 0.41f, 0.19f), 1.25f, 0.08f);
  around(K_POD, at(2.30f, 0.15f, 0.18f), at(4.25f, 0.62f, 0.80f), 1.25f, 0.12f);
  around(K_AIRBOX, at(2.85f, 0.73f, -0.12f), at(3.19f, 0.95f, 0.12f), 1.0f, 0.10f);
  around(K_COCKPIT, at(2.20f, 0.59f, -0.215f), at(3.04f, 0.85f, 0.215f), -1.0f, -0.03f);
  around(K_CABIN, at(2.13f, 0.48f, -0.15f), at(3.06f, 0.96f, 0.69f), 1.25f, 0.018f);
  around(K_HELMET, at(2.52f, 0.56f, -0.15f), at(2.82f, 0.86f, 0.15f), 1.25f, 0.0f);
  around(K_HALO, at(2.13f, 0.58f, -0.04f), at(3.06f, 0.96f, 0.30f), 1.0f, 0.0225f);
  around(K_MIRROR, at(2.28f, 0.48f, 0.44f), at(2.47f, 0.71f, 0.69f), 1.0f, 0.0f);
  around(K_SUSF, v3(0.84f, fminf(b + 0.15f, 0.21f), 0.13f), v3(1.44f, fmaxf(b + 0.49f, 0.54f), 0.66f), 1.0f, 0.0f);
  around(K_SUSR, v3(4.26f, fminf(b + 0.13f, 0.20f), 0.14f), v3(4.84f, fmaxf(b + 0.44f, 0.55f), 0.57f), 1.0f, 0.0f);
  around(K_TAIL, at(4.78f, 0.26f, -0.07f), at(5.42f, 0.50f, 0.07f), 1.25f, 0.0f);
  around(K_FIN, at(3.40f, 0.64f, -0.008f), at(4.50f, 0.84f, 0.008f), 1.0f, 0.0f);
  around(K_LIGHT, at(4.90f, 0.26f, -0.07f), at(5.42f, 0.50f, 0.07f), 1.0f, 0.0f);
  around(K_FENCE, at(1.56f, 0.0f, 0.248f), at(2.12f, 0.16f, 0.432f), 1.0f, 0.0f);
  around(K_STRAKE, at(4.28f, 0.0f, 0.292f), at(4.96f, 0.34f, 0.508f), 1.0f, 0.0f);
  around(K_EDGE, at(2.23f, 0.03f, 0.76f), at(3.87f, 0.085f, 0.81f), 1.0f, 0.0f);

  box(B_BODY, at(2.72f, 0.52f, 0.0f), v3(2.74f, 0.62f, 0.95f), 0.0f);
  taper(T_MID, 2.20f, 3.06f, y0z(0.42f), y0z(0.42f), v2(0.25f, 0.30f), v2(0.25f, 0.34f), 0.16f, 0.16f);
  const uint32_t nose = host_variant(S.s.nose);
  const float x0 = (nose == 1u) ? 0.34f : 0.10f, y0 = b + ((nose == 2u) ? 0.25f : 0.17f);
  const V2 s0 = nose == 1u ? v2(0.075f, 0.15f) : (nose == 2u ? v2(0.045f, 0.075f) : v2(0.055f, 0.11f));
  taper(T_NOSE, x0, 1.26f, v2(y0, 0.0f), y0z(0.36f), s0, v2(0.15f, 0.17f), 0.04f, 0.12f);
  ell(E_NOSE, v3(x0 + 0.02f, y0, 0.0f), v3(0.09f, s0.x, s0.y));
  F.pylon = nose != 0u;
  box(B_PYLON, v3(x0 + 0.06f, 0.5f * (yw + y0), 0.09f), v3(0.09f, 0.5f * (y0 - yw) + 0.02f, 0.006f), 0.004f);
  taper(T_SCUTTLE, 1.20f, 2.24f, y0z(0.36f), y0z(0.42f), v2(0.15f, 0.17f), v2(0.25f, 0.29f), 0.12f, 0.16f);
  const uint32_t cover = host_variant(S.s.cover);
  if (cover == 1u) taper(T_COVER, 2.96f, 4.86f, y0z(0.60f), y0z(0.40f), v2(0.32f, 0.31f), v2(0.12f, 0.13f), 0.15f, 0.08f);
  else if (cover == 2u) taper(T_COVER, 2.96f, 4.70f, y0z(0.57f), y0z(0.34f), v2(0.29f, 0.19f), v2(0.06f, 0.05f), 0.12f, 0.04f);
  else taper(T_COVER, 2.96f, 4.86f, y0z(0.58f), y0z(0.36f), v2(0.30f, 0.24f), v2(0.08f, 0.07f), 0.14f, 0.06f);
  taper(T_KEEL, 1.30f, 4.70f, y0z(0.22f), y0z(0.20f), v2(0.19f, 0.19f), v2(0.17f, 0.14f), 0.06f, 0.05f);
  const uint32_t pod = host_variant(S.s.sidepod);
  F.pod_k[0] = 0.05f; F.pod_k[1] = 0.04f; F.pod_k[2] = 0.02f;
  F.pod_caps = pod == 1u ? 0u : (pod == 2u ? 2u : 1u);
  cap(C_CARVE + 1, at(2.55f, 0.66f, 0.52f), at(4.00f, 0.40f, 0.36f), 0.11f);
  if (pod == 1u) {
    taper(T_POD, 2.30f, 4.05f, v2(b + 0.40f, 0.36f), v2(b + 0.24f, 0.24f), v2(0.16f, 0.08f), v2(0.07f, 0.05f), 0.06f, 0.04f);
    cap(C_CARVE, v3(0.0f, 0.0f, 0.0f), v3(1.0f, 0.0f, 0.0f), 0.0f);
    box(B_CARVE, at(2.27f, 0.42f, 0.38f), v3(0.06f, 0.12f, 0.05f), 0.03f);
  } else if (pod == 2u) {
    taper(T_POD, 2.30f, 4.25f, v2(b + 0.41f, 0.52f), v2(b + 0.24f, 0.30f), v2(0.18f, 0.28f), v2(0.08f, 0.11f), 0.10f, 0.05f);
    cap(C_CARVE, at(2.30f, 0.13f, 0.84f), at(3.70f, 0.08f, 0.58f), 0.15f);
    box(B_CARVE, at(2.28f, 0.47f, 0.57f), v3(0.06f, 0.10f, 0.17f), 0.05f);
  } else if (pod == 3u) {
    taper(T_POD, 2.30f, 4.25f, v2(b + 0.47f, 0.52f), v2(b + 0.26f, 0.28f), v2(0.15f, 0.25f), v2(0.07f, 0.10f), 0.12f, 0.05f);
    cap(C_CARVE, at(2.25f, 0.17f, 0.86f), at(3.70f, 0.10f, 0.56f), 0.22f);
    box(B_CARVE, at(2.28f, 0.52f, 0.55f), v3(0.06f, 0.07f, 0.17f), 0.04f);
  } else {
    taper(T_POD, 2.30f, 4.25f, v2(b + 0.41f, 0.52f), v2(b + 0.22f, 0.28f), v2(0.18f, 0.25f), v2(0.07f, 0.10f), 0.12f, 0.05f);
    cap(C_CARVE, at(2.30f, 0.13f, 0.82f), at(3.70f, 0.08f, 0.56f), 0.16f);
    box(B_CARVE, at(2.28f, 0.47f, 0.57f), v3(0.06f, 0.10f, 0.17f), 0.05f);
  }
  box(B_AIRBOX, at(3.02f, 0.84f, 0.0f), v3(0.17f, 0.11f, 0.12f), 0.08f);
  ell(E_AIR, at(2.85f, 0.86f, 0.0f), v3(0.09f, 0.066f, 0.078f));
  box(B_COCKPIT, at(2.62f, 0.72f, 0.0f), v3(0.42f, 0.13f, 0.215f), 0.10f);
  ell(E_HELMET, at(2.67f, 0.71f, 0.0f), v3(0.15f, 0.13f, 0.12f));
  cap(C_HALO, at(2.17f, 0.62f, 0.0f), at(2.36f, 0.90f, 0.0f), 0.034f);
  cap(C_HALO + 1, at(2.36f, 0.90f, 0.0f), at(2.52f, 0.92f, 0.20f), 0.031f);
  cap(C_HALO + 2, at(2.52f, 0.92f, 0.20f), at(2.82f, 0.88f, 0.26f), 0.031f);
  cap(C_HALO + 3, at(2.82f, 0.88f, 0.26f), at(3.02f, 0.74f, 0.25f), 0.033f);
  box(B_MIRROR, at(2.32f, 0.67f, 0.60f), v3(0.035f, 0.035f, 0.085f), 0.02f);
  cap(C_MIRROR, at(2.36f, 0.66f, 0.53f), at(2.45f, 0.50f, 0.46f), 0.011f);
  const float fz = FWZ - FHW - 0.05f, rz = RWZ - RHW - 0.05f;
  cap(C_SUSF, at(1.10f, 0.43f, 0.17f), v3(FA + 0.02f, WR + 0.16f, fz), 0.017f);
  cap(C_SUSF + 1, at(1.42f, 0.40f, 0.17f), v3(FA + 0.02f, WR + 0.16f, fz), 0.017f);
  cap(C_SUSF + 2, at(0.98f, 0.19f, 0.15f), v3(FA, WR - 0.13f, fz), 0.017f);
  cap(C_SUSF + 3, at(1.38f, 0.17f, 0.15f), v3(FA, WR - 0.13f, fz), 0.017f);
  cap(C_SUSF + 4, v3(FA + 0.03f, WR - 0.10f, FWZ - FHW - 0.07f), at(1.20f, 0.47f, 0.16f), 0.014f);
  cap(C_SUSF + 5, at(0.86f, 0.29f, 0.16f), v3(0.88f, WR + 0.02f, fz), 0.013f);
  cap(C_SUSR, at(4.30f, 0.42f, 0.20f), v3(RA, WR + 0.17f, rz), 0.017f);
  cap(C_SUSR + 1, at(4.78f, 0.40f, 0.16f), v3(RA, WR + 0.17f, rz), 0.017f);
  cap(C_SUSR + 2, at(4.28f, 0.16f, 0.24f), v3(RA, WR - 0.14f, rz), 0.017f);
  cap(C_SUSR + 3, at(4.82f, 0.15f, 0.18f), v3(RA, WR - 0.14f, rz), 0.017f);
  cap(C_SUSR + 4, v3(RA - 0.03f, WR + 0.14f, RWZ - RHW - 0.07f), at(4.40f, 0.18f, 0.22f), 0.014f);
  taper(T_TAIL, 4.78f, 5.40f, y0z(0.33f), y0z(0.33f), v2(0.07f, 0.065f), v2(0.045f, 0.045f), 0.04f, 0.03f);
  box(B_FIN, at(3.95f, 0.74f, 0.0f), v3(0.55f, 0.10f, 0.008f), 0.006f);
  box(B_LIGHT, at(5.405f, 0.33f, 0.0f), v3(0.012f, 0.028f, 0.05f), 0.006f);
  cap(C_EXHAUST, at(4.95f, 0.44f, 0.0f), at(5.13f, 0.45f, 0.0f), 0.042f);
  cap(C_BORE, at(5.0f, 0.44f, 0.0f), at(5.2f, 0.45f, 0.0f), 0.028f);
  box(B_FLOOR, at(3.26f, 0.2f, 0.4f), v3(1.75f, 0.22f, 0.42f), 0.0f);
  for (int i = 0; i < 2; i++) {
    box(B_FENCE + i, at(1.84f, 0.08f, 0.26f + (float)i * 0.16f), v3(0.28f, 0.08f, 0.012f), 0.0f);
    box(B_STRAKE + i, at(4.62f, 0.17f, 0.30f + (float)i * 0.20f), v3(0.34f, 0.17f, 0.008f), 0.0f);
  }
  cap(C_EDGE, at(2.25f, 0.065f, 0.79f), at(3.85f, 0.05f, 0.78f), 0.02f);
  box(B_FRONT, v3(0.24f, yw + 0.17f, 0.48f), v3(0.36f, 0.34f, 0.50f), 0.0f);
  box(B_REAR, at(5.20f, 0.64f, 0.27f), v3(0.46f, 0.56f, 0.29f), 0.0f);
  const uint32_t fw = host_variant(S.s.front_wing);
  auto plate = [&](float x, float y, float hx, float hy, float r) {
    F.ep[0] = x; F.ep[1] = y; F.ep[2] = hx; F.ep[3] = hy; F.ep[4] = r;
  };
  F.front_wings = fw == 3u ? 2u : 4u;
  if (fw == 1u) {
    wing(0, -0.03f, yw, 0.31f, 2.0f * DEG + ff * 0.1f, 0.034f, 0.0f, 0.94f, 0.03f, 0.2f, 0.5f);
    wing(1, 0.21f, yw + 0.036f, 0.17f, 9.0f * DEG + ff * 0.45f, 0.024f, 0.0f, 0.94f, 0.15f, 0.35f, 0.3f);
    wing(2, 0.335f, yw + 0.075f + ff * 0.03f, 0.14f, 17.0f * DEG + ff * 0.75f, 0.020f, 0.10f, 0.94f, 0.19f, 0.35f, 0.25f);
    wing(3, 0.425f, yw + 0.118f + ff * 0.07f, 0.12f, 26.0f * DEG + ff, 0.018f, 0.12f, 0.94f, 0.22f, 0.4f, 0.25f);
    plate(0.25f, yw + 0.17f, 0.29f, 0.20f, 0.08f);
  } else if (fw == 2u) {
    wing(0, -0.03f, yw, 0.31f, 3.0f * DEG + ff * 0.1f, 0.034f, 0.0f, 0.94f, -0.02f, 0.15f, 0.55f);
    wing(1, 0.21f, yw + 0.04f, 0.19f, 13.0f * DEG + ff * 0.45f, 0.024f, 0.0f, 0.94f, -0.04f, 0.35f, 0.35f);
    wing(2, 0.35f, yw + 0.085f + ff * 0.03f, 0.16f, 22.0f * DEG + ff * 0.75f, 0.020f, 0.06f, 0.94f, -0.06f, 0.4f, 0.35f);
    wing(3, 0.45f, yw + 0.13f + ff * 0.07f, 0.13f, 31.0f * DEG + ff, 0.018f, 0.08f, 0.94f, -0.08f, 0.45f, 0.35f);
    plate(0.25f, yw + 0.06f, 0.29f, 0.10f, 0.06f);
  } else if (fw == 3u) {
    wing(0, -0.03f, yw, 0.30f, 1.0f * DEG + ff * 0.05f, 0.030f, 0.0f, 0.94f, 0.0f, 0.1f, 0.6f);
    wing(1, 0.20f, yw + 0.03f, 0.16f, 4.0f * DEG + ff * 0.3f, 0.022f, 0.0f, 0.94f, 0.02f, 0.2f, 0.5f);
    plate(0.22f, yw + 0.05f, 0.26f, 0.085f, 0.05f);
  } else {
    wing(0, -0.03f, yw, 0.31f, 2.0f * DEG + ff * 0.1f, 0.034f, 0.0f, 0.94f, 0.06f, 0.2f, 0.5f);
    wing(1, 0.21f, yw + 0.036f, 0.17f, 9.0f * DEG + ff * 0.45f, 0.024f, 0.0f, 0.94f, 0.09f, 0.25f, 0.45f);
    wing(2, 0.335f, yw + 0.075f + ff * 0.03f, 0.14f, 17.0f * DEG + ff * 0.75f, 0.020f, 0.10f, 0.94f, 0.11f, 0.25f, 0.4f);
    wing(3, 0.425f, yw + 0.118f + ff * 0.07f, 0.12f, 26.0f * DEG + ff, 0.018f, 0.12f, 0.94f, 0.13f, 0.25f, 0.4f);
    plate(0.25f, yw + 0.085f, 0.29f, 0.115f, 0.07f);
  }
  box(B_FOOT, v3(0.22f, yw - 0.008f, 0.94f - 0.04f), v3(0.30f, 0.006f, 0.06f), 0.004f);
  wing(4, 4.98f, yr, S.chord_m, S.ang_m, 0.05f, 0.0f, 0.50f, S.rise_m, 0.12f, 0.22f);
  wing(5, (4.98f + S.rear_c * (S.chord_m - 0.01f)) + -0.03f, (yr + S.rear_s * (S.chord_m - 0.01f)) + 0.035f, S.chord_f,
       S.ang_f, 0.03f, 0.0f, 0.49f, S.rise_m * 0.8f, 0.10f, 0.28f);
  cap(C_POST, v3(5.26f, yr + 0.05f, 0.0f), v3(5.30f, yr + 0.12f, 0.0f), 0.024f);
  box(B_POST, v3(5.09f, 0.5f * (b + 0.36f + yr + 0.06f), 0.06f), v3(0.07f, 0.5f * (yr + 0.06f - b - 0.36f), 0.008f), 0.006f);
  for (int i = 0; i < 2; i++) {
    const V3 c = i == 0 ? v3(FA, WR26, FWZ * BODY_Z) : v3(RA26, WR26, RWZ * BODY_Z);
    const float hw = i == 0 ? FHW26 : RHW26;
    box(B_WHEEL + i, c, v3(WR26 + 0.02f, WR26 + 0.02f, hw + 0.2f), 0.0f);
    box(B_DUCT + i, v3(c.x - 0.04f, c.y + 0.21f, c.z - hw - 0.05f), v3(0.16f, 0.012f, 0.05f), 0.006f);
  }
}

// Shape plus its shape-wide constants.
SceneParam make_scene(const wt_shape& shape, const CarView& car = CarView{}) {
  SceneParam P;
  Scene& S = P.s;
  S.s = shape;
  S.car = car;
  // Shape-wide constants, evaluated once (same functions and operation order as per cell).
  const float th = wtm::atanf((shape.rear_ride - shape.ride_h) / (RA26 - FA));
  S.rake_c = wtm::cosf(th);
  S.rake_s = wtm::sinf(th);
  // Rear-wing variant parameters (f1.ts:260-272).
  const float vr = shape.rear_wing + 0.5f;
  const uint32_t v = (vr == vr && vr > 0.0f) ? (vr >= 4294967296.0f ? 4294967295u : (uint32_t)vr) : 0u;
  S.chord_m = 0.36f; S.ang_m = shape.rear_main; S.rise_m = -0.10f;
  S.chord_f = 0.26f; S.ang_f = shape.rear_flap; S.ep_hx = 0.33f; S.ep_hy = 0.29f;
  if (v == 1u) {
    S.chord_m = 0.42f; S.ang_m = S.ang_m + 3.0f * DEG; S.rise_m = -0.15f;
    S.chord_f = 0.32f; S.ang_f = S.ang_f + 6.0f * DEG; S.ep_hx = 0.36f; S.ep_hy = 0.33f;
  } else if (v == 2u) {
    S.chord_m = 0.27f; S.ang_m = S.ang_m - 5.0f * DEG; S.rise_m = 0.02f;
    S.chord_f = 0.15f; S.ang_f = S.ang_f * 0.55f; S.ep_hx = 0.30f; S.ep_hy = 0.25f;
  }
  S.rear_c = wtm::cosf(S.ang_m);
  S.rear_s = wtm::sinf(S.ang_m);
  S.f1 = nullptr;
  P.f1 = F1Tables{};
  if (shape.kind == WT_KIND_F1) f1_tables(S, P.f1);
  return P;
}

}  // namespace
}  // namespace wt
