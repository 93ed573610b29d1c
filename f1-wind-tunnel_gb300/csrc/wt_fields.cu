// Field consumers of the reference as CUDA kernels into headless buffers:
//   sampleFlow / vorticityAt   FIELD_SAMPLING, src/engine/wgsl.ts:324-366
//   particle pass (RK2)        PARTICLES_SIM, wgsl.ts:516-594 (+ VIEW, wgsl.ts:430-457)
//   streamline pass            STREAM_SIM, src/engine/render-wgsl.ts:520-576
// They read the (u, rho) fields of the last step call and the temperatures.
// Arithmetic follows the WGSL text operation for operation (build with
// -fmad=false) and the WGSL builtin definitions the oracle's runtime models
// (min/max/clamp by comparison, mix(a, b, t) = a (1 - t) + b t, dot summed
// x, y, z, length = sqrt(dot), normalize = componentwise division by the
// length, float -> int truncating and saturating), so results are bit-identical
// to the reference's shaders run on the CPU.  sin/cos come from wt_fmath.h.
#include <cuda_runtime.h>
#include <stdint.h>

#include "wt_fieldfn.cuh"
#include "wt_fields.h"
#include "wt_fmath.h"
#include "wt_lattice.cuh"

namespace wt {
namespace {


// pcg hash and rand (wgsl.ts:531-539)
__device__ __forceinline__ uint32_t pcg(uint32_t v) {
  const uint32_t s = v * 747796405u + 2891336453u;
  const uint32_t w = ((s >> ((s >> 28u) + 4u)) ^ s) * 277803737u;
  return (w >> 22u) ^ w;
}
__device__ __forceinline__ float rnd(uint32_t& seed) {
  seed = pcg(seed);
  return (float)seed / 4294967296.0f;  // the reference's 4294967295.0 as f32
}

__device__ __forceinline__ V3 domain_max(const FieldGrid& g) {
  return v3(g.ox + (float)g.nx * g.h, g.oy + (float)g.ny * g.h, g.oz + (float)g.nz * g.h);
}

// spawn (wgsl.ts:542-562)
__device__ void spawn(const FieldGrid& g, const PSimArgs& ps, uint32_t i, uint32_t& seed, float4& pos, float4& vel) {
  V3 p;
  if (ps.spawnMode == 1u) {
    const uint32_t lanes = ps.rakeRows * ps.rakeCols;
    const uint32_t lane = i % lanes;
    const uint32_t row = lane / ps.rakeCols, col = lane % ps.rakeCols;
    const float fy = ((float)row + 0.5f) / (float)ps.rakeRows;
    const float fz = ((float)col + 0.5f) / (float)ps.rakeCols;
    p = v3(ps.smin[0], wmix(ps.smin[1], ps.smax[1], fy), wmix(ps.smin[2], ps.smax[2], fz));
    const float r0 = rnd(seed) * 0.12f;
    const float r1 = (rnd(seed) - 0.5f) * 0.012f;
    const float r2 = (rnd(seed) - 0.5f) * 0.012f;
    p = add(p, v3(r0, r1, r2));
  } else {
    const float r0 = rnd(seed), r1 = rnd(seed), r2 = rnd(seed);
    p = v3(ps.smin[0] + r0 * 0.15f, wmix(ps.smin[1], ps.smax[1], r1), wmix(ps.smin[2], ps.smax[2], r2));
  }
  if (ps.scatter != 0u) p.x = wmix(ps.smin[0], domain_max(g).x - g.h * 2.0f, rnd(seed));
  pos = make_float4(p.x, p.y, p.z, 0.0f);
  vel = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
}

// Particle pass cs_main (wgsl.ts:566-594): one thread per particle.
__global__ void particles_kernel(FieldGrid g, PSimArgs ps, ViewArgs view, float4* __restrict__ parts) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ps.count) return;
  uint32_t seed = pcg(i * 9781u + ps.frame * 6271u + 17u);
  float4 pos = parts[2 * i], vel = parts[2 * i + 1];
  const float max_life = ps.life * (0.6f + 0.4f * (float)(pcg(i * 31u) % 1000u) / 1000.0f);
  const V3 hi = domain_max(g);
  if (ps.scatter != 0u || pos.w > max_life) spawn(g, ps, i, seed, pos, vel);
  const V3 p0 = v3(pos.x, pos.y, pos.z);
  const Sample s1 = sample_flow(g, p0);
  const V3 mid = add(p0, mul(mul(mul(s1.u, g.h), ps.dt), 0.5f));
  const Sample s2 = sample_flow(g, mid);
  V3 d = mul(mul(s2.u, g.h), ps.dt);
  const float dl = len3(d);
  if (dl > g.h * 2.0f) d = mul(d, g.h * 2.0f / dl);
  V3 np = add(p0, d);
  const bool dead = np.x > hi.x - g.h * 1.5f || np.y < 0.0f || np.y > hi.y || np.z > hi.z || s2.fluid < 0.05f;
  if (dead) {
    spawn(g, ps, i, seed, pos, vel);
    pos.w = 0.0f;
    parts[2 * i] = pos;
    parts[2 * i + 1] = vel;
    return;
  }
  if (np.z < 0.0f) np.z = -np.z;
  const Sample sv = sample_flow(g, np);
  parts[2 * i] = make_float4(np.x, np.y, np.z, pos.w + 1.0f);
  parts[2 * i + 1] = make_float4(d.x, d.y, d.z, wclamp(field_value(g, view, ps.colorMode, sv, np), 0.0f, 1.0f));
}

// seedOf (render-wgsl.ts:537-550)
__device__ V3 seed_of(const StreamArgs& st, uint32_t line) {
  if (st.seedMode == 1u) {
    const uint32_t ei = min(line / st.perEmitter, st.emitters - 1u);
    const uint32_t k = line % st.perEmitter;
    const float4 e = make_float4(st.emit[ei][0], st.emit[ei][1], st.emit[ei][2], st.emit[ei][3]);
    const float a = ((float)k + 0.5f) / (float)st.perEmitter * 6.2831853f + st.time * 0.6f;
    const float ring = 0.35f + 0.65f * (float)(k % 3u) / 2.0f;
    const V3 off = mul(mul(v3(0.0f, wtm::cosf(a), wtm::sinf(a)), e.w), ring);
    return add(v3(e.x, e.y, e.z), off);
  }
  const uint32_t row = line / st.cols, col = line % st.cols;
  const float fy = ((float)row + 0.5f) / (float)st.rows;
  const float fz = ((float)col + 0.5f) / (float)st.cols;
  return v3(st.smin[0], wmix(st.smin[1], st.smax[1], fy), wmix(st.smin[2], st.smax[2], fz));
}

// The velocity and fluid weight of sampleFlow (wgsl.ts:332-357) by one warp at one
// point.  Lane 4 k + c stands for corner k and, with c < 3, axis and component c: it
// holds coordinate c of the point (pa), reads component c of the corner's cell (c =
// 3: its density, which says whether the cell is fluid), and gets u_c.  The
// operations and their order per value are sample_flow's; the corners' products are
// formed side by side and summed in order.
__device__ __forceinline__ float sample_u_warp(const FieldGrid& g, float rh, bool fast_h, float pa, float& fluid) {
  const uint32_t lane = threadIdx.x, c = lane & 3u, quad = lane & 28u, k = lane >> 2;
  const bool one = c == 0 ? k & 1u : c == 1 ? k >> 1 & 1u : k >> 2 & 1u;  // the upper corner along axis c
  const float o = c == 0 ? g.ox : c == 1 ? g.oy : g.oz;
  const int n = (int)(c == 0 ? g.nx : c == 1 ? g.ny : g.nz);
  const uint32_t stride = c == 0 ? 1u : c == 1 ? g.nx : g.nx * g.ny;
  const float gg = div_known((c < 2 ? pa : fabsf(pa)) - o, g.h, rh, fast_h) - 0.5f;
  const int i0 = __float2int_rd(gg);  // saturating, NaN to 0
  const float f = gg - (float)i0;
  int q = i0 + (one ? 1 : 0);
  if (c >= 2) q ^= q >> 31;  // z: -q - 1 below the symmetry plane
  const uint32_t part = (uint32_t)min(max(q, 0), n - 1) * stride;
  const float wa = one ? f : 1.0f - f;
  const uint32_t id = __shfl_sync(0xffffffffu, part, quad) + __shfl_sync(0xffffffffu, part, quad + 1) +
                      __shfl_sync(0xffffffffu, part, quad + 2);
  const float val = __ldg(reinterpret_cast<const float*>(g.fields + id) + c);
  const float w = __shfl_sync(0xffffffffu, wa, quad) * __shfl_sync(0xffffffffu, wa, quad + 1) *
                  __shfl_sync(0xffffffffu, wa, quad + 2);
  const uint32_t wet = __ballot_sync(0xffffffffu, val > 0.0f);  // bits 4 k + 3
  const float term = c == 3 ? w : val * w;
  float acc = 0.0f;
#pragma unroll
  for (uint32_t j = 0; j < 8; j++) {
    const float t = __shfl_sync(0xffffffffu, term, 4 * j + c);
    if (wet >> (4 * j + 3) & 1u) acc = acc + t;
  }
  const float wsum = __shfl_sync(0xffffffffu, acc, 3);
  const bool dry = wsum < 1e-5f;
  const float ws = dry ? 1.0f : wsum;
  fluid = dry ? 0.0f : wsum;
  const float r = div_known(acc, ws, __frcp_rn(ws), div_range(ws));
  return dry ? 0.0f : c == 2 && pa < 0.0f ? -r : r;
}

// length(u) of a vector held in lanes 0-2, in every lane.
__device__ __forceinline__ float len3_warp(float ua) {
  const float q = ua * ua;
  return __fsqrt_rn(__shfl_sync(0xffffffffu, q, 0) + __shfl_sync(0xffffffffu, q, 1) + __shfl_sync(0xffffffffu, q, 2));
}
// A component of u / len (lanes c < 3; the others' quotients are not used).
__device__ __forceinline__ float unit_warp(float ua, float len) {
  const bool fast = div_range(len);
  return div_known(ua, len, __frcp_rn(fast ? len : 1.0f), fast);
}

// Streamline pass cs_main (render-wgsl.ts:551-575): one line per block of one
// warp.  A line is a chain of dependent RK2 steps, two field samples each, so its
// time is the chain's latency: the lanes share out each sample's corners and
// components, and the colours, which no step depends on, are left to the whole warp
// (a point per lane) once STREAM_CHUNK steps are done.  One lane doing all of it took
// 1.37 us a step; lines packed 32 to a warp gather from 32 places per load.
constexpr uint32_t STREAM_CHUNK = 128;

__global__ void __launch_bounds__(32) streamlines_kernel(FieldGrid g, StreamArgs st, ViewArgs view,
                                                        float4* __restrict__ pts) {
  __shared__ float rec[STREAM_CHUNK][3];  // the points of a chunk
  const uint32_t line = blockIdx.x, lane = threadIdx.x, c = lane & 3u;
  const uint32_t base = line * st.steps;
  const V3 seed = seed_of(st, line);
  float pa = c == 0 ? seed.x : c == 1 ? seed.y : seed.z;
  const V3 hi = v3(g.ox + (float)g.nx * g.h, g.oy + (float)g.ny * g.h, g.oz + (float)g.nz * g.h);
  const bool fast_h = div_range(g.h);
  const float rh = __frcp_rn(fast_h ? g.h : 1.0f);
  bool alive = true;
  uint32_t k = 0;
  while (alive && k < st.steps) {
    const uint32_t k0 = k, k1 = min(st.steps, k + STREAM_CHUNK);
    for (; k < k1; k++) {
      float fluid, fluid2;
      const float s1 = sample_u_warp(g, rh, fast_h, pa, fluid);
      const float len1 = len3_warp(s1);
      if (fluid < 0.3f || len1 < view.uIn * 0.03f) {
        alive = false;
        break;
      }
      if (lane < 3) rec[k - k0][lane] = pa;
      const float mid = pa + (unit_warp(s1, len1) * st.stepLen) * 0.5f;
      const float s2 = sample_u_warp(g, rh, fast_h, c == 3 ? pa : mid, fluid2);
      const float dir = fluid2 > 0.3f ? s2 : s1;
      const float step = unit_warp(dir, len3_warp(dir)) * st.stepLen;
      if (c < 3) pa = pa + step;
      // past the domain (lane c tests its coordinate)
      const bool out = c == 0 ? pa > hi.x - g.h * 3.0f : c == 1 ? pa < 0.01f || pa > hi.y : c == 2 && wabs(pa) > hi.z;
      if (__any_sync(0xffffffffu, out)) {
        alive = false;
        k++;
        break;
      }
    }
    __syncwarp();
    for (uint32_t i = k0 + lane; i < k; i += 32) {
      const V3 p = v3(rec[i - k0][0], rec[i - k0][1], rec[i - k0][2]);
      const Sample s = sample_flow(g, p);
      pts[base + i] = make_float4(p.x, p.y, p.z, wclamp(field_value(g, view, st.colorMode, s, p), 0.0f, 1.0f));
    }
    __syncwarp();
  }
  const float px = __shfl_sync(0xffffffffu, pa, 0), py = __shfl_sync(0xffffffffu, pa, 1), pz = __shfl_sync(0xffffffffu, pa, 2);
  for (uint32_t i = k + lane; i < st.steps; i += 32) pts[base + i] = make_float4(px, py, pz, -1.0f);
}

__global__ void sample_points_kernel(FieldGrid g, const float* __restrict__ pts, uint32_t n, float* __restrict__ out,
                                     float* __restrict__ vort) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const V3 p = v3(pts[3 * k], pts[3 * k + 1], pts[3 * k + 2]);
  const Sample s = sample_flow(g, p);
  out[6 * k + 0] = s.u.x; out[6 * k + 1] = s.u.y; out[6 * k + 2] = s.u.z;
  out[6 * k + 3] = s.rho; out[6 * k + 4] = s.temp; out[6 * k + 5] = s.fluid;
  if (vort) vort[k] = vorticity_at(g, p);
}

}  // namespace

cudaError_t launch_particles(const FieldGrid& g, const PSimArgs& ps, const ViewArgs& v, float4* parts, cudaStream_t s) {
  if (ps.count == 0) return cudaSuccess;
  particles_kernel<<<(ps.count + 127) / 128, 128, 0, s>>>(g, ps, v, parts);
  return cudaGetLastError();
}

cudaError_t launch_streamlines(const FieldGrid& g, const StreamArgs& st, const ViewArgs& v, float4* pts,
                               cudaStream_t s) {
  if (st.lines == 0) return cudaSuccess;
  streamlines_kernel<<<st.lines, 32, 0, s>>>(g, st, v, pts);
  return cudaGetLastError();
}

cudaError_t launch_sample_points(const FieldGrid& g, const float* pts, uint32_t n, float* out, float* vort,
                                 cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  sample_points_kernel<<<(n + 127) / 128, 128, 0, s>>>(g, pts, n, out, vort);
  return cudaGetLastError();
}

}  // namespace wt
