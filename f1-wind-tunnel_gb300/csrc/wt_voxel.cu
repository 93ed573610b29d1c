// Voxelizer (VOXELIZE, src/engine/wgsl.ts:294-321) and the cell words the
// step kernels read.
//
// The signed-distance scenes are the reference's analytic ones
// (src/engine/wgsl.ts:20-76,101-116 primitives and scene switch;
// src/engine/f1.ts:20-320 generic F1, :397-407 heat emission).  Solid flags
// are a threshold test on the distance at the cell centre, so every float
// operation is kept in the reference's order and this unit is built with
// -fmad=false: flags and emission match the CPU model bit for bit.  sin, cos
// and atan are the project's functions (wt_fmath.h); shape-wide values (rake
// rotation, rear main-plane direction) are computed once on the host with the
// same functions, which gives the same bits as evaluating them per cell.
//
// The cell-word pass stages a tile of solid flags (with a 2-cell halo in x for
// the belt test and 1 in y and z) in shared memory; coordinates are clamped to
// the lattice when loading, which makes the z = -1 halo the z = 0 mirror image
// the reference reads through its symmetry plane (wgsl.ts:218).
#include "wt_internal.h"
#include "wt_lattice.cuh"
#include "wt_scene.cuh"

namespace wt {
namespace {

__global__ void voxelize_kernel(const __grid_constant__ SceneParam P, uint32_t nx, uint32_t ny, uint32_t nz, float ox, float oy, float oz, float h,
                                uint8_t* __restrict__ solid, float* __restrict__ emit) {
  const Scene& S = P.s;
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
  const uint32_t z = blockIdx.z;
  if (x >= nx || y >= ny) return;
  const uint32_t idx = x + nx * (y + ny * z);
  const V3 p = v3(ox + ((float)x + 0.5f) * h, oy + ((float)y + 0.5f) * h, oz + ((float)z + 0.5f) * h);
  V2 r = scene_sdf(S, P.f1, p);
  const bool w17 = S.s.kind == WT_KIND_W17 && S.car.body != nullptr;
  // the W17's cooling ducts are carved out of its body (wgsl.ts:313) and marked
  // with emission -1 (wgsl.ts:319-320): the step relaxes the air there
  const float duct = w17 ? w17_duct(S, p) : 1e3f;
  if (w17 && ab(r.y - 12.0f) < 0.5f) r.x = mx(r.x, -duct);
  const bool inside = r.x < (w17 ? 0.45f : 0.3f) * h && x > 1u && x < nx - 2u;
  uint32_t group = 1u;
  if (ab(r.y - 7.0f) < 0.5f) group = 2u;
  if (ab(r.y - 8.0f) < 0.5f) group = 3u;
  solid[idx] = inside ? (uint8_t)group : (uint8_t)0;
  const float em = S.s.kind == WT_KIND_F1 ? f1_emission(S, p) : (w17 ? w17_emission(S, p) : 0.0f);
  emit[idx] = inside ? em : (w17 && duct < 0.0f ? -1.0f : 0.0f);
}

// ---------------------------------------------------------------- cell words
constexpr int TX = 32, TY = 4, TZ = 2;
constexpr int HX = 2, HY = 1, HZ = 1;
constexpr int SX = TX + 2 * HX, SY = TY + 2 * HY, SZ = TZ + 2 * HZ;

__global__ void cell_words_kernel(const uint8_t* __restrict__ solid, const float* __restrict__ emit,
                                  uint32_t* __restrict__ cellw, uint32_t nx, uint32_t ny, uint32_t nz) {
  __shared__ uint8_t tile[SZ][SY][SX];
  const int x0 = blockIdx.x * TX - HX, y0 = blockIdx.y * TY - HY, z0 = blockIdx.z * TZ - HZ;
  const int tid = threadIdx.x + TX * (threadIdx.y + TY * threadIdx.z);
  for (int k = tid; k < SX * SY * SZ; k += TX * TY * TZ) {
    const int lx = k % SX, ly = (k / SX) % SY, lz = k / (SX * SY);
    const int gx = min(max(x0 + lx, 0), (int)nx - 1);
    const int gy = min(max(y0 + ly, 0), (int)ny - 1);
    const int gz = min(max(z0 + lz, 0), (int)nz - 1);
    tile[lz][ly][lx] = solid[(uint32_t)gx + nx * ((uint32_t)gy + ny * (uint32_t)gz)];
  }
  __syncthreads();
  const uint32_t x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y, z = blockIdx.z * TZ + threadIdx.z;
  if (x >= nx || y >= ny || z >= nz) return;
  const uint32_t idx = x + nx * (y + ny * z);
  const int lx = threadIdx.x + HX, ly = threadIdx.y + HY, lz = threadIdx.z + HZ;
  if (tile[lz][ly][lx]) {
    cellw[idx] = CW_SOLID;
    return;
  }
  uint32_t w = 0u;
  const bool duct = emit[idx] < 0.0f;
  bool force = false;
  uint32_t groups = 0u;  // bit g: a non-mirrored link off group g
  sfor<19>([&](auto I) {
    constexpr int i = I;
    if constexpr (i != 0) {
      constexpr int cx = CXd(i), cy = CYd(i), cz = CZd(i);
      const int sx = (int)x - cx, sy = (int)y - cy, sz = (int)z - cz;
      // precedence of wgsl.ts:207-221: inlet, outlet, floor, far field come first
      if (sx < 0 || sx >= (int)nx || sy < 0 || sy >= (int)ny || sz >= (int)nz) return;
      const uint32_t g = tile[lz - cz][ly - cy][lx - cx];
      if (g) {  // z = -1 reads the clamped (mirrored) z = 0 flag
        w |= 1u << i;
        if (!(sz < 0)) {
          force = true;
          groups |= 1u << g;
        }
      }
    }
  });
  if (y == 0u) {  // belt contact patch (wgsl.ts:192-197)
    if (tile[lz][ly][lx - 2] || tile[lz][ly][lx + 2] || tile[lz][ly + 1][lx] || tile[lz - 1][ly][lx] ||
        tile[lz + 1][ly][lx])
      w |= CW_BELT;
  }
  if (duct) w |= CW_DUCT;
  if (force && !duct) w |= CW_FORCE;
  if (groups == 2u || groups == 4u || groups == 8u) w |= (groups == 2u ? 1u : groups == 4u ? 2u : 3u) << CW_GROUP_SHIFT;
  cellw[idx] = w;
}

// Per step-kernel block: whether it carries a force link, and the cells of each
// solid group (0 fluid) added to counts[0..3].
__global__ void block_flags_kernel(const uint32_t* __restrict__ cellw, const uint8_t* __restrict__ solid, uint32_t nx,
                                   uint32_t ny, int32_t* __restrict__ flags, uint32_t* __restrict__ counts) {
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
  const uint32_t z = blockIdx.z;
  const bool in = x < nx && y < ny;
  const uint32_t idx = in ? x + nx * (y + ny * z) : 0u;
  const bool f = in && (cellw[idx] & CW_FORCE) != 0u;
  const uint32_t v = in ? solid[idx] : 0u, g = v ? (v - 1u) % 3u + 1u : 0u;
  const uint32_t lane = (threadIdx.x + blockDim.x * threadIdx.y) & 31u;
#pragma unroll
  for (uint32_t k = 1; k < 4; k++) {  // few warps hold solid cells; the fluid count follows from the others
    const unsigned m = __ballot_sync(0xffffffffu, g == k);
    if (m && lane == 0) atomicAdd(counts + k, (unsigned)__popc(m));
  }
  const int any = __syncthreads_or(f);
  if (threadIdx.x == 0 && threadIdx.y == 0)
    flags[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = any ? 1 : 0;
}

// In place: flags[b] becomes the block's slot (the number of flagged blocks before
// it), or -1; counts[0] their number.  One block, each thread a run of blocks.
__global__ void __launch_bounds__(1024) block_slots_kernel(int32_t* __restrict__ flags, uint32_t nblocks,
                                                           uint32_t* __restrict__ counts) {
  __shared__ uint32_t warp_sum[32];
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const uint32_t per = (nblocks + 1023u) / 1024u, b0 = min(t * per, nblocks), b1 = min(b0 + per, nblocks);
  uint32_t n = 0;
#pragma unroll 8
  for (uint32_t b = b0; b < b1; b++) n += (uint32_t)flags[b];
  uint32_t inc = n;  // inclusive sums over the warp, then the warps
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= (uint32_t)d) inc += v;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t v = warp_sum[lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, v, d);
      if (lane >= (uint32_t)d) v += u;
    }
    warp_sum[lane] = v;
  }
  __syncthreads();
  uint32_t slot = inc - n + (warp ? warp_sum[warp - 1] : 0u);
#pragma unroll 8
  for (uint32_t b = b0; b < b1; b++) {
    const int32_t f = flags[b];
    flags[b] = f ? (int32_t)slot : -1;
    slot += (uint32_t)f;
  }
  if (t == 1023) counts[0] = slot;
}

__global__ void links_out_kernel(const uint32_t* __restrict__ cellw, uint32_t* __restrict__ links, uint64_t n) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const uint32_t w = cellw[i];
    links[i] = (w & CW_SOLID) ? 0u : (w & (CW_LINKS | CW_BELT));
  }
}
__global__ void solid_u32_kernel(const uint8_t* __restrict__ s, uint32_t* __restrict__ out, uint64_t n) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = s[i];
}
__global__ void solid_from_u32_kernel(const uint32_t* __restrict__ in, uint8_t* __restrict__ s, uint64_t n) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) s[i] = (uint8_t)(in[i] > 3u ? 3u : in[i]);
}

}  // namespace

// Scene distance at the cell centres of `grid` (the first component of sceneSdf).
__global__ void sdf_sample_kernel(const __grid_constant__ SceneParam P, uint32_t nx, uint32_t ny, uint32_t nz, float ox, float oy, float oz,
                                  float h, float* __restrict__ out) {
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
  const uint32_t z = blockIdx.z;
  if (x >= nx || y >= ny) return;
  const V3 p = v3(ox + ((float)x + 0.5f) * h, oy + ((float)y + 0.5f) * h, oz + ((float)z + 0.5f) * h);
  out[x + nx * (y + ny * z)] = scene_sdf(P.s, P.f1, p).x;
}


cudaError_t launch_sdf_sample(const wt_shape& shape, const wt_grid& grid, float* out, cudaStream_t s) {
  const SceneParam S = make_scene(shape);
  const dim3 block(32, 4, 1);
  const dim3 g((grid.nx + 31) / 32, (grid.ny + 3) / 4, grid.nz);
  sdf_sample_kernel<<<g, block, 0, s>>>(S, grid.nx, grid.ny, grid.nz, grid.origin[0], grid.origin[1], grid.origin[2],
                                        grid.h, out);
  return cudaGetLastError();
}

cudaError_t launch_voxelize(const wt_shape& shape, const CarView& car, const wt_grid& grid, uint8_t* solid, float* emit,
                            cudaStream_t s) {
  const SceneParam S = make_scene(shape, car);
  const dim3 block(32, 4, 1);
  const dim3 g((grid.nx + 31) / 32, (grid.ny + 3) / 4, grid.nz);
  voxelize_kernel<<<g, block, 0, s>>>(S, grid.nx, grid.ny, grid.nz, grid.origin[0], grid.origin[1], grid.origin[2],
                                      grid.h, solid, emit);
  return cudaGetLastError();
}

cudaError_t launch_cell_words(const uint8_t* solid, const float* emit, uint32_t* cellw, uint32_t nx, uint32_t ny,
                              uint32_t nz, cudaStream_t s) {
  const dim3 block(TX, TY, TZ);
  const dim3 g((nx + TX - 1) / TX, (ny + TY - 1) / TY, (nz + TZ - 1) / TZ);
  cell_words_kernel<<<g, block, 0, s>>>(solid, emit, cellw, nx, ny, nz);
  return cudaGetLastError();
}

cudaError_t launch_block_slots(const uint32_t* cellw, const uint8_t* solid, const StepGeom& g, uint32_t nx, uint32_t ny,
                               int32_t* slots, uint32_t* counts, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(counts, 0, 4 * sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  block_flags_kernel<<<g.grid, g.block, 0, s>>>(cellw, solid, nx, ny, slots, counts);
  block_slots_kernel<<<1, 1024, 0, s>>>(slots, g.nblocks, counts);
  return cudaGetLastError();
}

__global__ void put_reduce_args_kernel(ReduceArgs* dst, ReduceArgs a) { *dst = a; }
cudaError_t launch_put_reduce_args(ReduceArgs* dst, const ReduceArgs& a, cudaStream_t s) {
  put_reduce_args_kernel<<<1, 1, 0, s>>>(dst, a);
  return cudaGetLastError();
}

cudaError_t launch_links_out(const uint32_t* cellw, uint32_t* links, uint64_t n, cudaStream_t s) {
  links_out_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(cellw, links, n);
  return cudaGetLastError();
}
cudaError_t launch_solid_u32(const uint8_t* solid, uint32_t* out, uint64_t n, cudaStream_t s) {
  solid_u32_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(solid, out, n);
  return cudaGetLastError();
}
cudaError_t launch_solid_from_u32(const uint32_t* in, uint8_t* solid, uint64_t n, cudaStream_t s) {
  solid_from_u32_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(in, solid, n);
  return cudaGetLastError();
}

}  // namespace wt
