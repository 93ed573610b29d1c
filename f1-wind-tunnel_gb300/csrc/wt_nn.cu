// Element-wise and reduction operators of the warm-start network (include/wt_net.h):
// weight re-layout for the data gradient, 2x2x2 average pooling and nearest 2x
// upsampling with their gradients, skip additions, ReLU masking of gradients,
// bias gradients, the masked mean-square loss and the Adam update.  All are
// memory-bound one-pass kernels over channels-last tensors.
//
// Tensors whose addresses are 16-byte aligned and whose channels come in whole
// 16-byte chunks (or, element-wise, whatever their length) take kernels that move 16
// bytes per access and decode one voxel per chunk with 32-bit divisions; others take
// the element-wise kernels below them.  One element per thread with 64-bit
// divisions ran at 0.5-2.2 TB/s on the network's level-0 tensors (19-38 MB, in
// the L2).  Both do the same operations in the same order per element.
#include <cuda_bf16.h>
#include <stdint.h>

#include <mutex>
#include <string>

#include "wt_internal.h"
#include "wt_net.h"

namespace wt {
namespace {

constexpr uint32_t TB = 256;

inline uint32_t blocks_for(uint64_t n) {
  uint64_t b = (n + TB - 1) / TB;
  return (uint32_t)(b < 65535ull * 64 ? b : 65535ull * 64);
}

inline bool aligned16(const void* a, const void* b = nullptr, const void* c = nullptr, const void* d = nullptr) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
           reinterpret_cast<uintptr_t>(d)) & 15u) == 0;
}

// Eight bf16 of a 16-byte chunk.
struct Bf8 {
  uint4 v;
  __device__ __forceinline__ float get(int i) const {
    const uint32_t w = i < 2 ? v.x : i < 4 ? v.y : i < 6 ? v.z : v.w;
    return __uint_as_float((i & 1) ? (w & 0xffff0000u) : (w << 16));
  }
  __device__ __forceinline__ void set(const float (&f)[8]) {
    auto two = [](float lo, float hi) {
      return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(lo)) |
             ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(hi)) << 16);
    };
    v = make_uint4(two(f[0], f[1]), two(f[2], f[3]), two(f[4], f[5]), two(f[6], f[7]));
  }
};

// Chunk i of a coarse grid (d, h, w) with cc chunks per voxel: its fine-grid origin
// (the voxel's first child) in chunks.
struct Fine {
  uint32_t origin, row, plane;  // chunks; from one child row / plane to the next
};
__device__ __forceinline__ Fine fine_of(uint32_t i, uint32_t d, uint32_t h, uint32_t w, uint32_t cc) {
  const uint32_t vox = i / cc, k = i - vox * cc, q = vox / w, x = vox - q * w, r = q / h, y = q - r * h;
  // r = b d + z, and the fine plane of (b, z) is 2 r
  Fine f;
  f.row = 2 * w * cc;
  f.plane = 2 * h * f.row;
  f.origin = 2 * r * f.plane + 2 * y * f.row + 2 * x * cc + k;
  return f;
}
__device__ __forceinline__ uint32_t child(const Fine& f, uint32_t cc, int q) {
  return f.origin + (q >> 2) * f.plane + ((q >> 1) & 1) * f.row + (q & 1) * cc;
}

// y = mean of the 8 fine chunks (d, h, w coarse).
__global__ void pool2_fwd_vec_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, uint32_t n, uint32_t d, uint32_t h,
                                     uint32_t w, uint32_t cc) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Fine f = fine_of(i, d, h, w, cc);
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const Bf8 v{x[child(f, cc, q)]};
#pragma unroll
    for (int e = 0; e < 8; e++) s[e] += v.get(e);
  }
#pragma unroll
  for (int e = 0; e < 8; e++) s[e] *= 0.125f;
  Bf8 o;
  o.set(s);
  y[i] = o.v;
}
// 8 fine chunks = the coarse one (forward upsampling, 8 bf16), or an eighth of it (pooling's gradient, 4 floats).
template <bool SCALE>
__global__ void spread2_vec_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, uint32_t n, uint32_t d, uint32_t h,
                                   uint32_t w, uint32_t cc) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Fine f = fine_of(i, d, h, w, cc);
  uint4 v = x[i];
  if constexpr (SCALE)
    v = make_uint4(__float_as_uint(__uint_as_float(v.x) * 0.125f), __float_as_uint(__uint_as_float(v.y) * 0.125f),
                   __float_as_uint(__uint_as_float(v.z) * 0.125f), __float_as_uint(__uint_as_float(v.w) * 0.125f));
#pragma unroll
  for (int q = 0; q < 8; q++) y[child(f, cc, q)] = v;
}
// The coarse chunk (4 floats) = sum of its 8 fine ones.
__global__ void up2_bwd_vec_kernel(const float4* __restrict__ dy, float4* __restrict__ dx, uint32_t n, uint32_t d, uint32_t h,
                                   uint32_t w, uint32_t cc) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Fine f = fine_of(i, d, h, w, cc);
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const float4 v = dy[child(f, cc, q)];
    s.x += v.x;
    s.y += v.y;
    s.z += v.z;
    s.w += v.w;
  }
  dx[i] = s;
}

__global__ void weight_transpose_kernel(const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ wt,
                                        uint32_t cout, uint32_t taps, uint32_t cin) {
  const uint64_t n = (uint64_t)cout * taps * cin;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t ci = i % cin, t = (i / cin) % taps, co = (uint32_t)(i / ((uint64_t)cin * taps));
    wt[((uint64_t)ci * taps + t) * cout + co] = w[i];
  }
}

// y[b][z][y][x][c] = mean of the 8 fine cells x[b][2z+i][2y+j][2x+k][c] (d, h, w fine).
__global__ void pool2_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, uint32_t batch,
                                 uint32_t d, uint32_t h, uint32_t w, uint32_t c) {
  const uint32_t dc = d / 2, hc = h / 2, wc = w / 2;
  const uint64_t n = (uint64_t)batch * dc * hc * wc * c;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t ch = i % c;
    uint64_t v = i / c;
    const uint32_t xc = v % wc; v /= wc;
    const uint32_t yc = v % hc; v /= hc;
    const uint32_t zc = v % dc;
    const uint64_t b = v / dc;
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const uint64_t src = (((b * d + 2 * zc + (q >> 2)) * h + 2 * yc + ((q >> 1) & 1)) * w + 2 * xc + (q & 1)) * c + ch;
      s += __bfloat162float(x[src]);
    }
    y[i] = __float2bfloat16_rn(s * 0.125f);
  }
}

// dx[fine] = dy[parent] / 8 (d, h, w fine).
__global__ void pool2_bwd_kernel(const float* __restrict__ dy, float* __restrict__ dx, uint32_t batch, uint32_t d,
                                 uint32_t h, uint32_t w, uint32_t c) {
  const uint64_t n = (uint64_t)batch * d * h * w * c;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t ch = i % c;
    uint64_t v = i / c;
    const uint32_t xx = v % w; v /= w;
    const uint32_t yy = v % h; v /= h;
    const uint32_t zz = v % d;
    const uint64_t b = v / d;
    const uint64_t src = (((b * (d / 2) + zz / 2) * (h / 2) + yy / 2) * (w / 2) + xx / 2) * c + ch;
    dx[i] = dy[src] * 0.125f;
  }
}

// y[fine] = x[parent] (d, h, w coarse).
__global__ void up2_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, uint32_t batch,
                               uint32_t d, uint32_t h, uint32_t w, uint32_t c) {
  const uint32_t df = 2 * d, hf = 2 * h, wf = 2 * w;
  const uint64_t n = (uint64_t)batch * df * hf * wf * c;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t ch = i % c;
    uint64_t v = i / c;
    const uint32_t xx = v % wf; v /= wf;
    const uint32_t yy = v % hf; v /= hf;
    const uint32_t zz = v % df;
    const uint64_t b = v / df;
    y[i] = x[(((b * d + zz / 2) * h + yy / 2) * w + xx / 2) * c + ch];
  }
}

// dx[coarse] = sum of dy over its 8 fine children (d, h, w coarse).
__global__ void up2_bwd_kernel(const float* __restrict__ dy, float* __restrict__ dx, uint32_t batch, uint32_t d,
                               uint32_t h, uint32_t w, uint32_t c) {
  const uint64_t n = (uint64_t)batch * d * h * w * c;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t ch = i % c;
    uint64_t v = i / c;
    const uint32_t xc = v % w; v /= w;
    const uint32_t yc = v % h; v /= h;
    const uint32_t zc = v % d;
    const uint64_t b = v / d;
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const uint64_t src =
          (((b * 2 * d + 2 * zc + (q >> 2)) * 2 * h + 2 * yc + ((q >> 1) & 1)) * 2 * w + 2 * xc + (q & 1)) * c + ch;
      s += dy[src];
    }
    dx[i] = s;
  }
}

// Element-wise kernels over n values: nv chunks of 8 by 16-byte accesses (0 where an
// address is not aligned), the rest one by one.
__global__ void add_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                           __nv_bfloat16* __restrict__ y, uint64_t nv, uint64_t n) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < nv) {
    const Bf8 u{reinterpret_cast<const uint4*>(a)[i]}, v{reinterpret_cast<const uint4*>(b)[i]};
    float f[8];
#pragma unroll
    for (int e = 0; e < 8; e++) f[e] = u.get(e) + v.get(e);
    Bf8 o;
    o.set(f);
    reinterpret_cast<uint4*>(y)[i] = o.v;
  } else {
    for (uint64_t k = 8 * nv + (i - nv); k < n; k += (uint64_t)gridDim.x * blockDim.x - nv)
      y[k] = __float2bfloat16_rn(__bfloat162float(a[k]) + __bfloat162float(b[k]));
  }
}

__global__ void grad_to_bf16_kernel(const float* __restrict__ g, const float* __restrict__ g2,
                                    const __nv_bfloat16* __restrict__ act, __nv_bfloat16* __restrict__ out, uint64_t nv,
                                    uint64_t n) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < nv) {
    const float4 u0 = reinterpret_cast<const float4*>(g)[2 * i], u1 = reinterpret_cast<const float4*>(g)[2 * i + 1];
    float f[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    if (g2) {
      const float4 v0 = reinterpret_cast<const float4*>(g2)[2 * i], v1 = reinterpret_cast<const float4*>(g2)[2 * i + 1];
      const float q[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
      for (int e = 0; e < 8; e++) f[e] += q[e];
    }
    if (act) {
      const Bf8 m{reinterpret_cast<const uint4*>(act)[i]};
#pragma unroll
      for (int e = 0; e < 8; e++)
        if (!(m.get(e) > 0.0f)) f[e] = 0.0f;
    }
    Bf8 o;
    o.set(f);
    reinterpret_cast<uint4*>(out)[i] = o.v;
  } else {
    for (uint64_t k = 8 * nv + (i - nv); k < n; k += (uint64_t)gridDim.x * blockDim.x - nv) {
      float v = g[k];
      if (g2) v += g2[k];
      if (act && !(__bfloat162float(act[k]) > 0.0f)) v = 0.0f;
      out[k] = __float2bfloat16_rn(v);
    }
  }
}

// Bias gradient in two passes with a fixed summation order: block b of the first
// pass sums rows [b * chunk, (b + 1) * chunk) of every channel (each thread the rows
// of its phase, the phases folded in order) into partial[b][c]; the second pass sums
// the blocks in order, which is kept because a training run amplifies the last bit.  Eight
// channels a thread and 32 phases per channel in the second pass took 103 us of a batch-16
// step, this 175, one thread per channel over global memory 10 us a layer more.
constexpr uint32_t BG_BLOCKS = 512;

__global__ void bias_grad_partial_kernel(const __nv_bfloat16* __restrict__ dy, float* __restrict__ partial,
                                         uint64_t rows, uint32_t c, uint64_t chunk) {
  __shared__ float red[TB];
  const uint32_t phases = TB / c, ch = threadIdx.x % c, ph = threadIdx.x / c;
  const uint64_t r0 = (uint64_t)blockIdx.x * chunk, r1 = min(rows, r0 + chunk);
  float acc = 0.0f;
#pragma unroll 8
  for (uint64_t r = r0 + ph; r < r1; r += phases) acc += __bfloat162float(dy[r * c + ch]);
  red[threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.x < c) {
    float t = 0.0f;
    for (uint32_t q = 0; q < phases; q++) t += red[q * c + threadIdx.x];
    partial[(size_t)blockIdx.x * c + threadIdx.x] = t;
  }
}
// Eight channels to a block: the partial sums through shared memory, then in order (a thread
// walking them in global memory waits for each load).
__global__ void bias_grad_final_kernel(const float* __restrict__ partial, float* __restrict__ db, uint32_t nblocks,
                                       uint32_t c) {
  __shared__ float sh[BG_BLOCKS * 8];
  const uint32_t c0 = blockIdx.x * 8, n = min(8u, c - c0);
  for (uint32_t i = threadIdx.x; i < nblocks * 8; i += TB)
    if ((i & 7u) < n) sh[i] = partial[(size_t)(i >> 3) * c + c0 + (i & 7u)];
  __syncthreads();
  if (threadIdx.x < n) {
    float t = 0.0f;
#pragma unroll 8
    for (uint32_t b = 0; b < nblocks; b++) t += sh[8 * b + threadIdx.x];
    db[c0 + threadIdx.x] = t;
  }
}

// Per-block partial loss in double (fixed order), gradient written per element.
__global__ void mse_kernel(const __nv_bfloat16* __restrict__ pred, uint32_t cp, const float* __restrict__ target,
                           const float* __restrict__ mask, uint64_t rows, float inv_norm,
                           __nv_bfloat16* __restrict__ dpred, double* __restrict__ partial, bool vec) {
  __shared__ double red[TB];
  double acc = 0.0;
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < rows; r += (uint64_t)gridDim.x * blockDim.x) {
    const float mk = mask ? mask[r] : 1.0f;
    if (vec) {  // cp == 8, aligned: one chunk per row
      const Bf8 pv{reinterpret_cast<const uint4*>(pred)[r]};
      const float4 t4 = reinterpret_cast<const float4*>(target)[r];
      const float tv[4] = {t4.x, t4.y, t4.z, t4.w};
      float gk[8] = {};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float e = pv.get(k) - tv[k];
        acc += (double)(mk * e * e);
        gk[k] = 2.0f * mk * e * inv_norm;
      }
      Bf8 o;
      o.set(gk);
      reinterpret_cast<uint4*>(dpred)[r] = o.v;
      continue;
    }
    for (uint32_t k = 0; k < cp; k++) {
      float gk = 0.0f;
      if (k < 4) {
        const float e = __bfloat162float(pred[r * cp + k]) - target[r * 4 + k];
        acc += (double)(mk * e * e);
        gk = 2.0f * mk * e * inv_norm;
      }
      dpred[r * cp + k] = __float2bfloat16_rn(gk);
    }
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (uint32_t s = TB / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// *out += the n <= 1024 partial sums: each thread four of them in order, then a fixed tree.
__global__ void sum_partials_kernel(const double* __restrict__ partial, uint32_t n, double* __restrict__ out) {
  __shared__ double red[TB];
  double s = 0.0;
  for (uint32_t i = threadIdx.x; i < n; i += TB) s += partial[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (uint32_t k = TB / 2; k > 0; k >>= 1) {
    if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out += red[0];
}

__device__ __forceinline__ float adam_one(float p, float gi, float& m, float& v, float lr, float b1, float b2, float eps,
                                          float c1, float c2) {
  const float mi = b1 * m + (1.0f - b1) * gi;
  const float vi = b2 * v + (1.0f - b2) * gi * gi;
  m = mi;
  v = vi;
  const float upd = lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  return p - upd;
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, __nv_bfloat16* __restrict__ pb, uint64_t nv, uint64_t n, float lr,
                            float b1, float b2, float eps, float c1, float c2) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < nv) {  // four at a time
    float4 p4 = reinterpret_cast<float4*>(p)[i], m4 = reinterpret_cast<float4*>(m)[i], v4 = reinterpret_cast<float4*>(v)[i];
    const float4 g4 = reinterpret_cast<const float4*>(g)[i];
    p4.x = adam_one(p4.x, g4.x, m4.x, v4.x, lr, b1, b2, eps, c1, c2);
    p4.y = adam_one(p4.y, g4.y, m4.y, v4.y, lr, b1, b2, eps, c1, c2);
    p4.z = adam_one(p4.z, g4.z, m4.z, v4.z, lr, b1, b2, eps, c1, c2);
    p4.w = adam_one(p4.w, g4.w, m4.w, v4.w, lr, b1, b2, eps, c1, c2);
    reinterpret_cast<float4*>(p)[i] = p4;
    reinterpret_cast<float4*>(m)[i] = m4;
    reinterpret_cast<float4*>(v)[i] = v4;
    if (pb) {
      __nv_bfloat162 lo = __floats2bfloat162_rn(p4.x, p4.y), hi = __floats2bfloat162_rn(p4.z, p4.w);
      uint2 o;
      memcpy(&o.x, &lo, 4);
      memcpy(&o.y, &hi, 4);
      reinterpret_cast<uint2*>(pb)[i] = o;
    }
  } else {
    for (uint64_t k = 4 * nv + (i - nv); k < n; k += (uint64_t)gridDim.x * blockDim.x - nv) {
      const float pi = adam_one(p[k], g[k], m[k], v[k], lr, b1, b2, eps, c1, c2);
      p[k] = pi;
      if (pb) pb[k] = __float2bfloat16_rn(pi);
    }
  }
}

__global__ void to_bf16_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, uint64_t n) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16_rn(x[i]);
}

int done(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    net_error() = std::string(what) + ": " + cudaGetErrorString(e);
    return WT_ERR_CUDA;
  }
  return WT_OK;
}

int bad(const char* what) {
  net_error() = std::string(what) + ": invalid argument";
  return WT_ERR_ARG;
}

// Threads for nv chunks of `per` values and the values past them (at least one thread more than chunks).
inline uint32_t blocks_chunks(uint64_t nv, uint64_t n, uint64_t per) { return blocks_for(nv + (n - per * nv) + 1); }
// Chunks of `per` values of an element-wise call; 0 where they would not all be covered by one grid.
inline uint64_t chunks(uint64_t n, uint64_t per, bool aligned) {
  const uint64_t nv = aligned ? n / per : 0;
  return nv < (uint64_t)TB * 65535ull * 63 ? nv : 0;
}
// Whether a pooling or upsampling call takes 16-byte chunks: coarse chunks n and all fine ones below 2^31.
inline bool grid_chunks(uint64_t n, uint32_t c, uint32_t per, const void* a, const void* b) {
  return c % per == 0 && aligned16(a, b) && 8 * n < (1ull << 31);
}

inline cudaStream_t S(void* s) { return static_cast<cudaStream_t>(s); }
typedef __nv_bfloat16 bf;

// Where a call's partial sums lie between its two launches.  Each stream has a buffer of
// its own (by the stream's id, which the process never gives out again), used in
// stream order; the lock is held while both launches are enqueued, so that calls of
// several threads on one stream do not interleave.  Streams past the first
// SCRATCH_STREAMS, and calls under capture, whose graph may be replayed beside the
// stream, take stream-ordered memory for the call (which everywhere would cost 13 us a
// call: a batch-16 training step 2720 -> 2930 us).  The buffers, 8 MB at most, stay to the
// end of the process.
constexpr size_t SCRATCH_STREAMS = 16, SCRATCH_BYTES = (size_t)BG_BLOCKS * TB * sizeof(float);

class Scratch {
 public:
  Scratch(size_t bytes, cudaStream_t s) : lock_(mutex()), stream_(s) {
    struct Entry {
      int dev;
      unsigned long long id;
      void* p;
    };
    static Entry entries[SCRATCH_STREAMS];
    static size_t count = 0;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    Entry e = {};
    if (cudaStreamIsCapturing(s, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone && bytes <= SCRATCH_BYTES &&
        cudaGetDevice(&e.dev) == cudaSuccess && cudaStreamGetId(s, &e.id) == cudaSuccess) {
      for (size_t k = 0; k < count; k++)
        if (entries[k].dev == e.dev && entries[k].id == e.id) p_ = entries[k].p;
      if (!p_ && count < SCRATCH_STREAMS && cudaMallocAsync(&e.p, SCRATCH_BYTES, s) == cudaSuccess) {
        entries[count++] = e;
        p_ = e.p;
      }
    }
    if (p_) return;
    own_ = cudaMallocAsync(&p_, bytes, s) == cudaSuccess;
    if (!own_) p_ = nullptr;
  }
  ~Scratch() {
    if (own_) cudaFreeAsync(p_, stream_);
  }
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  template <class T> T* as() const { return static_cast<T*>(p_); }

 private:
  static std::mutex& mutex() {
    static std::mutex m;
    return m;
  }
  std::lock_guard<std::mutex> lock_;
  void* p_ = nullptr;
  bool own_ = false;
  cudaStream_t stream_;
};

}  // namespace
}  // namespace wt

using namespace wt;

extern "C" {

int wt_nn_weight_transpose(const void* w, void* wt, uint32_t cout, uint32_t taps, uint32_t cin, void* stream) {
  if (!w || !wt || !cout || !taps || !cin) return bad("wt_nn_weight_transpose");
  const uint64_t n = (uint64_t)cout * taps * cin;
  weight_transpose_kernel<<<blocks_for(n), TB, 0, S(stream)>>>(static_cast<const bf*>(w), static_cast<bf*>(wt), cout,
                                                                taps, cin);
  return done("wt_nn_weight_transpose");
}

int wt_nn_pool2_forward(const void* x, void* y, uint32_t batch, uint32_t d, uint32_t h, uint32_t w, uint32_t c,
                        void* stream) {
  if (!x || !y || !c || (d | h | w) & 1u || !d || !h || !w) return bad("wt_nn_pool2_forward");
  const uint64_t n = (uint64_t)batch * (d / 2) * (h / 2) * (w / 2) * c;
  if (n && grid_chunks(n / 8, c, 8, x, y)) {
    pool2_fwd_vec_kernel<<<blocks_for(n / 8), TB, 0, S(stream)>>>(static_cast<const uint4*>(x), static_cast<uint4*>(y),
                                                                  (uint32_t)(n / 8), d / 2, h / 2, w / 2, c / 8);
    return done("wt_nn_pool2_forward");
  }
  pool2_fwd_kernel<<<blocks_for(n), TB, 0, S(stream)>>>(static_cast<const bf*>(x), static_cast<bf*>(y), batch, d, h,
                                                         w, c);
  return done("wt_nn_pool2_forward");
}

int wt_nn_pool2_backward(const float* dy, float* dx, uint32_t batch, uint32_t d, uint32_t h, uint32_t w, uint32_t c,
                         void* stream) {
  if (!dy || !dx || !c || (d | h | w) & 1u || !d || !h || !w) return bad("wt_nn_pool2_backward");
  const uint64_t n = (uint64_t)batch * d * h * w * c;
  if (n && grid_chunks(n / 32, c, 4, dy, dx)) {
    spread2_vec_kernel<true><<<blocks_for(n / 32), TB, 0, S(stream)>>>(reinterpret_cast<const uint4*>(dy), reinterpret_cast<uint4*>(dx),
                                                                       (uint32_t)(n / 32), d / 2, h / 2, w / 2, c / 4);
    return done("wt_nn_pool2_backward");
  }
  pool2_bwd_kernel<<<blocks_for(n), TB, 0, S(stream)>>>(dy, dx, batch, d, h, w, c);
  return done("wt_nn_pool2_backward");
}

int wt_nn_up2_forward(const void* x, void* y, uint32_t batch, uint32_t d, uint32_t h, uint32_t w, uint32_t c,
                      void* stream) {
  if (!x || !y || !c || !d || !h || !w) return bad("wt_nn_up2_forward");
  const uint64_t n = (uint64_t)batch * 8 * d * h * w * c;
  if (n && grid_chunks(n / 64, c, 8, x, y)) {
    spread2_vec_kernel<false><<<blocks_for(n / 64), TB, 0, S(stream)>>>(static_cast<const uint4*>(x), static_cast<uint4*>(y),
                                                                        (uint32_t)(n / 64), d, h, w, c / 8);
    return done("wt_nn_up2_forward");
  }
  up2_fwd_kernel<<<blocks_for(n), TB, 0, S(stream)>>>(static_cast<const bf*>(x), static_cast<bf*>(y), batch, d, h, w,
                                                       c);
  return done("wt_nn_up2_forward");
}

int wt_nn_up2_backward(const float* dy, float* dx, uint32_t batch, uint32_t d, uint32_t h, uint32_t w, uint32_t c,
                       void* stream) {
  if (!dy || !dx || !c || !d || !h || !w) return bad("wt_nn_up2_backward");
  const uint64_t n = (uint64_t)batch * d * h * w * c;
  if (n && grid_chunks(n / 4, c, 4, dy, dx)) {
    up2_bwd_vec_kernel<<<blocks_for(n / 4), TB, 0, S(stream)>>>(reinterpret_cast<const float4*>(dy), reinterpret_cast<float4*>(dx),
                                                                (uint32_t)(n / 4), d, h, w, c / 4);
    return done("wt_nn_up2_backward");
  }
  up2_bwd_kernel<<<blocks_for(n), TB, 0, S(stream)>>>(dy, dx, batch, d, h, w, c);
  return done("wt_nn_up2_backward");
}

int wt_nn_add(const void* a, const void* b, void* y, uint64_t n, void* stream) {
  if (!a || !b || !y) return bad("wt_nn_add");
  if (n == 0) return WT_OK;
  const uint64_t nv = chunks(n, 8, aligned16(a, b, y));
  add_kernel<<<blocks_chunks(nv, n, 8), TB, 0, S(stream)>>>(static_cast<const bf*>(a), static_cast<const bf*>(b),
                                                             static_cast<bf*>(y), nv, n);
  return done("wt_nn_add");
}

int wt_nn_grad_to_bf16(const float* g, const float* g2, const void* act, void* out, uint64_t n, void* stream) {
  if (!g || !out) return bad("wt_nn_grad_to_bf16");
  if (n == 0) return WT_OK;
  const uint64_t nv = chunks(n, 8, aligned16(g, g2, act, out));
  grad_to_bf16_kernel<<<blocks_chunks(nv, n, 8), TB, 0, S(stream)>>>(g, g2, static_cast<const bf*>(act), static_cast<bf*>(out),
                                                                     nv, n);
  return done("wt_nn_grad_to_bf16");
}

int wt_nn_bias_grad(const void* dy, float* db, uint64_t rows, uint32_t c, void* stream) {
  if (!dy || !db || !c || c > TB || TB % c) return bad("wt_nn_bias_grad");
  const uint64_t chunk = rows ? (rows + BG_BLOCKS - 1) / BG_BLOCKS : 1;
  const uint32_t nb = (uint32_t)(rows ? (rows + chunk - 1) / chunk : 1);
  const Scratch scratch((size_t)nb * c * sizeof(float), S(stream));
  float* const partial = scratch.as<float>();
  if (!partial) return bad("wt_nn_bias_grad scratch");
  bias_grad_partial_kernel<<<nb, TB, 0, S(stream)>>>(static_cast<const bf*>(dy), partial, rows, c, chunk);
  bias_grad_final_kernel<<<(c + 7) / 8, TB, 0, S(stream)>>>(partial, db, nb, c);
  return done("wt_nn_bias_grad");
}

int wt_nn_mse(const void* pred, uint32_t cp, const float* target, const float* mask, uint64_t rows, float norm,
              void* dpred, double* loss_sum, void* stream) {
  if (!pred || !target || !dpred || !loss_sum || cp < 4 || !(norm > 0.0f)) return bad("wt_nn_mse");
  const uint32_t nb = (uint32_t)((rows + TB - 1) / TB < 1024 ? (rows + TB - 1) / TB : 1024);
  const uint32_t grid = nb ? nb : 1;
  const Scratch scratch(grid * sizeof(double), S(stream));
  double* const partial = scratch.as<double>();
  if (!partial) return bad("wt_nn_mse scratch");
  mse_kernel<<<grid, TB, 0, S(stream)>>>(static_cast<const bf*>(pred), cp, target, mask, rows, 1.0f / norm,
                                         static_cast<bf*>(dpred), partial, cp == 8 && aligned16(pred, target, dpred));
  sum_partials_kernel<<<1, TB, 0, S(stream)>>>(partial, grid, loss_sum);
  return done("wt_nn_mse");
}

int wt_nn_adam(float* param, const float* grad, float* m, float* v, void* param_bf16, uint64_t n, float lr,
               float beta1, float beta2, float eps, uint32_t step, void* stream) {
  if (!param || !grad || !m || !v || step == 0) return bad("wt_nn_adam");
  if (n == 0) return WT_OK;
  const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
  const uint64_t nv = chunks(n, 4, aligned16(param, grad, m, v) && (reinterpret_cast<uintptr_t>(param_bf16) & 7u) == 0);
  adam_kernel<<<blocks_chunks(nv, n, 4), TB, 0, S(stream)>>>(param, grad, m, v, static_cast<bf*>(param_bf16), nv, n, lr, beta1,
                                                             beta2, eps, c1, c2);
  return done("wt_nn_adam");
}

int wt_nn_to_bf16(const float* x, void* y, uint64_t n, void* stream) {
  if (!x || !y) return bad("wt_nn_to_bf16");
  if (n == 0) return WT_OK;
  to_bf16_kernel<<<blocks_for(n), TB, 0, S(stream)>>>(x, static_cast<bf*>(y), n);
  return done("wt_nn_to_bf16");
}

}  // extern "C"
