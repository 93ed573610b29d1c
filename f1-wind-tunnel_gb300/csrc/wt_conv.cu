// 3-D convolution of the warm-start network as an implicit GEMM on the
// 5th-generation tensor cores (tcgen05, kind::f16 with BF16 operands, FP32
// accumulation in tensor memory).
//
//   FWD    D[m][co]        = sum_k A[m][k] B[co][k],  A[m][(t,ci)]  = x[m + off(t)][ci],  B = w[co][(t,ci)]
//   DGRAD  D[m][ci]        = sum_k A[m][k] B[ci][k],  A[m][(t,co)]  = dy[m - off(t)][co], B = wt[ci][(t,co)]
//   WGRAD  D[(t,ci)][co]   = sum_m A[(t,ci)][m] B[co][m], A = x[m + off(t)][ci], B = dy[m][co]
// (m a voxel of the batch's grid, out-of-grid neighbours read as zero).
//
// FWD and DGRAD (conv_rows_kernel): a block holds one input tile with its halo in
// shared memory and runs all 27 taps on it; a tap is a shift of the matrix
// descriptor's start address, so every input value is fetched once per tile
// instead of once per tap.  WGRAD (conv_wgrad_kernel) does the same with voxels as K.
// Grids too narrow for such tiles are gathered voxel by voxel (conv_gather_kernel).
// The accumulators live in tensor memory; the epilogues read them with
// tcgen05.ld (warp w owns lanes 32w..32w+31).  Every mbarrier wait is bounded:
// on expiry the kernel raises g_conv_error, still waits (bounded) for its own
// MMAs, frees its tensor memory and returns.
#include <atomic>
#include <cuda_bf16.h>
#include <stdint.h>

#include <string>

#include "wt_conv_plan.h"
#include "wt_internal.h"
#include "wt_net.h"

namespace wt {

__device__ int g_conv_error;

std::string& net_error() {
  thread_local std::string e;
  return e;
}

namespace {

constexpr uint32_t BM = 128;
constexpr uint32_t WAIT_LIMIT = 1u << 21;

enum Mode { FWD = 0, DGRAD = 1, WGRAD = 2 };

// Poll budget of the pipeline's stage waits for the next launches (see
// wt_net_set_stage_wait_limit); the drain before tensor memory is freed always
// uses WAIT_LIMIT.
std::atomic<uint32_t> g_stage_wait{WAIT_LIMIT};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptors (tcgen05) are start address (bits 0-13), leading and
// stride byte offsets (16-29, 32-45), all >> 4; bits 46-47 = 1 (the descriptor version of this
// architecture); no swizzle, base offset 0.

// Instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A and B BF16
// (bits 7-9 = 1, 10-12 = 1), both K-major (bits 15, 16 = 0) or both M/N-major (1),
// N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t m, uint32_t n, uint32_t mn_major = 0) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (mn_major * 3u << 15) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ int tap_dz(uint32_t t, uint32_t taps) { return taps == 27 ? (int)(t / 9) - 1 : 0; }
__device__ __forceinline__ int tap_dy(uint32_t t, uint32_t taps) { return taps == 27 ? (int)((t / 3) % 3) - 1 : 0; }
__device__ __forceinline__ int tap_dx(uint32_t t, uint32_t taps) { return taps == 27 ? (int)(t % 3) - 1 : 0; }

// ---------------------------------------------------------------------------
// FWD / DGRAD: the input tile with its halo stays in shared memory for all taps.
//
// Rows.  The grid's (batch item, z, y) rows are numbered in one sequence with a
// zero row after each plane and a zero plane after each batch item, so that a
// tap's dz and dy are one fixed distance in that numbering and out-of-grid
// neighbours fall on zeros.  A block computes 16 such rows by 8 XG voxels along x:
// XG matrix tiles of M = 128 (16 rows x 8 voxels), N = nt output channels each.
// Shared memory holds, per group of 8 input channels (a plane), nrows x W voxels
// of 16 bytes: 8 voxels along x are one core matrix (128 B contiguous), the 16
// rows of a tile are the M groups (stride = row pitch), the planes the K groups.
// A tap only moves the descriptor's start address (by 16 B along x, by rows along
// y and z).  The rows a tile needs are either one run (short planes) or three
// bands, one per dz.
//
// Measured, the network's 12 distinct layers at batch 16 / 1 (us in all): forward
// 1675 -> 395 / 782 -> 144 (launch-bound), data gradient 1530 -> 394, against the
// gather of 27 x the input per tile; the deepest chain (K = 3456, 72 voxels) 166 ->
// 17.  What bounds it now: an MMA of M 128 with N 16 takes 39 cycles (64 with N
// 128), so the narrow layers use a few per cent of the tensor pipe, and the halo
// (3.4 x the input at 24 x 24 planes).
//
// K order is the gather's: taps in order, channels in order, 16 per MMA, so the
// sums have the same bits whatever the tiling.  A channel count of 8 puts two taps
// in one MMA (FWD); other odd plane counts, and DGRAD with 8, pair their last plane
// with a plane of zeros.  Weights come in stages of `ups` MMAs of K through a ring of
// D stages (cp.async).
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16u : 0u) : "memory");
}
// Voxel index of x position 0 of numbered row R, or -1 for a zero row.
__device__ __forceinline__ int32_t row_voxel(const RowArgs& p, int64_t R) {
  if (R < 0 || R >= (int64_t)p.rows) return -1;
  const uint32_t r = (uint32_t)R, q = r / p.hp, y = r - q * p.hp, b = q / p.dp, z = q - b * p.dp;
  if (y >= p.h || z >= p.d) return -1;
  return (int32_t)(((b * p.d + z) * p.h + y) * p.w);  // fewer than 2^31 voxels (+ a row's padding: checked on the host)
}

// Threads: eight warps load (and later run the epilogue), a ninth issues the MMAs.
// Stage st of the weights goes to ring slot st % depth once the MMAs of stage
// st - depth are done (done[slot], committed by the issuing lane); full[slot]
// completes when its copies have landed, and the issuing warp makes them visible to
// the tensor cores.  At most two stages of MMAs are in flight.

// mbar_wait that also ends when the block has been told to stop.
__device__ __forceinline__ bool mbar_wait_or(uint32_t bar, uint32_t parity, const volatile uint32_t* stop, uint32_t limit = WAIT_LIMIT) {
  if (limit && mbar_wait(bar, parity, 1)) return true;
  for (uint32_t i = 0; i < limit && !*stop; i += 16)
    if (mbar_wait(bar, parity, 16)) return true;
  return false;
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}

template <int MODE, int XG>
__global__ void __launch_bounds__(ROW_THREADS) conv_rows_kernel(RowArgs p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  // barriers, the tensor-memory slot and the stop flag; the voxel of each tile row;
  // the MMAs' input descriptors (low words) and weight columns; the input planes;
  // the weight ring
  uint64_t* const full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* const done = full + ROW_DEPTH_MAX;
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(smem + 256);
  uint32_t* const stop = tmem_slot + 1;
  int32_t* const rowvox = reinterpret_cast<int32_t*>(smem + 272);
  uint32_t* const adesc = reinterpret_cast<uint32_t*>(smem + ROW_HEAD);
  const uint32_t units4 = (p.units + 3) & ~3u;
  int32_t* const kcol = reinterpret_cast<int32_t*>(adesc + units4);
  const uint32_t sa_ofs = row_tables(p.units);
  const uint32_t sa = smem_u32(smem) + sa_ofs, sb = sa + p.planes * p.pitch;
  const uint32_t t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31u;
  const uint32_t x0 = (blockIdx.x % p.ctiles) * XG * 8u, r0 = (blockIdx.x / p.ctiles) * ROW_TILE;
  const uint32_t n0 = blockIdx.y * p.nt;
  const uint32_t nst = (p.units + p.ups - 1) / p.ups, depth = p.depth;
  const uint32_t rowp = p.W * 16u, blbo = p.nt * 16u + 16u, stage_bytes = 2u * p.ups * blbo;
  const uint32_t cols = XG * p.nt <= 32 ? 32u : XG * p.nt <= 64 ? 64u : XG * p.nt <= 128 ? 128u : XG * p.nt <= 256 ? 256u : 512u;
  const uint32_t groups = min((uint32_t)XG, (p.w - x0 + 7u) / 8u);

  if (t < p.nrows) {
    int64_t R;
    if (p.run) R = (int64_t)r0 - (p.band0 + p.zstep) + t;
    else R = (int64_t)r0 + ((int64_t)(t / (ROW_TILE + 2)) - 1) * p.hp + (t % (ROW_TILE + 2)) - 1;
    rowvox[t] = row_voxel(p, R);
  }
  if (warp == ROW_LOADERS / 32) {
    if (lane == 0) {
      for (uint32_t i = 0; i < depth; i++) {
        mbar_init(smem_u32(&full[i]), ROW_LOADERS);
        mbar_init(smem_u32(&done[i]), 1);
      }
      *stop = 0u;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  } else if (p.planes > p.cg) {
    for (uint32_t i = t * 16u; i < p.pitch; i += ROW_LOADERS * 16u)
      *reinterpret_cast<uint4*>(smem + sa_ofs + p.cg * p.pitch + i) = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  // per MMA: its input descriptor's low word (start address, K stride) and the weight
  // columns of its two K halves (-1: zeros)
  for (uint32_t u = t; u < p.units; u += ROW_THREADS) {
    uint32_t tap, g = 0, lbo = p.pitch;
    int32_t k0 = (int32_t)(16u * u), k1 = k0 + 8;
    if (p.upt) {
      tap = u / p.upt;
      g = 2u * (u - tap * p.upt);
      k0 = (int32_t)((tap * p.cg + g) * 8u);
      k1 = g + 1 < p.cg ? k0 + 8 : -1;
    } else if (p.cg == 1) {
      tap = 2u * u;
    } else {
      tap = u / (p.cg >> 1);
      g = 2u * (u - tap * (p.cg >> 1));
    }
    auto tap_off = [&](uint32_t tp) -> uint32_t {
      const int sg = (MODE == FWD) ? 1 : -1;
      const int dz = sg * tap_dz(tp, p.taps), dy = sg * tap_dy(tp, p.taps), dx = sg * tap_dx(tp, p.taps);
      return (p.band0 + (uint32_t)(dz + (int)p.halo) * p.zstep + (uint32_t)dy) * rowp + (uint32_t)((int)p.halo + dx) * 16u;
    };
    const uint32_t off = tap_off(tap);
    if (!p.upt && p.cg == 1 && tap + 1 < p.taps) lbo = tap_off(tap + 1) - off;
    adesc[u] = ((sa + g * p.pitch + off) >> 4) | ((lbo >> 4) << 16);
    kcol[2 * u] = k0;
    kcol[2 * u + 1] = k1 < (int32_t)p.K ? k1 : -1;
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  bool ok = true;
  if (warp == ROW_LOADERS / 32) {
    // One elected lane issues from unrolled code on tabulated descriptors: an MMA then
    // takes its own 39 (N 16) to 64 (N 128) cycles.  (With the taps' arithmetic or a
    // loop over the x groups between the MMAs, each took 160-260.)
    const uint32_t idesc = idesc_bf16(BM, p.nt);
    const uint64_t ahi = (uint64_t)((rowp >> 4) | (1u << 14)) << 32, bhi = (uint64_t)((128u >> 4) | (1u << 14)) << 32;
    uint32_t elected;
    asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(elected));
    uint32_t slot = 0, phase = 0, tslot = 0, tphase = 0;  // tslot, tphase: of stage kt - 2
    for (uint32_t kt = 0; kt < nst; kt++) {
      if (kt >= 2) {  // MMAs of stage kt-2 done
        ok = mbar_wait(smem_u32(&done[tslot]), tphase, p.stage_wait);
        if (++tslot == depth) {
          tslot = 0;
          tphase ^= 1u;
        }
      }
      ok = ok && mbar_wait_or(smem_u32(&full[slot]), phase, stop);
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        if (elected) *reinterpret_cast<volatile uint32_t*>(stop) = 1u;
        // the MMAs issued so far still end before the tensor memory is freed
        if (kt > 0) {
          const uint32_t last = slot ? slot - 1 : depth - 1;
          mbar_wait(smem_u32(&done[last]), slot ? phase : phase ^ 1u, WAIT_LIMIT);
        }
        break;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elected) {
        const uint32_t u0 = kt * p.ups, u1 = min(p.units, u0 + p.ups), bstep = 2u * blbo >> 4;
        uint32_t blo = ((sb + slot * stage_bytes) >> 4) | ((blbo >> 4) << 16);
        for (uint32_t u = u0; u < u1; u += 4) {
          const uint4 a4 = *reinterpret_cast<const uint4*>(adesc + u);
          const uint32_t al[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
          for (uint32_t i = 0; i < 4; i++) {
            if (i == 0 || u + i < u1) {
              const uint64_t ad = ahi | al[i], bd = bhi | (blo + i * bstep);
#pragma unroll
              for (uint32_t xg = 0; xg < XG; xg++)  // x groups past the grid: their columns are not read
                mma_bf16(tmem + xg * p.nt, ad + xg * 8u, bd, idesc, u + i);
            }
          }
          blo += 4u * bstep;
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&done[slot]))
                     : "memory");
      }
      __syncwarp();
      if (++slot == depth) {
        slot = 0;
        phase ^= 1u;
      }
    }
    if (ok) {
      const uint32_t last = slot ? slot - 1 : depth - 1;
      ok = mbar_wait(smem_u32(&done[last]), slot ? phase : phase ^ 1u, WAIT_LIMIT);
    }
  } else {
    // the input tile: 16-byte chunks, channels fastest
    const uint32_t per_row = p.W * p.cg, q = ROW_LOADERS / per_row, rem = ROW_LOADERS - q * per_row;
    uint32_t r = t / per_row, e = t - r * per_row;
#pragma unroll 4
    for (uint32_t i = t; i < p.nrows * per_row; i += ROW_LOADERS) {
      const int32_t v0 = rowvox[r];
      const uint32_t xx = (e * p.cg_magic) >> 16, g = e - xx * p.cg;
      const uint32_t x = x0 + xx - p.halo;  // wraps below 0: past the grid
      const bool in = v0 >= 0 && x < p.w && (uint32_t)v0 + x < p.M;
      cp16(sa + g * p.pitch + (r * p.W + xx) * 16u, in ? p.a + (size_t)((uint32_t)v0 + x) * p.C + g * 8u : p.a, in);
      r += q;
      e += rem;
      if (e >= per_row) {
        e -= per_row;
        r++;
      }
    }
    // Weights: thread t copies K half t & (halves - 1) of every stage for its rows.
    const uint32_t halves = 2u * p.ups, hf = t & (halves - 1u), nstep = ROW_LOADERS / halves;  // halves: 8, 16 or 32
    const uint32_t dst0 = sb + hf * blbo;
    uint32_t slot = 0, phase = 1;
    for (uint32_t st = 0; st < nst; st++) {
      if (st >= depth && !mbar_wait_or(smem_u32(&done[slot]), phase, stop)) {
        *reinterpret_cast<volatile uint32_t*>(stop) = 1u;
        ok = false;
        break;
      }
      const uint32_t u2 = st * halves + hf;
      const int32_t k = u2 < 2u * p.units ? kcol[u2] : -1;
      const __nv_bfloat16* const src = p.b + (size_t)n0 * p.K + (k < 0 ? 0 : k);
      for (uint32_t n = t / halves; n < p.nt; n += nstep) {
        const bool in = k >= 0 && n0 + n < p.N;
        cp16(dst0 + slot * stage_bytes + n * 16u, in ? src + (size_t)n * p.K : p.b, in);
      }
      // arrives once all copies of this thread so far (with stage 0, the input tile's too) have landed
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[slot])) : "memory");
      if (++slot == depth) {
        slot = 0;
        phase ^= 1u;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncwarp();
  ok = __syncthreads_and(ok);
  if (!ok && t == 0) atomicExch(&g_conv_error, 1);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  // ---- epilogue: lane = voxel (t & 7) of row (t & 127) >> 3 of the tile, 16 columns
  // per tcgen05.ld; the two halves of the loading warps take them in turn
  if (ok && warp < ROW_LOADERS / 32) {
    const uint32_t row = r0 + ((t & 127u) >> 3), taddr = tmem + (((warp & 3u) * 32u) << 16);
    const int32_t v0 = row_voxel(p, row);
    const uint32_t per = p.nt / 16u, total = groups * per;
    for (uint32_t c = warp >> 2; c < total; c += 2) {
      __syncwarp();
      const uint32_t xg = c / per, c0 = 16u * (c - xg * per), x = x0 + 8u * xg + (t & 7u);
      uint32_t r[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
            "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
          : "r"(taddr + xg * p.nt + c0)
          : "memory");
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (v0 < 0 || x >= p.w || (uint32_t)v0 + x >= p.M) continue;
      const size_t o = (size_t)((uint32_t)v0 + x) * p.N;
#pragma unroll
      for (int hh = 0; hh < 2; hh++) {  // 8 columns at a time
        const uint32_t col = n0 + c0 + 8u * hh;
        if (col >= p.N) break;  // N is a multiple of 8
        if constexpr (MODE == FWD) {
          __nv_bfloat16 v[8];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            float f = __uint_as_float(r[8 * hh + j]);
            if (p.bias) f += __ldg(p.bias + col + j);
            if (p.relu) f = fmaxf(f, 0.0f);
            v[j] = __float2bfloat16_rn(f);
          }
          __nv_bfloat16* const y = reinterpret_cast<__nv_bfloat16*>(p.out) + o + col;
          if (p.vec) {
            uint4 w;
            memcpy(&w, v, 16);
            *reinterpret_cast<uint4*>(y) = w;
          } else {
#pragma unroll
            for (int j = 0; j < 8; j++) y[j] = v[j];
          }
        } else {
          float* const dx = reinterpret_cast<float*>(p.out) + o + col;
          if (p.vec) {
            *reinterpret_cast<uint4*>(dx) = make_uint4(r[8 * hh], r[8 * hh + 1], r[8 * hh + 2], r[8 * hh + 3]);
            *reinterpret_cast<uint4*>(dx + 4) = make_uint4(r[8 * hh + 4], r[8 * hh + 5], r[8 * hh + 6], r[8 * hh + 7]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; j++) dx[j] = __uint_as_float(r[8 * hh + j]);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == ROW_LOADERS / 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
  }
}

// ---------------------------------------------------------------------------
// WGRAD: D[co][(dy, ci)] += sum over a tile's voxels of dy[m][co] x[m + off][ci].
//
// A block owns one dz and one or all three dx (its accumulators in tensor memory)
// and the rows that start in its share of the voxels, in tiles (up to 16 numbered rows x 8 XG
// voxels, as above) for which it
// loads the output gradient and, with its halo, the input, into two buffers in
// turn.  Both operands are M/N-major: 8 channels of a voxel are 16 contiguous
// bytes, 8 voxels along x one core matrix, and the channel groups of a row are laid
// out one after the other (group pitch), rows following at channel groups x group
// pitch.  So the N groups of one MMA run through the channels of three successive
// rows: the taps dy = -1, 0, 1 come in one MMA of N = 3 cin (up to 256), with K =
// two groups of 8 voxels.  Only rows of the grid are walked: the K steps of a tile
// are tabulated by the loaders from the rows' validity, an odd group paired with
// zeros.  Measured, the network's 12 distinct layers at batch 16 / 1 (us in all, with
// the reduction): 3620 -> 860 / 1390 -> 252 against a gather of every tap's K slices
// through registers with 2-byte stores.  What bounds it now: on the wide layers the
// MMAs (cout of 8-16 uses an eighth to a quarter of M), on the others the copies'
// latency per tile.  M is 64 or 128: rows above cout are computed from whatever follows in
// shared memory and not read.
// Voxels of the tile's gradient rows and x rows (-1: zeros) and its K steps.
struct WgTile {
  int32_t yv[ROW_TILE], xv[ROW_TILE + 2];
  uint32_t steps, xl;      // first voxel in x; bit 31: the block's last tile
  uint2 step[WG_STEPS];    // descriptor low words of dy and x
};
static_assert(sizeof(WgTile) == 400 && WG_HEAD % 128 == 0, "tables fit the head");

template <int NM>
__global__ void __launch_bounds__(WG_THREADS) conv_wgrad_kernel(WgradArgs p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* const full = reinterpret_cast<uint64_t*>(smem);  // [WG_BUFS]
  uint64_t* const done = full + WG_BUFS;
  uint64_t* const tfull = done + WG_BUFS;     // [WG_TABLES]: a table is there
  uint64_t* const tfree = tfull + WG_TABLES;  // its readers are through with it
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(smem + 192);
  uint32_t* const stop = tmem_slot + 1;
  uint32_t* const nonzero = tmem_slot + 2;  // 0: no row of the grid in this block's tiles, the accumulators are unset
  WgTile* const tile = reinterpret_cast<WgTile*>(smem + 256);  // [WG_TABLES]
  const uint32_t s0 = smem_u32(smem) + WG_HEAD;
  const uint32_t zero = s0 + p.nbuf * p.buf;  // a zero row of the gradient tile, and three of the x tile
  const uint32_t t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31u;
  const uint32_t split = blockIdx.x, tg = blockIdx.y / p.chunks, g0 = (blockIdx.y - tg * p.chunks) * p.cgx;
  const int dz = p.halo ? (int)(p.dxs == 3 ? tg : tg / 3u) - 1 : 0;
  const uint32_t dx0 = p.halo && p.dxs == 1 ? tg % 3u : 0u;  // first dx + 1 of this block
  // this block's rows: those that start in its voxels, as numbered rows [rb, re)
  auto numbered = [&](uint32_t q) {
    const uint32_t zz = q / p.h, bb = zz / p.d;
    return (bb * p.dp + zz - bb * p.d) * p.hp + q - zz * p.h;
  };
  const uint32_t q0 = (uint32_t)min((uint64_t)p.vrows, split * p.k_chunk / p.w), q1 = (uint32_t)min((uint64_t)p.vrows, (split + 1) * p.k_chunk / p.w);
  const bool any = q0 < q1;
  const uint32_t rb = any ? numbered(q0) : 0u, re = any ? numbered(q1 - 1) + 1 : 0u;
  // dx = -1 never reads the last column; where a row's last group reaches past the
  // grid, its gradient there is zero and so has to be x (0 times infinity)
  const uint32_t xlim = p.halo && p.dxs == 1 && dx0 == 0 ? p.w - 1 : p.w;
  const uint32_t rpx = p.cgx * p.gpx, rpy = p.cgy * p.gpy;

  if (warp == ROW_LOADERS / 32) {
    if (lane == 0) {
      for (uint32_t i = 0; i < WG_BUFS; i++) {
        mbar_init(smem_u32(&full[i]), ROW_LOADERS);
        mbar_init(smem_u32(&done[i]), 1);
      }
      for (uint32_t i = 0; i < WG_TABLES; i++) {
        mbar_init(smem_u32(&tfull[i]), 1);
        mbar_init(smem_u32(&tfree[i]), ROW_LOADERS / 32 + 1);
      }
      *stop = 0u;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(p.cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  } else if (warp < ROW_LOADERS / 32) {
    for (uint32_t i = t * 16u; i < p.zbytes; i += ROW_LOADERS * 16u)
      *reinterpret_cast<uint4*>(smem + WG_HEAD + p.nbuf * p.buf + i) = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  bool ok = true;
  if (warp == ROW_LOADERS / 32) {
    const uint32_t idesc = idesc_bf16(p.m, p.n, 1);
    const uint64_t ahi = (uint64_t)((p.gpy >> 4) | (1u << 14)) << 32, bhi = (uint64_t)((p.gpx >> 4) | (1u << 14)) << 32;
    uint32_t elected;
    asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(elected));
    uint32_t acc = 0, kt = 0, b = 0, phase = 0, tab = 0, tphase = 0;
    for (bool more = any; more; kt++) {
      ok = mbar_wait_or(smem_u32(&tfull[tab]), tphase, stop) && mbar_wait_or(smem_u32(&full[b]), phase, stop, p.stage_wait);
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        if (elected) *reinterpret_cast<volatile uint32_t*>(stop) = 1u;
        break;
      }
      more = !(tile[tab].xl >> 31);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elected) {
        const WgTile& T = tile[tab];
        const uint32_t steps = T.steps, bs = p.bstep >> 4;
#pragma unroll 4
        for (uint32_t s = 0; s < steps; s++) {
          const uint2 v = T.step[s];
#pragma unroll
          for (uint32_t j = 0; j < NM; j++) mma_bf16(tmem + j * p.n, ahi | v.x, bhi | (v.y + j * bs), idesc, acc);
          acc = 1u;
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&done[b]))
                     : "memory");
      }
      __syncwarp();
      if (elected) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tfree[tab])) : "memory");
      if (++tab == WG_TABLES) {
        tab = 0;
        tphase ^= 1u;
      }
      if (++b == p.nbuf) {
        b = 0;
        phase ^= 1u;
      }
    }
    if (elected) *nonzero = acc;
    if (kt > 0) {
      const uint32_t last = smem_u32(&done[b ? b - 1 : p.nbuf - 1]), ph = b ? phase : phase ^ 1u;
      ok = mbar_wait(last, ph, WAIT_LIMIT) && ok;  // before the tensor memory is freed, whatever came before
    }
  } else if (warp == ROW_LOADERS / 32 + 1) {
    // Rows and K steps of the tile at row r0 and voxel x0 (buffer b), by one warp; the first
    // row that it leaves.  With an odd number of groups in all, the last row is left to
    // the next tile: K steps are the 16 voxels that follow one another in the grid.
    auto make_table = [&](uint32_t r0, uint32_t x0, uint32_t b, WgTile& T) -> uint32_t {
      const uint32_t base = s0 + b * p.buf;
      const uint32_t ng = min(p.xg, p.groups - (x0 >> 3));
      auto voxel = [&](int64_t R) -> int32_t {
        if (R < 0 || R >= (int64_t)p.rows) return -1;
        const uint32_t r = (uint32_t)R, q = r / p.hp, y = r - q * p.hp, bb = q / p.dp, z = q - bb * p.dp;
        return y < p.h && z < p.d ? (int32_t)(((bb * p.d + z) * p.h + y) * p.w) : -1;
      };
      if (lane < p.xrows) T.xv[lane] = voxel((int64_t)r0 + dz * (int)p.hp + lane - p.halo);
      int32_t yv = lane < p.rt && r0 + lane < re ? voxel((int64_t)r0 + lane) : -1;
      uint32_t valid = __ballot_sync(0xffffffffu, yv >= 0), next = r0 + p.rt;
      if (p.ctiles == 1 && next < re && (__popc(valid) * ng & 1u) && __popc(valid) > 1) {
        const uint32_t l = 31u - __clz(valid);
        valid &= ~(1u << l);
        next = r0 + l;
        if (lane == l) yv = -1;
      }
      const uint32_t units = __popc(valid) * ng;
      if (lane < p.rt) T.yv[lane] = yv;
      if (lane == 0) T.steps = (units + 1) / 2;
      const uint32_t u = 2u * lane;
      if (u < units) {
        auto place = [&](uint32_t v, uint32_t& row, uint32_t& g) {
          uint32_t rank = v / ng;
          g = v - rank * ng;
          uint32_t m = valid;
          for (; rank > 0; rank--) m &= m - 1;
          row = __ffs(m) - 1;
        };
        uint32_t ra, ga, rb, gb;
        place(u, ra, ga);
        const uint32_t aa = base + ra * rpy + ga * 128u, xa = base + p.xofs + ra * rpx + ga * 128u + (p.halo ? dx0 * 16u : 0u);
        // half a step: zeros against zeros (against another x, an infinity would give a NaN): the voxels past
        // the grid in the same row where the tile has a group of them, else the zero rows
        uint32_t la = zero - aa, lx = p.dxs == 1 && ng < p.xg ? 144u - 16u * dx0 : zero + rpy - xa;
        if (u + 1 < units) {
          place(u + 1, rb, gb);
          la = (rb - ra) * rpy + gb * 128u - ga * 128u;
          lx = (rb - ra) * rpx + gb * 128u - ga * 128u;
        }
        T.step[lane] = make_uint2((aa >> 4) | ((la >> 4) << 16), (xa >> 4) | ((lx >> 4) << 16));
      }
      return next;
    };
    // (Formed by a loading warp between its copies a table kept the others waiting for
    // 2300 cycles a tile.)
    uint32_t kt = 0, b = 0, tab = 0, phase = 1, r = rb, c = 0;
    for (bool more = any; more; kt++) {
      if (kt >= WG_TABLES) ok = mbar_wait_or(smem_u32(&tfree[tab]), phase, stop);
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        *reinterpret_cast<volatile uint32_t*>(stop) = 1u;
        break;
      }
      const uint32_t next = make_table(r, c * p.xg * 8u, b, tile[tab]);
      if (lane == 0) tile[tab].xl = c * p.xg * 8u | (c + 1 == p.ctiles && next >= re ? 1u << 31 : 0u);
      if (++c == p.ctiles) {
        c = 0;
        r = next;
        more = r < re;
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tfull[tab])) : "memory");
      if (++tab == WG_TABLES) {
        tab = 0;
        phase ^= 1u;
      }
      if (++b == p.nbuf) b = 0;
    }
  } else {
    uint32_t kt = 0, b = 0, phase = 1, tab = 0, tphase = 0;
    for (bool more = any; more; kt++) {
      const uint32_t base = s0 + b * p.buf;
      ok = mbar_wait_or(smem_u32(&tfull[tab]), tphase, stop) && (kt < p.nbuf || mbar_wait_or(smem_u32(&done[b]), phase, stop, p.stage_wait));
      if (!ok) {
        *reinterpret_cast<volatile uint32_t*>(stop) = 1u;
        break;
      }
      const WgTile& T = tile[tab];
      const uint32_t x0 = T.xl & 0x7fffffffu;
      more = !(T.xl >> 31);
      {
        const uint32_t per = 8u * p.xg * p.cgy, q = ROW_LOADERS / per, rem = ROW_LOADERS - q * per;
        uint32_t r = t / per, e = t - r * per;
#pragma unroll 4
        for (uint32_t k = t; k < p.rt * per; k += ROW_LOADERS) {
          const int32_t v0 = T.yv[r];
          const uint32_t xx = (e * p.magy) >> 16, g = e - xx * p.cgy, x = x0 + xx;
          const bool in = v0 >= 0 && x < p.w && (uint32_t)v0 + x < p.M;
          cp16(base + r * rpy + g * p.gpy + xx * 16u, in ? p.dy + (size_t)((uint32_t)v0 + x) * p.cout + g * 8u : p.dy, in);
          r += q;
          e += rem;
          if (e >= per) {
            e -= per;
            r++;
          }
        }
      }
      {
        const uint32_t per = p.W * p.cgx, q = ROW_LOADERS / per, rem = ROW_LOADERS - q * per;
        uint32_t r = t / per, e = t - r * per;
#pragma unroll 4
        for (uint32_t k = t; k < p.xrows * per; k += ROW_LOADERS) {
          const int32_t v0 = T.xv[r];
          const uint32_t xx = (e * p.magx) >> 16, g = e - xx * p.cgx, x = x0 + xx - p.halo;
          const bool in = v0 >= 0 && x < xlim && (uint32_t)v0 + x < p.M && (g0 + g) * 8u < p.cin;
          cp16(base + p.xofs + r * rpx + g * p.gpx + xx * 16u, in ? p.x + (size_t)((uint32_t)v0 + x) * p.cin + (g0 + g) * 8u : p.x, in);
          r += q;
          e += rem;
          if (e >= per) {
            e -= per;
            r++;
          }
        }
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[b])) : "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tfree[tab])) : "memory");
      if (++tab == WG_TABLES) {
        tab = 0;
        tphase ^= 1u;
      }
      if (++b == p.nbuf) {
        b = 0;
        phase ^= 1u;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncwarp();
  ok = __syncthreads_and(ok);
  if (!ok && t == 0) atomicExch(&g_conv_error, 1);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  // ---- epilogue: lane = output channel, columns = (dy, ci) of each dx (or ci of each dy)
  if (ok && warp < ROW_LOADERS / 32) {
    // M 128: lane = row; M 64: rows 16 w .. 16 w + 15 in the first lanes of quarter w
    const uint32_t co = p.m == 64 ? ((warp & 3u) * 16u + lane) | (lane & 16u ? 128u : 0u) : t & 127u, taddr = tmem + (((warp & 3u) * 32u) << 16), per = p.n / 16u;
    const uint32_t cb = 8u * p.cgx;  // channels of this block
    const uint32_t used = NM == 3 && p.dxs == 1 ? cb : (p.halo ? 3u : 1u) * cb;  // columns of an accumulator
    float* const out = p.ws + (size_t)split * p.taps * p.cin * p.cout + co;
    const bool zeros = *nonzero == 0u;
    for (uint32_t c = warp >> 2; c < NM * per; c += 2) {
      __syncwarp();
      const uint32_t j = c / per, c0 = 16u * (c - j * per);
      uint32_t r[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
            "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
          : "r"(taddr + j * p.n + c0)
          : "memory");
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (co >= p.cout) continue;
#pragma unroll
      for (uint32_t k = 0; k < 16; k++) {
        const uint32_t col = c0 + k;
        if (col >= used) break;
        uint32_t ci = col, tap = 0;
        if (p.halo) {
          const uint32_t dyi = NM == 3 && p.dxs == 1 ? j : col / cb;
          if (!(NM == 3 && p.dxs == 1)) ci = col - dyi * cb;
          tap = (uint32_t)(dz + 1) * 9u + dyi * 3u + (p.dxs == 3 ? j : dx0);
        }
        ci += 8u * g0;
        if (ci >= p.cin) continue;
        const uint32_t row = tap * p.cin + ci;
        out[(size_t)row * p.cout] = zeros ? 0.0f : __uint_as_float(r[k]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == ROW_LOADERS / 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.cols) : "memory");
  }
}

// ---------------------------------------------------------------------------
// All three gathered voxel by voxel: the grids whose rows fill too little of a tile of
// numbered rows (one voxel a row: 1 of 8, and a zero row for each where planes have one
// row), and those whose numbered rows pass 31 bits.  gather_is_cheaper (wt_conv_plan.h)
// says which.
//
// A block: 128 threads, a 128 x N tile (N <= 128).  K runs in slices of 64 through two
// shared-memory stages: all threads gather a slice of A (128 rows) and B (N rows) into
// the K-major core-matrix layout (8 rows x 16 bytes; core matrices 128 B apart along K,
// 1024 B along M/N), one thread issues four MMAs (K = 16 each) and commits them to the
// stage's mbarrier, and the next slice is gathered into the other stage meanwhile.  What
// bounds it is that chain, 1.5 us and up a slice.
constexpr int GA_K = 64, GA_THREADS = 128;
constexpr uint32_t GA_STAGE = BM * GA_K * 2;          // one operand slice, 16 KB
constexpr uint32_t GA_SMEM = 4 * GA_STAGE + 64;       // A0 A1 B0 B1, barriers, tensor-memory slot
constexpr uint32_t GA_COLS = 128;

struct GatherArgs {
  uint32_t d, h, w;
  uint32_t cin, cout, taps;
  uint32_t M, N, K;        // GEMM extents
  uint32_t k_chunk;        // K per split (WGRAD; a multiple of GA_K), K otherwise
  const __nv_bfloat16* a;  // FWD x, DGRAD dy, WGRAD x
  const __nv_bfloat16* b;  // FWD w, DGRAD wt, WGRAD dy
  const float* bias;
  void* out;               // FWD bf16 y[M][cout], DGRAD f32 dx[M][cin], WGRAD f32 ws[split][M][N]
  int relu;
  uint32_t stage_wait;
};

// Shared-memory matrix descriptor from byte offsets.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)(addr >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46;
}

// Byte offset of 16-byte chunk (row r, k-group g) in the core-matrix layout.
__device__ __forceinline__ uint32_t chunk_off(uint32_t r, uint32_t g) { return ((r >> 3) * 8u + g) * 128u + (r & 7u) * 16u; }

__device__ __forceinline__ uint4 ld16(const __nv_bfloat16* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }

// Grid position of a voxel (x fastest, then y, z, batch item).
struct VoxPos {
  int x, y, z;
  int64_t vox;
  bool ok;
};

__device__ __forceinline__ VoxPos vox_pos(const GatherArgs& p, uint32_t m, uint32_t end) {
  VoxPos r;
  r.ok = m < end;
  const uint32_t mm = r.ok ? m : 0u;
  r.x = (int)(mm % p.w);
  r.y = (int)((mm / p.w) % p.h);
  r.z = (int)((mm / (p.w * p.h)) % p.d);
  r.vox = mm;
  return r;
}

// Index of the voxel r + (dz, dy, dx) in the same batch item, or -1 outside the grid.
__device__ __forceinline__ int64_t nbr(const GatherArgs& p, const VoxPos& r, int dz, int dy, int dx) {
  const int xx = r.x + dx, yy = r.y + dy, zz = r.z + dz;
  if ((unsigned)xx >= p.w || (unsigned)yy >= p.h || (unsigned)zz >= p.d) return -1;
  return r.vox + ((int64_t)dz * p.h + dy) * p.w + dx;
}

// Gather K slice [k0, k0 + 64) of both operands into the stage buffers sa, sb.
//   FWD / DGRAD: thread t owns A row t (a voxel, position precomputed in `row`)
//   and B row t (a weight row); each 16-byte chunk is 8 consecutive channels of
//   one tap, one vector load.
//   WGRAD: K runs over voxels; thread t owns voxel k0 + (t & 63) and half
//   (t >> 6) of the A rows (taps x channels) and B rows (output channels); it
//   loads 8 channels of its voxel with one vector load and stores them into 8
//   rows of the K-major tile (2-byte stores).
// Rows past the MMA's N (B) are never read and not written; K past the range
// is zero in both operands.
template <int MODE>
__device__ __forceinline__ void gather(const GatherArgs& p, const VoxPos& row, uint32_t tile_m, uint32_t n_mma,
                                       uint32_t k0, uint32_t k_end, uint8_t* sa, uint8_t* sb) {
  const uint32_t t = threadIdx.x;
  if constexpr (MODE == FWD || MODE == DGRAD) {
    const uint32_t C = (MODE == FWD) ? p.cin : p.cout;
    const int sg = (MODE == FWD) ? 1 : -1;
    uint32_t tap = k0 / C, c = k0 % C;
#pragma unroll
    for (uint32_t g = 0; g < 8; g++) {
      const uint32_t k = k0 + 8 * g;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (row.ok && k < k_end) {
        const int64_t sv = nbr(p, row, sg * tap_dz(tap, p.taps), sg * tap_dy(tap, p.taps), sg * tap_dx(tap, p.taps));
        if (sv >= 0) v = ld16(p.a + (size_t)sv * C + c);
      }
      *reinterpret_cast<uint4*>(sa + chunk_off(t, g)) = v;
      c += 8;
      if (c >= C) {
        c = 0;
        tap++;
      }
    }
    if (t < n_mma) {
#pragma unroll
      for (uint32_t g = 0; g < 8; g++) {
        const uint32_t k = k0 + 8 * g;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (t < p.N && k < k_end) v = ld16(p.b + (size_t)t * p.K + k);
        *reinterpret_cast<uint4*>(sb + chunk_off(t, g)) = v;
      }
    }
  } else {
    const uint32_t j = t & 63u, half = t >> 6;
    const VoxPos m = vox_pos(p, k0 + j, k_end);
    const uint32_t jo = (j & 7u) * 2u, jg = j >> 3;
    // A rows half*64 .. +63 = (tap, ci) rows tile_m + ...
#pragma unroll
    for (uint32_t q = 0; q < 8; q++) {
      const uint32_t r0 = half * 64u + 8u * q, R0 = tile_m + r0;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (m.ok && R0 < p.M) {
        const uint32_t tap = R0 / p.cin, ci = R0 % p.cin;
        const int64_t sv = nbr(p, m, tap_dz(tap, p.taps), tap_dy(tap, p.taps), tap_dx(tap, p.taps));
        if (sv >= 0) v = ld16(p.a + (size_t)sv * p.cin + ci);
      }
      const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 8; e++)
        *reinterpret_cast<uint16_t*>(sa + chunk_off(r0 + e, jg) + jo) = (uint16_t)(w4[e >> 1] >> ((e & 1) * 16));
    }
    // B rows (output channels) half*64 .. +63, only those the MMA reads
#pragma unroll
    for (uint32_t q = 0; q < 8; q++) {
      const uint32_t r0 = half * 64u + 8u * q;
      if (r0 >= n_mma) break;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (m.ok && r0 < p.N) v = ld16(p.b + (size_t)m.vox * p.cout + r0);
      const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 8; e++)
        *reinterpret_cast<uint16_t*>(sb + chunk_off(r0 + e, jg) + jo) = (uint16_t)(w4[e >> 1] >> ((e & 1) * 16));
    }
  }
}

template <int MODE>
__global__ void __launch_bounds__(GA_THREADS, 1) conv_gather_kernel(GatherArgs p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  // stage s: A at smem + s * GA_STAGE, B at smem + (2 + s) * GA_STAGE
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 4 * GA_STAGE);  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 4 * GA_STAGE + 16);
  const uint32_t t = threadIdx.x, warp = t >> 5;
  const uint32_t tile_m = blockIdx.x * BM;
  const uint32_t k_begin = blockIdx.y * p.k_chunk;
  const uint32_t k_end = min(p.K, k_begin + p.k_chunk);
  const uint32_t nk = (k_end > k_begin) ? (k_end - k_begin + GA_K - 1) / GA_K : 0;
  const uint32_t n_mma = ((p.N + 15) / 16) * 16;
  const uint32_t idesc = idesc_bf16(BM, n_mma);

  if (t == 0) {
    mbar_init(smem_u32(&bars[0]), 1);
    mbar_init(smem_u32(&bars[1]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(GA_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  const VoxPos row_pos = vox_pos(p, tile_m + t, p.M);  // FWD / DGRAD: this thread's A row (a voxel)
  bool ok = true;
  uint32_t issued = 0;  // K slices whose MMAs were issued (uniform across the block)
  for (uint32_t kt = 0; kt < nk; kt++) {
    const uint32_t s = kt & 1u;
    bool w = true;
    if (kt >= 2) w = mbar_wait(smem_u32(&bars[s]), ((kt >> 1) - 1) & 1u, p.stage_wait);  // MMAs of slice kt-2 done
    if (!__syncthreads_and(w)) {  // the block stops together
      ok = false;
      break;
    }
    uint8_t* const sa = smem + s * GA_STAGE;
    uint8_t* const sb = smem + (2u + s) * GA_STAGE;
    gather<MODE>(p, row_pos, tile_m, n_mma, k_begin + kt * GA_K, k_end, sa, sb);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (t == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a0 = smem_u32(sa), b0 = smem_u32(sb);
#pragma unroll
      for (uint32_t kk = 0; kk < GA_K / 16; kk++) {
        const uint64_t ad = smem_desc(a0 + kk * 256u, 128u, 1024u);
        const uint64_t bd = smem_desc(b0 + kk * 256u, 128u, 1024u);
        const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&bars[s]))
                   : "memory");
    }
    issued++;
  }
  // All MMAs done: the last commit covers every earlier one of the issuing thread.
  if (issued > 0) {
    const uint32_t last = issued - 1;
    const bool done = mbar_wait(smem_u32(&bars[last & 1u]), (last >> 1) & 1u, WAIT_LIMIT);
    ok = ok && done;
  }
  if (!ok && t == 0) atomicExch(&g_conv_error, 1);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  // ---- epilogue: lane = row t of the tile, 16 columns per tcgen05.ld
  const uint32_t row = tile_m + t;
  const uint32_t taddr = tmem + ((warp * 32u) << 16);
  for (uint32_t c0 = 0; c0 < n_mma; c0 += 16) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr + c0)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (!ok || row >= p.M || nk == 0) continue;
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const uint32_t col = c0 + j;
      if (col >= p.N) break;
      float v = __uint_as_float(r[j]);
      if constexpr (MODE == FWD) {
        if (p.bias) v += p.bias[col];
        if (p.relu) v = fmaxf(v, 0.0f);
        reinterpret_cast<__nv_bfloat16*>(p.out)[(size_t)row * p.N + col] = __float2bfloat16_rn(v);
      } else if constexpr (MODE == DGRAD) {
        reinterpret_cast<float*>(p.out)[(size_t)row * p.N + col] = v;
      } else {
        reinterpret_cast<float*>(p.out)[((size_t)blockIdx.y * p.M + row) * p.N + col] = v;
      }
    }
  }
  if (nk == 0 && row < p.M) {  // empty K range: the product is zero
    for (uint32_t col = 0; col < p.N; col++) {
      if constexpr (MODE == FWD) {
        float v = p.bias ? p.bias[col] : 0.0f;
        if (p.relu) v = fmaxf(v, 0.0f);
        reinterpret_cast<__nv_bfloat16*>(p.out)[(size_t)row * p.N + col] = __float2bfloat16_rn(v);
      } else if constexpr (MODE == DGRAD) {
        reinterpret_cast<float*>(p.out)[(size_t)row * p.N + col] = 0.0f;
      } else {
        reinterpret_cast<float*>(p.out)[((size_t)blockIdx.y * p.M + row) * p.N + col] = 0.0f;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(GA_COLS) : "memory");
  }
}

// dw[co][t][ci] = sum over splits of ws[split][(t, ci)][co]: a block takes 32
// outputs, its eight warps every eighth split each (in FP64, folded in order).
__global__ void wgrad_reduce_kernel(const float* __restrict__ ws, float* __restrict__ dw, uint32_t splits,
                                    uint32_t rows, uint32_t cout, uint32_t taps, uint32_t cin) {
  __shared__ double red[8][32];
  const uint32_t lane = threadIdx.x & 31u, ph = threadIdx.x >> 5;
  const uint32_t i = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (i < rows * cout)
#pragma unroll 4
    for (uint32_t k = ph; k < splits; k += 8) s += ws[(size_t)k * rows * cout + i];
  red[ph][lane] = s;
  __syncthreads();
  if (ph != 0 || i >= rows * cout) return;
  for (uint32_t q = 1; q < 8; q++) s += red[q][lane];
  const uint32_t row = i / cout, co = i % cout;  // row = t * cin + ci
  const uint32_t tap = row / cin, ci = row % cin;
  dw[((size_t)co * taps + tap) * cin + ci] = (float)s;
}

int nfail(int code, const std::string& m) {
  net_error() = m;
  return code;
}

int check_shape(const wt_conv_shape* s, const char* what) {
  if (!s) return nfail(WT_ERR_ARG, std::string(what) + ": null shape");
  if (s->taps != 27 && s->taps != 1) return nfail(WT_ERR_ARG, std::string(what) + ": taps must be 27 or 1");
  if (s->cin == 0 || s->cout == 0 || s->cin % 8 || s->cout % 8 || s->cin > 128 || s->cout > 128)
    return nfail(WT_ERR_ARG, std::string(what) + ": channel counts must be multiples of 8 in [8, 128]");
  if (s->batch == 0 || s->d == 0 || s->h == 0 || s->w == 0) return nfail(WT_ERR_ARG, std::string(what) + ": empty grid");
  if ((uint64_t)s->batch * s->d * s->h * s->w >= (1ull << 31)) return nfail(WT_ERR_ARG, std::string(what) + ": grid too large");
  return WT_OK;
}

template <int MODE>
int launch_gather(const GatherArgs& p, uint32_t splits, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(conv_gather_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GA_SMEM);
  if (e != cudaSuccess) return nfail(WT_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  conv_gather_kernel<MODE><<<dim3((p.M + BM - 1) / BM, splits), GA_THREADS, GA_SMEM, st>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return nfail(WT_ERR_CUDA, std::string("conv kernel launch: ") + cudaGetErrorString(e));
  return WT_OK;
}

GatherArgs gather_args(const wt_conv_shape* s, const void* a, const void* b, void* out) {
  GatherArgs p = {};
  p.d = s->d, p.h = s->h, p.w = s->w;
  p.cin = s->cin, p.cout = s->cout, p.taps = s->taps;
  p.a = static_cast<const __nv_bfloat16*>(a);
  p.b = static_cast<const __nv_bfloat16*>(b);
  p.out = out;
  p.stage_wait = g_stage_wait.load();
  return p;
}

template <int MODE, int XG>
int launch_rows_xg(const RowArgs& p, uint32_t smem, dim3 grid, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(conv_rows_kernel<MODE, XG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
  if (e != cudaSuccess) return nfail(WT_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  conv_rows_kernel<MODE, XG><<<grid, ROW_THREADS, smem, st>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return nfail(WT_ERR_CUDA, std::string("conv kernel launch: ") + cudaGetErrorString(e));
  return WT_OK;
}

template <int MODE>
int launch_rows(const wt_conv_shape* s, const void* a, const void* b, const float* bias, void* out, int relu, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  RowArgs p = {};
  RowPlan q = {};
  if (!plan_rows(*s, MODE == FWD, p, q) || gather_is_cheaper(p, q)) {
    GatherArgs ga = gather_args(s, a, b, out);
    ga.bias = bias;
    ga.relu = relu;
    ga.M = s->batch * s->d * s->h * s->w;
    ga.N = p.N;
    ga.K = ga.k_chunk = p.K;
    return launch_gather<MODE>(ga, 1, st);
  }
  p.a = static_cast<const __nv_bfloat16*>(a);
  p.b = static_cast<const __nv_bfloat16*>(b);
  p.bias = bias;
  p.out = out;
  p.relu = relu;
  p.stage_wait = g_stage_wait.load();
  p.vec = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const dim3 grid(q.blocks, q.nblocks);
  if (q.xg == 4) return launch_rows_xg<MODE, 4>(p, q.smem, grid, st);
  if (q.xg == 2) return launch_rows_xg<MODE, 2>(p, q.smem, grid, st);
  return launch_rows_xg<MODE, 1>(p, q.smem, grid, st);
}

int launch_wgrad(const wt_conv_shape* s, const void* x, const void* dy, float* ws, uint32_t splits, cudaStream_t st) {
  WgradArgs p = {};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.dy = static_cast<const __nv_bfloat16*>(dy);
  p.ws = ws;
  uint32_t nm = 0, smem = 0;
  if (!plan_wgrad(*s, splits, p, nm, smem) || gather_is_cheaper(p, splits)) {
    GatherArgs ga = gather_args(s, x, dy, ws);
    ga.M = s->taps * s->cin;
    ga.N = s->cout;
    ga.K = s->batch * s->d * s->h * s->w;
    ga.k_chunk = (uint32_t)p.k_chunk;
    return launch_gather<WGRAD>(ga, splits, st);
  }
  p.stage_wait = p.M / splits > 128 ? g_stage_wait.load() : WAIT_LIMIT;  // up to two K slices of 64 voxels: no stage to wait for
  const dim3 grid(splits, (p.halo ? (p.dxs == 3 ? 3 : 9) : 1) * p.chunks);
  const auto kernel = nm == 3 ? conv_wgrad_kernel<3> : conv_wgrad_kernel<1>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
  if (e != cudaSuccess) return nfail(WT_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  kernel<<<grid, WG_THREADS, smem, st>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return nfail(WT_ERR_CUDA, std::string("conv kernel launch: ") + cudaGetErrorString(e));
  return WT_OK;
}

}  // namespace
}  // namespace wt

using namespace wt;

extern "C" {

int wt_conv3d_forward(const wt_conv_shape* s, const void* x, const void* w, const float* bias, void* y, int relu,
                      void* stream) {
  int rc = check_shape(s, "wt_conv3d_forward");
  if (rc) return rc;
  if (!x || !w || !y) return nfail(WT_ERR_ARG, "wt_conv3d_forward: null tensor");
  return launch_rows<FWD>(s, x, w, bias, y, relu, stream);
}

int wt_conv3d_backward_data(const wt_conv_shape* s, const void* dy, const void* wt, float* dx, void* stream) {
  int rc = check_shape(s, "wt_conv3d_backward_data");
  if (rc) return rc;
  if (!dy || !wt || !dx) return nfail(WT_ERR_ARG, "wt_conv3d_backward_data: null tensor");
  return launch_rows<DGRAD>(s, dy, wt, nullptr, dx, 0, stream);
}

size_t wt_conv3d_workspace_bytes(const wt_conv_shape* s) {
  if (check_shape(s, "wt_conv3d_workspace_bytes")) return 0;
  const uint64_t vox = (uint64_t)s->batch * s->d * s->h * s->w;
  return (size_t)wgrad_splits(vox) * s->taps * s->cin * s->cout * sizeof(float);
}

int wt_conv3d_backward_weight(const wt_conv_shape* s, const void* x, const void* dy, float* dw, void* workspace,
                              void* stream) {
  int rc = check_shape(s, "wt_conv3d_backward_weight");
  if (rc) return rc;
  if (!x || !dy || !dw || !workspace) return nfail(WT_ERR_ARG, "wt_conv3d_backward_weight: null tensor");
  const uint64_t vox = (uint64_t)s->batch * s->d * s->h * s->w;
  const uint32_t splits = wgrad_splits(vox), rows = s->taps * s->cin, total = rows * s->cout;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rc = launch_wgrad(s, x, dy, static_cast<float*>(workspace), splits, st);
  if (rc) return rc;
  wgrad_reduce_kernel<<<(total + 31) / 32, 256, 0, st>>>(static_cast<const float*>(workspace), dw, splits, rows, s->cout,
                                                           s->taps, s->cin);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return nfail(WT_ERR_CUDA, std::string("wgrad reduce: ") + cudaGetErrorString(e));
  return WT_OK;
}

int wt_net_check(void) {
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return nfail(WT_ERR_CUDA, std::string("wt_net_check: ") + cudaGetErrorString(e));
  int flag = 0, zero = 0;
  cudaMemcpyFromSymbol(&flag, g_conv_error, sizeof(int));
  cudaMemcpyToSymbol(g_conv_error, &zero, sizeof(int));
  return flag;
}

const char* wt_net_last_error(void) { return net_error().c_str(); }

uint32_t wt_net_set_stage_wait_limit(uint32_t polls) { return g_stage_wait.exchange(polls); }

}  // extern "C"
