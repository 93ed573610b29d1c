// How the convolution kernels of wt_conv.cu tile a call: their argument blocks and the
// host's plan of shared memory, tensor memory and grid, free of CUDA so that a host
// program can evaluate it for every shape.
#pragma once
#include <stdint.h>

#include "wt_net.h"

struct __nv_bfloat16;

namespace wt {
namespace {

constexpr uint32_t SMS = 152, SMEM_MAX = 227 * 1024, SMEM_THIRD = 74 * 1024;
constexpr uint32_t ROW_TILE = 16, ROW_ROWS = 3 * (ROW_TILE + 2), ROW_HEAD = 512;  // ROW_HEAD: barriers, slot, ROW_ROWS row voxels
// Threads that load, and with the issuing warp; stages of the weight ring at most.
constexpr uint32_t ROW_LOADERS = 256, ROW_THREADS = ROW_LOADERS + 32, ROW_DEPTH_MAX = 16;

struct RowArgs {
  const __nv_bfloat16* a;  // FWD x, DGRAD dy
  const __nv_bfloat16* b;  // FWD w, DGRAD wt: [N][taps][C]
  const float* bias;
  void* out;               // FWD bf16 y[M][N], DGRAD f32 dx[M][N]
  uint32_t C, N, K, taps;  // input channels, output channels, taps * C
  uint32_t d, h, w, M;     // grid (one batch item) and voxels in all
  uint32_t hp, dp, rows;   // rows per plane and planes per item with their zero row / plane; rows in all
  uint32_t cg, planes;     // channel groups; planes in shared memory (the last one zero if cg is odd)
  uint32_t W, nrows, pitch;  // shared-memory tile: voxels per row, rows, bytes per plane
  uint32_t halo, run;      // 1 for 27 taps; 1 when the rows are one run
  uint32_t band0, zstep;   // shared-memory row of tile row 0 for dz = -1, and from one dz to the next
  uint32_t ctiles;         // tiles along x
  uint32_t nt, units, ups, upt;  // N per block; MMAs of K; MMAs per stage; MMAs per tap where K is padded per tap, else 0
  uint32_t depth;            // stages in the weight ring
  uint32_t cg_magic;       // ceil(2^16 / cg)
  int relu, vec;           // vec: out is 16-byte aligned and N a multiple of 8
  uint32_t stage_wait;
};

// Bytes of the head and of the MMAs' tables.
constexpr uint32_t row_tables(uint32_t units) { return (ROW_HEAD + (units + 3) / 4 * 4 * 12 + 127) / 128 * 128; }

struct WgradArgs {
  const __nv_bfloat16 *x, *dy;
  float* ws;               // [split][taps * cin][cout]
  uint32_t cin, cout, taps;
  uint32_t d, h, w, M, hp, dp, rows;  // as RowArgs
  uint32_t cgx, cgy;       // channel groups of x in a block, and of dy
  uint32_t chunks;         // blocks along cin
  uint32_t nbuf;           // tile buffers
  uint32_t magx, magy;     // ceil(2^16 / cgx), ceil(2^16 / cgy)
  uint32_t halo, W;        // voxels per row of the x tile
  uint32_t gpx, gpy;       // bytes per channel group of a row
  uint32_t xrows;          // rows of the x tile
  uint32_t xofs, buf;      // offset of the x tile in a buffer, bytes per buffer
  uint32_t xg, ctiles, rt; // voxel groups and rows of a tile
  uint32_t vrows;          // rows of the grid
  uint64_t k_chunk;        // voxels of a split
  uint32_t groups;         // x groups of a row of the grid
  uint32_t dxs;            // dx per block: 3, or 1 (one also splits cin into chunks)
  uint32_t m, n, bstep;    // M and N of one MMA; bytes between the x operands of an MMA and the next of its K step
  uint32_t cols;           // tensor-memory columns
  uint32_t stage_wait;     // polls of the waits for a tile and for its buffer
  uint32_t zbytes;         // the zero rows: one of the gradient's tile and, where half a K step may need them, three of the x tile's
};

constexpr uint32_t WG_STEPS = 32, WG_BUFS = 4, WG_TABLES = WG_BUFS + 2;  // K steps of a tile
constexpr uint32_t WG_HEAD = 256 + WG_TABLES * 400 + 32;               // barriers, tables
constexpr uint32_t WG_THREADS = ROW_THREADS + 32;                        // loaders, issuer, table warp

constexpr uint32_t WGRAD_SPLITS_MAX = 64;

uint32_t wgrad_splits(uint64_t voxels) {
  // about 4096 voxels (64 slices of 64) per split, at most WGRAD_SPLITS_MAX
  uint64_t s = (voxels + 4095) / 4096;
  if (s < 1) s = 1;
  if (s > WGRAD_SPLITS_MAX) s = WGRAD_SPLITS_MAX;
  return (uint32_t)s;
}

// A channel group's pitch such that eight successive 16-byte copies (channel groups
// fastest, then voxels) fall in different banks: 64, 32 or 16 mod 128 bytes.
uint32_t pad_pitch(uint32_t bytes, uint32_t cg) {
  const uint32_t want = cg >= 8 ? 16u : cg >= 4 ? 32u : cg >= 2 ? 64u : 0u;
  return bytes + (want + 128u - bytes % 128u) % 128u;
}

// What plan_rows settles beside the arguments.
struct RowPlan {
  uint32_t xg, blocks, nblocks, smem;  // voxel groups of a tile; blocks along the voxels and along N
};

// Tiling of conv_rows_kernel.  Wide tiles (xg groups of 8 voxels along x) share
// their halo and their weights; narrow ones and a split of N give a small grid
// enough blocks.  Shared memory of a block stays below a third of an SM's where it
// can, so that several blocks overlap their loads, MMAs and epilogues.
// False: the numbered rows do not fit 31 bits.
bool plan_rows(const wt_conv_shape& s, bool forward, RowArgs& p, RowPlan& q) {
  p.C = forward ? s.cin : s.cout;
  p.N = forward ? s.cout : s.cin;
  p.taps = s.taps;
  p.K = p.taps * p.C;
  p.M = s.batch * s.d * s.h * s.w;
  p.halo = s.taps == 27 ? 1u : 0u;
  uint32_t batch = s.batch;
  if (p.halo) {
    p.d = s.d, p.h = s.h, p.w = s.w;
    p.hp = p.h + 1, p.dp = p.d + 1;
  } else {  // pointwise: the voxels in rows of 32
    batch = 1, p.d = 1, p.w = 32, p.h = (p.M + 31) / 32;
    p.hp = p.h, p.dp = 1;
  }
  const uint64_t rows = ((uint64_t)batch * p.dp - p.halo) * p.hp - p.halo;  // up to the last row of the grid
  if (rows >= (1ull << 31)) return false;
  p.rows = (uint32_t)rows;
  p.cg = p.C / 8;
  p.planes = p.cg + (p.cg & 1u);
  p.cg_magic = (65536u + p.cg - 1) / p.cg;
  const uint64_t halo_rows = p.halo * ((uint64_t)p.hp + 1);
  p.run = !p.halo || ROW_TILE + 2 * halo_rows <= ROW_ROWS;
  p.nrows = p.run ? ROW_TILE + 2 * (uint32_t)halo_rows : ROW_ROWS;
  p.band0 = p.halo;  // row -1 of the first band is shared-memory row 0
  p.zstep = !p.halo ? 0 : p.run ? p.hp : ROW_TILE + 2;
  if (p.cg & 1u) {
    p.upt = (p.cg + 1) / 2;
    if (p.cg == 1 && forward && p.h > 1) p.upt = 0;  // (planes of one row: the distance of two taps may be negative)
  }
  p.units = p.upt ? p.taps * p.upt : (p.K + 15) / 16;
  const uint32_t rt = (p.rows + ROW_TILE - 1) / ROW_TILE, groups = (p.w + 7) / 8, n16 = (p.N + 15) / 16 * 16;
  auto tile = [&](uint32_t xg) {
    p.W = 8 * xg + 2 * p.halo;
    p.pitch = p.nrows * p.W * 16;
    p.pitch = pad_pitch(p.pitch, p.cg);
    p.ctiles = (groups + xg - 1) / xg;
  };
  // Longer stages where K is long: an MMA takes 40-70 cycles to issue, a stage's
  // waits about 400.  (Fewer than 32 MMAs: 4 to a stage, K slices of 64.)
  auto stage = [&](uint32_t nt) { return p.units < 32 ? 4u : p.units < 64 || nt > 32 ? 8u : 16u; };
  auto ring = [&](uint32_t nt) { return 2 * stage(nt) * (nt * 16 + 16); };
  uint32_t xg = 4;
  for (; xg > 1; xg >>= 1) {
    tile(xg);
    if (xg < 2 * groups && p.planes * p.pitch + 4 * ring(n16) <= (xg == 2 ? SMEM_MAX / 2 : SMEM_THIRD) - 4096 && xg * n16 <= 128 &&
        (uint64_t)rt * p.ctiles >= 2 * SMS)
      break;
  }
  tile(xg);
  p.nt = n16;
  while (p.nt > 16 && ((uint64_t)rt * p.ctiles * ((p.N + p.nt - 1) / p.nt) < SMS ||
                       row_tables(p.units) + p.planes * p.pitch + 4 * ring(p.nt) > SMEM_MAX))
    p.nt = (p.nt / 2 + 15) / 16 * 16;
  p.ups = stage(p.nt);
  const uint32_t nst = (p.units + p.ups - 1) / p.ups, a_bytes = row_tables(p.units) + p.planes * p.pitch;
  q.xg = xg, q.blocks = rt * p.ctiles, q.nblocks = (p.N + p.nt - 1) / p.nt;
  // A deep ring hides the weights' latency; it must not cost resident blocks.
  auto per_sm = [&](uint32_t depth) {
    const uint32_t fit = SMEM_MAX / (a_bytes + depth * ring(p.nt)), have = (q.blocks * q.nblocks + SMS - 1) / SMS;
    return fit < have ? fit : have;
  };
  p.depth = ROW_DEPTH_MAX;
  while (p.depth > 4 && (p.depth >= 2 * nst || !per_sm(p.depth) || per_sm(p.depth) < per_sm(4))) p.depth /= 2;
  q.smem = a_bytes + p.depth * ring(p.nt);
  return true;
}

// Whether a 3x3x3 call is cheaper gathered voxel by voxel than on numbered rows.  Both
// times are estimated, in us.  A block of rows costs its weights (read anew by every
// block), its tile and its MMAs whatever part of the tile the grid fills; a block of 128
// gathered voxels a chain of K slices of 64, several blocks to an SM overlapping theirs.
// The constants fit 35 grids of rows of 1 to 40 voxels, from 1x1x1 on, at 512 to 262144
// voxels and 7 pairs of channels, both measured (rows, gather): 65536 of 1x1x1, 16
// channels 284 and 33, 128 channels 3705 and 434; 4096 of 1x4x4, 128 channels 623 and
// 477; 512 of 2x2x2, 64 channels 35 and 84.  The estimate picks the faster one there up
// to 1 % on average and 45 % at worst.
bool gather_is_cheaper(const RowArgs& p, const RowPlan& q) {
  if (!p.halo) return false;  // pointwise voxels are packed
  const double C = p.C, N = p.N, b = (double)((p.M + 127) / 128) / SMS;
  const double rows = (double)q.blocks * q.nblocks / SMS * (1.8 + 0.002 * C * p.nt + (0.02 + 0.01 * q.xg) * C);
  const double gather = (double)((p.K + 63) / 64) * (1.5 + (0.85 + 0.007 * N) * b) + 0.05 * N * b;
  return rows > gather;
}

// Tiling of conv_wgrad_kernel.  A block takes all three dx where their accumulators
// fit the tensor memory (9 cin columns), the splits alone give every SM a block and
// rows end with a group of 8; otherwise one dx, for a finer grid, and where that
// still leaves SMs idle, cin in chunks (16 channels at least).  The workspace bounds
// the splits.  False: the numbered rows do not fit 31 bits.
bool plan_wgrad(const wt_conv_shape& s, uint32_t splits, WgradArgs& p, uint32_t& nm, uint32_t& smem) {
  p.cin = s.cin, p.cout = s.cout, p.taps = s.taps;
  p.M = s.batch * s.d * s.h * s.w;
  p.k_chunk = (((uint64_t)p.M + splits - 1) / splits + 63) / 64 * 64;
  p.halo = s.taps == 27 ? 1u : 0u;
  uint32_t batch = s.batch;
  if (p.halo) {
    p.d = s.d, p.h = s.h, p.w = s.w;
    p.hp = p.h + 1, p.dp = p.d + 1;
  } else {
    batch = 1, p.d = 1, p.w = 32, p.h = (p.M + 31) / 32;
    p.hp = p.h, p.dp = 1;
  }
  const uint64_t rows = ((uint64_t)batch * p.dp - p.halo) * p.hp - p.halo;  // up to the last row of the grid
  if (rows >= (1ull << 31)) return false;
  p.rows = (uint32_t)rows;
  p.cgy = p.cout / 8;
  p.magy = (65536u + p.cgy - 1) / p.cgy;
  p.groups = (p.w + 7) / 8;
  p.vrows = p.halo ? batch * p.d * p.h : p.h;
  auto r16 = [](uint32_t v) { return (v + 15) / 16 * 16; };
  const uint32_t cg = p.cin / 8, n3 = r16(3 * p.cin);
  uint32_t blocks = splits * (p.halo ? 9 : 1);
  nm = 1;
  p.cgx = cg;
  p.dxs = 1;
  if (p.halo && 3 * n3 <= 512 && 3 * splits >= SMS && p.w % 8 == 0) {
    p.dxs = nm = 3;
    blocks = 3 * splits;
  } else {
    while (p.cgx > 2 && blocks * ((cg + p.cgx - 1) / p.cgx) < SMS) p.cgx = (p.cgx + 1) / 2;
    if (p.halo && 3 * p.cgx * 8 > 256) nm = 3;  // one MMA per dy
  }
  p.chunks = (cg + p.cgx - 1) / p.cgx;
  blocks *= p.chunks;
  p.m = p.cout <= 64 ? 64 : 128;  // (N 48: 29 and 44 cycles an MMA)
  p.n = r16((p.halo && !(nm == 3 && p.dxs == 1) ? 3 : 1) * p.cgx * 8);
  p.magx = (65536u + p.cgx - 1) / p.cgx;
  // Rows of up to 4 groups, or of 8, whole where they are full: the K steps are then the 16
  // voxels that follow one another in the grid, in their order, and the sums the same
  // bits as those of a plain walk over the voxels (a training run amplifies the last bit:
  // Adam's first steps divide gradients by themselves).  There the tile's rows shrink
  // until it fits, elsewhere its groups.  (Rows of 5 to 7 groups would fit the tables too:
  // whole, 16x24x24 rows of 40 to 56 took 310 to 400 us instead of 397 to 523 with 64
  // channels and 779 to 1002 instead of 529 to 699 with 128 to 64, and were not equal in
  // their bits where the tile's rows had to shrink.)  A tile of one group that is over a half SM is
  // taken all the same; 104 channels and more on both sides are over the whole of it
  // and take 14 rows.
  const bool eight = p.groups == 8 && p.w % 8 == 0, whole = eight || (p.groups <= 4 && p.w % 8 == 0);
  for (p.xg = eight ? 8 : p.groups >= 3 ? 4 : p.groups, p.rt = eight ? 8 : ROW_TILE; ;) {
    p.xrows = p.rt + 2 * p.halo;
    p.W = 8 * p.xg + 2 * p.halo;
    p.gpx = pad_pitch(p.W * 16, p.cgx);
    p.gpy = pad_pitch(8 * p.xg * 16, p.cgy);
    p.xofs = p.rt * p.cgy * p.gpy;
    p.buf = (p.xofs + p.xrows * p.cgx * p.gpx + 127) / 128 * 128;
    const uint32_t zrows = p.xg & 1u || (p.dxs == 3 && p.groups & 1u) ? 3 : 0;
    // after the buffers: the zero rows, and what the junk M rows and N columns of the last rows read
    const uint32_t zeros = (p.cgy * p.gpy + (zrows * p.cgx + 1) * p.gpx + 256 + 127) / 128 * 128, junk = 16 * p.gpy + 16 * p.gpx + 2048;
    const uint32_t rest = WG_HEAD + (zeros > junk ? zeros : junk), most = blocks > SMS ? SMEM_MAX / 2 : SMEM_MAX;
    p.zbytes = p.cgy * p.gpy + zrows * p.cgx * p.gpx;
    for (p.nbuf = WG_BUFS; p.nbuf > 2 && rest + p.nbuf * p.buf > most; p.nbuf--) {}
    smem = rest + p.nbuf * p.buf;
    if (smem <= most || (p.xg == 1 && smem <= SMEM_MAX && (!whole || p.rt == 4))) break;
    if (whole && p.rt > 4) p.rt /= 2;
    else if (p.xg > 1) p.xg /= 2, p.rt = ROW_TILE;
    else if (p.rt > 4) p.rt -= 2;
    else break;
  }
  p.bstep = p.dxs == 3 ? 16u : p.cgx * p.gpx;
  p.ctiles = (p.groups + p.xg - 1) / p.xg;
  for (p.cols = 32; p.cols < nm * p.n; p.cols *= 2) {}
  return true;
}

// The weight gradient's.  Both walk the voxels of a split as one chain (tiles of rows,
// slices of 64 voxels), so the tiles per 128 voxels decide: 5.6 of them while an SM has
// one block, less the more splits read wide tiles at a time; 4.1 where it has several;
// 3 where the splits would fill the device with three dx to a block but the row width
// forbids it.  On the same grids and larger ones (to 1048576 voxels) 1 to 2 % off the
// faster one on average.  Rows, gather: 4096 of 1x1x1, 64 channels 1176 and 247 us; 1024
// of 4x4x4, 16 channels 160 and 218; 262144 voxels in 3x3x4, 16 channels 412 and 246.
bool gather_is_cheaper(const WgradArgs& p, uint32_t splits) {
  if (!p.halo) return false;
  const double tiles = (double)((p.rows + ROW_TILE - 1) / ROW_TILE) * p.groups, blocks = (double)((p.M + 127) / 128);
  const double limit = 9 * splits <= SMS                               ? 5.6 - 5e-6 * p.cin * p.cout * splits
                       : 3 * splits >= SMS && p.w % 8 && p.cin < 64 ? 3.0
                                                                     : 4.1;
  return tiles > limit * blocks;
}

}  // namespace
}  // namespace wt
