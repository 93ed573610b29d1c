// Evaluates the host's plans of the convolutions (wt_conv_plan.h) for every channel
// count, row width and number of splits, and prints: plans, plans over a block's shared
// memory, plans over another limit (tensor memory, the MMA's N, the tables' K steps, the
// rows' table, the weight ring).
#include <initializer_list>
#include <stdio.h>

#include "wt_conv_plan.h"

using namespace wt;

int main() {
  long plans = 0, memory = 0, limits = 0;
  for (uint32_t taps : {27u, 1u})
    for (uint32_t cin = 8; cin <= 128; cin += 8)
      for (uint32_t cout = 8; cout <= 128; cout += 8)
        for (uint32_t w = 1; w <= 140; w++)
          for (uint32_t splits = 1; splits <= WGRAD_SPLITS_MAX; splits++) {
            const uint32_t h = (uint32_t)(((uint64_t)(splits - 1) * 4096 + w) / w);  // the least that takes these splits
            if (wgrad_splits((uint64_t)h * w) != splits) continue;
            const wt_conv_shape s = {1, 1, h, w, cin, cout, taps};
            WgradArgs p = {};
            uint32_t nm = 0, smem = 0;
            if (!plan_wgrad(s, splits, p, nm, smem)) limits++;
            plans++;
            memory += smem > SMEM_MAX;
            limits += p.cols > 512 || p.n > 256 || (p.rt * p.xg + 1) / 2 > WG_STEPS || p.nbuf < 2 || p.nbuf > WG_BUFS;
            for (bool forward : {true, false}) {
              RowArgs r = {};
              RowPlan q = {};
              if (!plan_rows(s, forward, r, q)) limits++;
              plans++;
              memory += q.smem > SMEM_MAX;
              limits += q.xg * r.nt > 512 || r.nt % 16 || r.nt > 128 || r.nt * q.nblocks < r.N || r.nrows > ROW_ROWS ||
                        r.depth < 3 || r.depth > ROW_DEPTH_MAX;
            }
          }
  printf("%ld %ld %ld\n", plans, memory, limits);
  // numbered rows beyond 31 bits, and rows that fill an eighth or less of a tile: gathered
  long gathered = 0;
  const wt_conv_shape wide[] = {{1u << 29, 1, 1, 1, 8, 8, 27}, {1u << 29, 1, 1, 3, 8, 8, 27}, {1, 46340, 46340, 1, 8, 16, 27},
                                {1, 1, (1u << 31) - 2, 1, 8, 8, 27}, {65536, 1, 1, 1, 128, 128, 27}, {65536, 1, 1, 1, 16, 16, 27}};
  for (const wt_conv_shape& s : wide) {
    const uint32_t splits = wgrad_splits((uint64_t)s.batch * s.d * s.h * s.w);
    WgradArgs p = {};
    uint32_t nm = 0, smem = 0;
    gathered += !plan_wgrad(s, splits, p, nm, smem) || gather_is_cheaper(p, splits);
    for (bool forward : {true, false}) {
      RowArgs r = {};
      RowPlan q = {};
      gathered += !plan_rows(s, forward, r, q) || gather_is_cheaper(r, q);
    }
  }
  printf("%ld\n", gathered);
}
