// Evaluates the host's plan of the weight gradient (wt_conv_plan.h) for every channel
// count, row width and number of splits, and prints: plans, plans over a block's shared
// memory, plans over the tensor memory, the MMA's N or the tables' K steps.
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
          }
  printf("%ld %ld %ld\n", plans, memory, limits);
}
