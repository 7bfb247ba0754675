// How the weight-gradient kernel (ctl_train.cuh) shares out a batch: CTAs per
// layer and accumulation chains per CTA.  Plain C++, also for the host.
#pragma once

#include <algorithm>

#ifdef __CUDACC__
#define CTL_HD __host__ __device__
#else
#define CTL_HD
#endif

namespace ctl {
namespace mlp {

constexpr int TR_L = 5;  // layers

// Accumulators of a layer that fit into TMEM, each one chain of MMAs: four of
// layer 0 (64 columns), two of the last (128 rows).
CTL_HD constexpr int wg_chains(int l) { return l == 0 ? 4 : l == TR_L - 1 ? 2 : 1; }

// 128-row tiles in a chain, at most: 512 rows, or 1/64 of a batch of 40,960
// rows or more (where the split-K GEMM with its 64 splits had chains of 1/64
// too).  A CTA gives each chain its share of its tiles, rounded up.
inline int wg_chain_tiles(int tiles) { return std::max(4, tiles / 64); }

// CTAs of layer l by the layer's MMA time per 128 rows (layer 0: a quarter of
// the columns; the last: half the rows), one per SM in all; more where that
// would make the chains longer.
inline int wg_ctas(int l, int tiles, int sms) {
    const double cost = l == 0 ? 0.35 : l == TR_L - 1 ? 0.5 : 1.0;  // 3.85 in all
    const int most = wg_chain_tiles(tiles) * wg_chains(l);
    return std::max(1, std::min(tiles, std::max((int)(sms * cost / 3.85), (tiles + most - 1) / most)));
}

}  // namespace mlp
}  // namespace ctl
