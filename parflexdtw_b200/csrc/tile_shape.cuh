// How a single tile with full outputs runs (pfx_flexdtw_tile): the rules alone,
// plain C++, compiled on the host too.
#pragma once
#include <stdint.h>

namespace pfx {

// Whether the tile goes to the cluster kernel (launch_tile_full) rather than
// to the one-CTA kernel (launch_stage1).
//
// Standard steps: from the size where the cluster pays for the two extra
// passes (kernels of one CTA and of the cluster: 64 x 64 0.095 and 0.089 ms, 100 x 100
// 0.16 and 0.12, 300 x 310 0.49 and 0.25, 1500 x 1801 10.1 and 1.06), and not
// where the tile is a ribbon of a few rows or columns (3000 x 2 1.79 and 1.87, 30
// x 3000 2.03 and 1.45, 3000 x 30 2.82 and 1.10).
//
// Other step sets take the careful loop, a step of which takes the cluster
// longer than a step of the one CTA, so the cluster has to need fewer by a
// factor: 1.1 with one step, 1.6 with two or three in another order. The
// one CTA walks W columns per 256 rows, and R more until its last strip starts;
// cluster_steps is the cluster's number (stage1_model_steps). Measured, three
// steps / two / one: 300 x 310 (1.1 times) 0.56 and 0.95 / 0.46 and 0.74 / 0.34
// and 0.44 ms; 1000 x 300 (1.0) 1.33 and 2.16 / 1.10 and 1.68 / 0.89 and 1.01; 700 x
// 600 (1.3) 1.90 and 2.01 / 1.63 and 1.56 / 1.26 and 0.90; 300 x 3000 (1.8) 4.97 and
// 4.84 / 4.14 and 3.79 / 3.08 and 2.29; 1000 x 1000 (1.8) 4.08 and 3.10 / 3.40 and
// 2.40 / 2.80 and 1.38; 1500 x 1801 (2.7) 11.3 and 5.08 / 9.71 and 3.94 / 8.27 and
// 2.28.
inline bool full_tile_on_cluster(int32_t R, int32_t W, int steps, bool std_steps,
                                 double cluster_steps) {
    if ((R < W ? R : W) < 16 || (int64_t)R * W < 4096) return false;
    if (std_steps) return true;
    const double one = (double)W * ((R + 255) / 256) + R;
    return one >= (steps == 1 ? 1.1 : 1.6) * cluster_steps;
}

// CTAs of cw warps for a tile of `strips` strips: a warp per strip up to 8
// CTAs, or as many (a power of two) as can be resident together here: fits(n)
// says whether a cluster of n can. 0: none can.
template <typename F>
inline int full_tile_ctas(int strips, int cw, F fits) {
    int cn = 1;
    while (cn < 8 && cn * cw < strips) cn *= 2;
    while (cn > 0 && !fits(cn)) cn /= 2;
    return cn;
}

}  // namespace pfx
