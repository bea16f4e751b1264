// step_pair.h -- host interface of the two-step kernels (step_pair.cuh).
#pragma once
#include "step_params.h"

namespace mrlbm {

// Rectangle of nodes x0..x1, y0..y1 (empty: x0 > x1).
struct PairRect { int x0, x1, y0, y1; };

// How one case's time steps are taken in pairs (step_pair.cuh).  `core` holds the nodes around the
// cylinder that are not stepped by the two-step tiles (its box and the nodes next to it); `halo` the
// nodes whose intermediate level those need (around them, and around every bilinear stencil node).
// The rows between the edges are cut into `chunks` chunks of equal height (to one row).
struct PairPlan {
    PairRect core, halo;
    int chunks;
};

// Columns of a strip whose level n + 2 a warp stores: all but the outermost lanes', whose neighbours'
// level n + 1 is another strip's.
constexpr int PAIR_COLS = 30;
// Strips a block steps side by side (warps x strips per warp), per precision, and the columns of its
// tensor copies: the strips, one column on either side for level n + 1 and one more for level n.
constexpr int PAIR_STRIPS64 = 4, PAIR_STRIPS32 = 8;
constexpr int PAIR_MINB = 4;                        // resident blocks per SM
constexpr int pair_box_cols(int strips) { return PAIR_COLS * strips + 4; }

// Lattices the pair kernels take: the strips on both sides must leave nodes between them.
constexpr int PAIR_MIN_NX = 12, PAIR_MIN_NY = 12;

// Chunks of rows for a lattice on which `resident` blocks run at once.  A block of height h takes about
// h + 3 row times (two more rows at the first level, and its start); all of them together that over
// `resident`, plus the last ones' tail of most of a block.  Low chunks repeat more rows, high ones
// leave a longer tail: of 6, 8, 12, 16 and 24 rows 2048 x 512 takes 20.1, 20.2, 20.9, 22.5 and 24.7 us per FP64
// step, 4099 x 1023 64.7, 62.9, 61.8, 62.3 and 64.0 us, and the estimate picks 8 and 16.
inline int pair_chunks(int nx, int ny, int strips_per_block, int resident) {
    const int bx = ((nx - 4 + PAIR_COLS - 1) / PAIR_COLS + strips_per_block - 1) / strips_per_block, n = ny - 4;
    int best = 1;
    long long best_t = -1;
    for (int h = 4; h <= 32; ++h) {
        const int chunks = (n + h - 1) / h;
        const long long t = (10ll * bx * chunks + 7ll * resident) * (h + 3);
        if (best_t < 0 || t < best_t) { best_t = t; best = chunks; }
    }
    return best;
}

// Two steps: p1 describes the first (src: level n, dst: the intermediate level's buffer, of which
// only the nodes the second step's auxiliary launch reads are written), p2 the second (src: that
// buffer, dst: level n + 2).  Two launches.  `flip`: walk the chunks of rows from the last to the
// first.  Returns 0, or -1 on a launch error.
int launch_pair_f64(const StepParams<double>& p1, const StepParams<double>& p2, const PairPlan& plan, bool flip, void* stream);
int launch_pair_f32(const StepParams<float>& p1, const StepParams<float>& p2, const PairPlan& plan, bool flip, void* stream);
constexpr int PAIR_LAUNCHES = 2;

}  // namespace mrlbm
