// Which of the split-precision mover's two gathers a launch takes; both give a
// particle the same bits.
#pragma once

#include <cmath>
#include <cstdint>

namespace gpat {

struct GatherLoad {
    int ndim;
    bool two_frames;
    int64_t n;         // particles of the launch
    double cells;      // of the run's grid
    double per_cell;   // particles of the run per cell
    double step;       // what diffusion along B moves a particle in a longest step, in cells
    int sm_count;
    double pushes;     // of a particle in the launch, at most
};

// Above half a cell the step's diffusion limit shortens it to that.  Where kappa rises
// with p, as p^(4/3) or so, twice what it is at p0: particles of sqrt(10) p0.
inline double gather_step(int ndim, double kpara0, bool kappa_rises, double dt_max, double dx,
                          double dy, double dz) {
    double h = std::fmin(dx, dy);
    if (ndim == 3) h = std::fmin(h, dz);
    const double step = std::sqrt(2.0 * std::fabs(kpara0) * dt_max) / h;
    return kappa_rises ? 2.0 * step : step;
}

// Whether particles end their pushes outside the box's cells often (MixedConsts::
// all_bounds): 2D 64^2, skipping the boundary test inside them over not skipping it,
// steps of 0.1 and less 0.94, 0.3 1.1 to 1.3.
inline int long_steps(double step) { return step >= 0.2; }

// Gathering by groups of lanes spares the L1 data pipe, and costs shuffles and
// weights computed twice (2D) or a turn through shared memory (3D).  It gains
// where that pipe is the bound: two frames, records that neighbouring lanes do not
// share.  Binned by cell they share them while the particles have moved less than
// some cells since, and where many particles stand in a cell.  Time of an interval
// of 200 to 300 pushes by single lanes over that by groups:
//   2D, one frame: 64^2 to 1024^2 cells, 2 to 128 a cell, step up to 0.3: 0.84 to
//     0.93; half a cell: 64^2 1.04 to 1.1, 256^2 and 512^2 0.85 (0.1 a cell) to 1.02,
//     1024^2 and 2048^2 1.03 to 1.27, and for sets that stand together, as those
//     injected at a shock do, 1.1 (3e4 on 512^2, 1e5 on 512 x 64); below one a cell on
//     1024^2 and 2048^2 at any step 1.0 to 1.27, on 256^2 and 512^2 0.9 to 1.0.
//   2D, two frames, 8 a cell: step 0.03 0.9, 0.1 0.96, 0.3 0.98 to 1.2, half a cell
//     1.26 to 1.4; 0.5 a cell: 1.0 to 1.5 at any step.
//   2D, 100 to 9000 particles, which leave each scheduler a warp that waits for its
//     own chain of operations: 0.75 to 0.83 (one frame), 0.74 to 0.9 (two); where dt_max
//     is far above the diffusion limit (steps of 2 cells and more by it), from 2500
//     particles on 1.08 to 1.2.
//   3D, one frame: step 0.03, 0.5 to 32 a cell: 0.78 to 0.98; step 0.1, 0.5 and 2 a
//     cell: 0.9 to 1.01, 8 and 32: 1.11 to 1.17; step 0.3: 1.0 to 1.07; half a cell
//     1.1 to 1.3; 0.1 a cell: 0.92 to 1.17.
//   3D, two frames: step 0.003: 0.77 to 0.96; 0.03, 0.5 and 2 a cell: 0.77 to 0.94, 8
//     and 32: 1.06 to 1.11; 0.1: 1.0 to 1.35; 0.3: 1.05 to 1.3; 0.1 a cell 1.04 to 1.4.
inline bool gathers_in_groups(const GatherLoad &g) {
    const double per_cell = g.per_cell;
    const bool few = g.pushes <= 16.0;
    if (g.ndim == 2) {
        if (few) return false;
        if (2 * g.n <= (int64_t)g.sm_count * 128)
            return g.step >= 2.0 && 8 * g.n > (int64_t)g.sm_count * 128;
        if (g.two_frames) return per_cell < 1.0 || g.step >= 0.25;
        if (g.step >= 0.45) return true;
        return per_cell < 1.0 && g.cells >= 4e5;
    }
    // a launch that leaves a particle a whole group of lanes (spread_of)
    if (2 * g.n <= (int64_t)g.sm_count * 128 * 4) return true;
    if (few) return false;
    if (per_cell < 0.3) return true;
    if (g.two_frames) return g.step >= (per_cell < 4.0 ? 0.06 : 0.015);
    return g.step >= (per_cell < 4.0 ? 0.12 : 0.06);
}

}  // namespace gpat
