// wave.cuh -- chunked wavefront schedules for the natural-order sweeps (Gauss-Seidel, DILU).
#pragma once
#include "case.cuh"

namespace ufvm {

// Chunks of a level of n rows on nsm SMs: contiguous row ranges of `rows` rows each (the last
// may be shorter), at most one chunk per SM.
struct WaveShape {
  int chunks = 1, rows = 1;
};
WaveShape wave_shape(int n, int nsm);

int wave_build(LinCtx& c, Level& L);                    // schedules of both directions (once per pattern)
// One symmetric Gauss-Seidel sweep. ctl: null, or the smoother call the sweep belongs to.
int wave_gs(LinCtx& c, Level& L, const SmoothCtl* ctl);
int wave_ilu_factor(LinCtx& c, Level& L, int quirks);   // dc = inverted DILU diagonal
// Forward and backward substitution of the residual L.r, x update.
int wave_ilu(LinCtx& c, Level& L, const SmoothCtl* ctl);
// Schedules and ELL copies of a one-chunk level for the small-level kernel.
int wave_prepare_gs(LinCtx& c, Level& L, struct PassArgs& f, struct PassArgs& b);
int wave_prepare_ilu(LinCtx& c, Level& L, struct PassArgs& f, struct PassArgs& b);
int wave_check(LinCtx& c);                              // error if a bounded wait of a sweep gave up

}  // namespace ufvm
