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
int wave_gs(LinCtx& c, Level& L);                       // one symmetric Gauss-Seidel sweep
int wave_ilu_factor(LinCtx& c, Level& L, int quirks);   // dc = inverted DILU diagonal
int wave_ilu(LinCtx& c, Level& L);                      // forward and backward substitution, x update
int wave_check(LinCtx& c);                              // error if a bounded wait of a sweep gave up

}  // namespace ufvm
