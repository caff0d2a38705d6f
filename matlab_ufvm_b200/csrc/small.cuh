// small.cuh -- smoother calls and AMG cycles on levels that one thread block handles.
#pragma once
#include "linsolve.cuh"
#include "wave_dev.cuh"

namespace ufvm {

// A level of at most kSmallRows rows is smoothed, restricted and prolongated by one block, and a run
// of such operations is one launch.
constexpr int kSmallRows = 2048;
inline bool small_level(const Level& L) { return L.n <= kSmallRows; }

// One level of the small-level kernel: its matrix and vectors, the prepared smoother, and the maps to
// the next coarser level.
struct SmallLev {
  int n, nc, width, ncolor, mcW;
  const int *rp, *col, *tpos, *lord, *parents, *childStart, *child, *mcRow, *mcCol, *colorStart;
  const double *ac, *anb, *mcAnb, *mcAc;
  double *bc, *x, *r, *dc, *rc;
  PassArgs f, b;
};

enum { SMALL_FACTOR = 0, SMALL_SMOOTH = 1, SMALL_RESTRICT = 2, SMALL_RESTRICT_KEEP = 3, SMALL_PROLONG = 4 };
struct SmallOp {
  int type, lev, iters;  // RESTRICT: lev -> lev + 1 (KEEP: the coarse correction is not cleared); PROLONG: lev -> lev - 1
  double rrf;
};
constexpr int kSmallOps = 160;
struct SmallProg {
  const SmallLev* lev;
  SmoothCtl* ctl;
  int* err;
  int smoother, quirks, nops, pre, max_cycles;  // ops [0, pre) run once; max_cycles > 0: the rest is one AMG cycle
  double rrf;                                   // AMG termination
  SmallOp op[kSmallOps];
};

int small_describe(LinCtx& c, Level& L, const Level* next, int smoother, SmallLev& out);
int small_run(LinCtx& c, const SmallProg& p);
int small_smooth(LinCtx& c, Level& L, int smoother, int n_iter, double rrf, int quirks);

}  // namespace ufvm
