// linsolve.cuh -- matrix-level operations on cconn-ordered CSR levels.
#pragma once
#include "case.cuh"

namespace ufvm {

// Names a stretch of work in which every level's matrix stays the same (see LinCtx::factor_epoch);
// inside another one it changes nothing.
struct EpochScope {
  LinCtx& c;
  const bool own;
  explicit EpochScope(LinCtx& ctx);
  ~EpochScope() {
    if (own) c.factor_epoch = 0;
  }
  EpochScope(const EpochScope&) = delete;
  EpochScope& operator=(const EpochScope&) = delete;
};

int scan_exclusive(LinCtx& c, const int* in, int* out, int n, int* total_host);
int residual(LinCtx& c, const Level& L, const double* x, double* r);
int sum_abs_residual(LinCtx& c, Level& L, double* out_host);  // r kept in L.r
int read_ctl(LinCtx& c, SmoothCtl* out);             // waits for the stream; error if a bounded wait gave up
int build_schedule(LinCtx& c, Level& L);
int build_coloring(LinCtx& c, Level& L);
int check_barrier(LinCtx& c);                        // error if a bounded wait of a sweep gave up
int gs_sweep(LinCtx& c, Level& L);                   // natural-order symmetric GS
int mcgs_prepare(LinCtx& c, Level& L);               // colour-major copy of the matrix and rhs
// multicolour symmetric GS (after mcgs_prepare); ctl as for the wavefront sweeps
int mcgs_sweep(LinCtx& c, Level& L, const SmoothCtl* ctl);
int ilu_factor(LinCtx& c, Level& L, int quirks);     // dc = DILU diagonal inverse
int ilu_sweep(LinCtx& c, Level& L);                  // one cfdSolveILU application
int solve_algebraic_system(LinCtx& c, Level& L, int smoother, int n_iter, double rrf, int quirks,
                           double* r0, double* r1, int* iters);
int restrict_residual(LinCtx& c, Level& F, Level& C);  // C.bc[P] = sum over F's children of P of F.r
int prolong(LinCtx& c, Level& F, const Level& C);      // F.dphi += C.dphi[parents]

}  // namespace ufvm
