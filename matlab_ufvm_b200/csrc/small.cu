// small.cu -- smoother calls and AMG cycles of small levels in one thread block.
//
//   smoother loop  solve/cfdSolveAlgebraicSystem.m:11-66
//   cycles         solve/AMG/cfdApplyAMG.m:27-52, cfdRestrict.m, cfdProlongate.m
//
// On a level of a few thousand rows a smoother call is a handful of microsecond kernels, and an AMG
// cycle a few dozen of those calls: launches, and waits of the host for each call's stopping test,
// were nearly all of its time (20 x 20 cavity: 5.9 ms for a p solve whose sweeps take under 0.5 ms).
// Here one block runs a whole list of operations, stopping tests included; on a case whose finest
// level is small, the list is the AMG solve. The sweeps are the wavefront passes of wave.cu on one
// chunk, and every row evaluates the same expressions in the same order; only sum |r|, which the
// stopping tests compare, is added up in another order than the multi-block kernels'.
//
// The bound on kSmallRows: the residual of n rows costs one block about n / 512 dependent loads
// (1.5 us each) against 4.5 us for a launch over all SMs, and the sweeps take one block either way.
#include "small.cuh"

#include "wave.cuh"

namespace ufvm {

namespace {

constexpr int kSmallWarps = 16, kSmallBlock = 32 * kSmallWarps;

struct SmallShared {
  double xs[kSmallRows + 1], red[32];
  unsigned long long turn[2][kSmallWarps];
  int dead;
  double sum;
  WaveArgs a;
};

// r = b - A x (x in shared memory), sum |r| over the block
__device__ double small_residual(const SmallLev& L, SmallShared& S) {
  double v = 0.0;
  for (int i = threadIdx.x; i < L.n; i += kSmallBlock) {
    const int k0 = L.rp[i], k1 = L.rp[i + 1];
    double ri = L.bc[i] - L.ac[i] * S.xs[i];
    for (int k = k0; k < k1; k += 8) {
      double p[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) p[t] = k + t < k1 ? L.anb[k + t] * S.xs[L.col[k + t]] : 0.0;
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (k + t < k1) ri = ri - p[t];
    }
    L.r[i] = ri;
    v = v + fabs(ri);
  }
  v = block_reduce<0>(v, S.red);
  if (threadIdx.x == 0) S.sum = v;
  __syncthreads();
  return S.sum;
}

// A forward and a backward pass (or the factorisation) of width class WP
template <int WP, int WIDE>
__device__ __noinline__ void small_passes(SmallShared& S, int sweep) {
  if (threadIdx.x < 2 * kSmallWarps) mb_init(&S.turn[threadIdx.x / kSmallWarps][threadIdx.x % kSmallWarps]);
  __syncthreads();
  if (sweep == 0) {
    wave_pass<OP_GS_FWD, WP, kSmallWarps, true, WIDE>(S.a, S.a.f, 0, S.xs, S.turn[0], &S.dead);
    wave_pass<OP_GS_BWD, WP, kSmallWarps, true, WIDE>(S.a, S.a.b, 0, S.xs, S.turn[1], &S.dead);
  } else if (sweep == 1) {
    wave_pass<OP_FACT, WP, kSmallWarps, true, WIDE>(S.a, S.a.f, 0, S.xs, S.turn[0], &S.dead);
  } else {
    wave_pass<OP_ILU_FWD, WP, kSmallWarps, true, WIDE>(S.a, S.a.f, 0, S.xs, S.turn[0], &S.dead);
    wave_pass<OP_ILU_BWD, WP, kSmallWarps, true, WIDE>(S.a, S.a.b, 0, S.xs, S.turn[1], &S.dead);
  }
  if (threadIdx.x < 2 * kSmallWarps)  // ready to be initialised again
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(
                     sm_addr(&S.turn[threadIdx.x / kSmallWarps][threadIdx.x % kSmallWarps]))
                 : "memory");
  __syncthreads();
}

__device__ void small_sweep(const SmallLev& L, SmallShared& S, int sweep) {
  if (L.width <= 6) small_passes<6, 0>(S, sweep);
  else if (L.width <= 10) small_passes<10, 0>(S, sweep);
  else if (L.width <= kWideRows) small_passes<16, 1>(S, sweep);
  else small_passes<16, 2>(S, sweep);
}

__device__ void small_args(const SmallLev& L, SmallShared& S, const SmallProg& p) {
  if (threadIdx.x == 0) {
    WaveArgs a{};
    a.n = L.n; a.chunks = 1; a.B = L.n; a.quirks = p.quirks;
    a.rp = L.rp; a.col = L.col; a.tpos = L.tpos; a.lord = L.lord;
    a.ac = L.ac; a.anb = L.anb; a.bc = L.bc;
    a.x = L.x; a.dc = L.dc; a.rc = L.rc; a.res = L.r;
    a.err = p.err;
    a.f = L.f; a.b = L.b;
    S.a = a;
    S.xs[L.n] = 1.0;
  }
  __syncthreads();
}

// one symmetric multicolour sweep (x in shared memory); the backward pass skips the repeated colour
__device__ void small_mc(const SmallLev& L, SmallShared& S) {
  for (int pass = 0; pass < 2; ++pass)
    for (int q = pass; q < L.ncolor; ++q) {
      const int c = pass == 0 ? q : L.ncolor - 1 - q;
      for (int p = L.colorStart[c] + (int)threadIdx.x; p < L.colorStart[c + 1]; p += kSmallBlock) {
        const int i = L.mcRow[p];
        double v = L.bc[i];
        for (int k = 0; k < L.mcW; k += 4) {
          int j[4];
          double w[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const bool in = k + t < L.mcW;
            j[t] = in ? L.mcCol[(size_t)(k + t) * L.n + p] : -1;
            w[t] = in ? L.mcAnb[(size_t)(k + t) * L.n + p] : 0.0;
          }
#pragma unroll
          for (int t = 0; t < 4; ++t)
            if (j[t] >= 0) v = v - w[t] * S.xs[j[t]];
          if (j[3] < 0) break;
        }
        S.xs[i] = v / L.mcAc[p];
      }
      __syncthreads();
    }
}

struct SmallResult {
  double r0, r1, sum;
  int iters;
};

__device__ SmallResult small_smooth_level(const SmallLev& L, SmallShared& S, const SmallProg& p, int n_iter,
                                          double rrf) {
  for (int i = threadIdx.x; i < L.n; i += kSmallBlock) S.xs[i] = L.x[i];
  __syncthreads();
  SmallResult R;
  R.sum = small_residual(L, S);
  R.r0 = R.r1 = R.sum / L.n;
  R.iters = 0;
  if (p.smoother != UFVM_SMOOTHER_MCGS) small_args(L, S, p);
  while (R.iters < n_iter && R.r1 > rrf * R.r0) {
    if (p.smoother == UFVM_SMOOTHER_ILU) {
      // the passes keep their own values in xs and update x in global memory
      small_sweep(L, S, 2);
      for (int i = threadIdx.x; i < L.n; i += kSmallBlock) S.xs[i] = L.x[i];
    } else if (p.smoother == UFVM_SMOOTHER_SOR) {
      small_sweep(L, S, 0);
    } else {
      small_mc(L, S);
    }
    __syncthreads();
    R.sum = small_residual(L, S);
    R.r1 = R.sum / L.n;
    ++R.iters;
  }
  if (p.smoother != UFVM_SMOOTHER_ILU)
    for (int i = threadIdx.x; i < L.n; i += kSmallBlock) L.x[i] = S.xs[i];
  __syncthreads();
  return R;
}

__global__ void __launch_bounds__(kSmallBlock, 1) k_small_ops(const __grid_constant__ SmallProg p) {
  __shared__ SmallShared S;
  if (threadIdx.x == 0) S.dead = 0;
  __syncthreads();
  SmallResult R{};
  auto run = [&](int from, int to) {
    for (int q = from; q < to; ++q) {
      const SmallOp& o = p.op[q];
      const SmallLev& L = p.lev[o.lev];
      if (o.type == SMALL_FACTOR) {
        small_args(L, S, p);
        small_sweep(L, S, 1);
      } else if (o.type == SMALL_SMOOTH) {
        R = small_smooth_level(L, S, p, o.iters, o.rrf);
      } else if (o.type == SMALL_PROLONG) {
        const SmallLev& F = p.lev[o.lev - 1];
        for (int i = threadIdx.x; i < F.n; i += kSmallBlock) F.x[i] = F.x[i] + L.x[F.parents[i]];
        __syncthreads();
      } else {
        const SmallLev& C = p.lev[o.lev + 1];
        for (int P = threadIdx.x; P < C.n; P += kSmallBlock) {
          double v = 0.0;
          for (int k = L.childStart[P]; k < L.childStart[P + 1]; ++k) v = v + L.r[L.child[k]];
          C.bc[P] = v;
          if (o.type == SMALL_RESTRICT) C.x[P] = 0.0;
        }
        __syncthreads();
      }
    }
  };
  run(0, p.pre);
  double init = 0.0;
  int cycles = 0;
  if (p.max_cycles > 0) {
    const SmallLev& L = p.lev[0];
    for (int i = threadIdx.x; i < L.n; i += kSmallBlock) S.xs[i] = L.x[i];
    __syncthreads();
    init = R.sum = small_residual(L, S);
    while (cycles < p.max_cycles && R.sum > p.rrf * init) {
      run(p.pre, p.nops);
      ++cycles;
    }
  } else {
    run(p.pre, p.nops);
  }
  if (threadIdx.x == 0) {
    SmoothCtl& c = *p.ctl;
    c.r0 = R.r0; c.r1 = R.r1; c.sum = R.sum; c.init = init;
    c.iters = R.iters; c.active = 0; c.cycles = cycles;
  }
}

}  // namespace

int small_describe(LinCtx& c, Level& L, const Level* next, int smoother, SmallLev& out) {
  UFVM_CHECK(dalloc(L.r, L.n));
  out = SmallLev{};
  if (smoother == UFVM_SMOOTHER_ILU) {
    UFVM_CHECK(wave_prepare_ilu(c, L, out.f, out.b));
    out.width = std::max(L.waveW[1], L.waveW[2]);
  } else if (smoother == UFVM_SMOOTHER_SOR) {
    UFVM_CHECK(wave_prepare_gs(c, L, out.f, out.b));
    out.width = L.waveW[0];
  } else {
    UFVM_CHECK(mcgs_prepare(c, L));
    out.ncolor = L.ncolor; out.mcW = L.mcW;
    out.mcRow = L.mcRow.p; out.mcCol = L.mcCol.p; out.mcAnb = L.mcAnb.p; out.mcAc = L.mcAc.p;
    out.colorStart = L.colorStart.p;
  }
  out.n = L.n;
  out.rp = L.rowptr.p; out.col = L.col.p; out.tpos = L.tpos.p; out.lord = L.lord.p;
  out.ac = L.ac.p; out.anb = L.anb.p; out.bc = L.bc.p; out.x = L.dphi.p; out.r = L.r.p;
  out.dc = L.dc.p; out.rc = L.rc.p;
  if (next) {
    out.nc = next->n;
    out.parents = L.parents.p; out.childStart = L.childStart.p; out.child = L.child.p;
  }
  return UFVM_OK;
}

int small_run(LinCtx& c, const SmallProg& p) {
  k_small_ops<<<1, kSmallBlock, 0, c.stream>>>(p);
  UFVM_LAUNCH_CHECK();
  return UFVM_OK;
}

// One smoother call on a single small level.
int small_smooth(LinCtx& c, Level& L, int smoother, int n_iter, double rrf, int quirks) {
  SmallLev d;
  UFVM_CHECK(small_describe(c, L, nullptr, smoother, d));
  UFVM_CHECK(dalloc(c.small, 1));
  UFVM_CUDA(cudaMemcpyAsync(c.small.p, &d, sizeof(d), cudaMemcpyHostToDevice, c.stream));
  SmallProg p{};
  p.lev = c.small.p;
  p.ctl = c.ctl.p;
  p.err = c.berr.p;
  p.smoother = smoother;
  p.quirks = quirks;
  if (smoother == UFVM_SMOOTHER_ILU) p.op[p.nops++] = SmallOp{SMALL_FACTOR, 0, 0, 0.0};
  p.op[p.nops++] = SmallOp{SMALL_SMOOTH, 0, n_iter, rrf};
  return small_run(c, p);
}

}  // namespace ufvm
