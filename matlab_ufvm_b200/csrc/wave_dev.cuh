// wave_dev.cuh -- device side of the wavefront sweeps (see wave.cu for how they work): one pass over
// a chunk, used by the chunked sweeps and by the small-level kernel.
#pragma once
#include <cstdint>

#include "case.cuh"

namespace ufvm {

struct PassArgs {
  const int *rows, *scol;  // this pass's schedule and ELL copy (W entries per row)
  const int2* plev;
  const int *task, *ntask;
  int W;
  const double* sa;
  double* pub;          // values this pass publishes to other chunks
  const double* other;  // values of other chunks that this pass does not change
};

struct WaveArgs {
  int n, chunks, B, quirks;
  const int *rp, *col, *tpos, *lord;  // factorisation
  const double *ac, *anb, *bc;
  double *x, *dc, *rc;
  const double* res;  // DILU: the residual the forward substitution starts from
  const SmoothCtl* ctl;  // null, or the smoother call this sweep belongs to
  double* loc;  // chunk values in global memory, for chunks that do not fit in shared memory
  int* err;
  PassArgs f, b;
};

namespace {

constexpr int kTaskRows = 32;        // rows of a task: one warp
constexpr long long kWaitPerRow = 2048;       // SM clocks that each row of a matrix that is one chain may add to a wait
constexpr unsigned long long kNotYet = ~0ull;  // "not published" pattern (cudaMemset 0xff)

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// ---------------------------------------------------------------- sweeps
enum { OP_GS_FWD = 0, OP_GS_BWD = 1, OP_FACT = 2, OP_ILU_FWD = 3, OP_ILU_BWD = 4 };

template <bool SM>
__device__ __forceinline__ double ld_loc(const double* p) { return SM ? *p : __ldcg(p); }
template <bool SM>
__device__ __forceinline__ void st_loc(double* p, double v) { if (SM) *p = v; else __stcg(p, v); }

// The bound of a wait: err[1] is the number of rows of the largest system (see LinCtx::ensure). It is
// read here, off the chain: as a kernel argument it cost the narrow sweeps up to 16%.
__device__ __forceinline__ long long wait_limit(const int* err) { return kFlagClocks + kWaitPerRow * err[1]; }

// The published value of another chunk's row, as bits (bounded wait).
__device__ __forceinline__ unsigned long long poll(const double* pub, int j, int* s_dead, int* err) {
  const unsigned long long* p = reinterpret_cast<const unsigned long long*>(pub) + j;
  unsigned long long v = ld_relaxed(p);
  if (v == kNotYet) {
    unsigned spins = 0;
    const long long t0 = clock64(), limit = wait_limit(err);
    while (v == kNotYet) {
      if ((++spins & 255u) == 0 && (*(volatile int*)s_dead || clock64() - t0 > limit)) {
        *(volatile int*)s_dead = 1;
        atomicExch(err, 1);
        return 0;
      }
      v = ld_relaxed(p);
    }
  }
  return v;
}

__device__ __forceinline__ void publish(double* pub, int i, double v) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  if (b == kNotYet) b = 0x7ff8000000000000ull;  // a NaN either way
  st_relaxed(reinterpret_cast<unsigned long long*>(pub) + i, b);
}

// v / d, correctly rounded, from the correctly rounded reciprocal y = 1 / d, which a row has ready
// before its turn: two residual corrections q += (v - d q) y. The first leaves q within one unit
// in the last place of v / d, and from there the second gives the rounded quotient (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev.
// 34 (1990), theorem on the final step of a division). It holds while no intermediate overflows or
// loses bits to underflow: exponents of d within +-300 (quotient_rec gives NaN for any other d, so
// that the quotient below is NaN too) and of the quotient within +-400, which bounds v. A zero v
// gives the right zero. Everything else takes the division itself. One division on the chain of a
// Gauss-Seidel step is 113 cycles, this one about 45 (dependent operations, measured alone).
__device__ __forceinline__ int expo(double x) { return (int)(((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 1023; }
__device__ __forceinline__ double quotient_rec(double d) {
  return abs(expo(d)) <= 300 ? 1.0 / d : __longlong_as_double(0x7ff8000000000000ll);
}
__device__ __forceinline__ double quotient(double v, double d, double y) {
  const double q0 = v * y;  // its exponent is within one of the quotient's: judged off the chain
  const bool odd = (unsigned)((__double2hiint(q0) & 0x7fffffff) - (623 << 20)) > (800u << 20);
  double r = __fma_rn(-d, q0, v);
  double q = __fma_rn(r, y, q0);
  r = __fma_rn(-d, q, v);
  q = __fma_rn(r, y, q);
  if (odd) q = v == 0.0 && q0 == 0.0 ? q0 : v / d;
  return q;
}

// The turn passes from task to task through mbarriers (one arrival per phase; task t uses barrier
// t % G, phase t / G): about 70 cycles from the store of a value to its load in the next warp,
// against 160 with named barriers.
__device__ __forceinline__ unsigned sm_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mb_init(unsigned long long* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sm_addr(b)) : "memory");
}
__device__ __forceinline__ void mb_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sm_addr(b)) : "memory");
}
__device__ __forceinline__ bool mb_try(unsigned long long* b, unsigned parity) {
  unsigned ok;
  asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
               : "=r"(ok) : "r"(sm_addr(b)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mb_wait(unsigned long long* b, unsigned parity, int* s_dead, int* err) {
  if (mb_try(b, parity)) return;
  const long long t0 = clock64(), limit = 2 * wait_limit(err);
  while (!mb_try(b, parity)) {
    if (*(volatile int*)s_dead) return;
    if (clock64() - t0 > limit) {
      *(volatile int*)s_dead = 1;
      atomicExch(err, 1);
    }
  }
}

// The value that entry e (a place in the chunk, or -(j + 3) for row j of another one) contributes to row
// i in its turn.
template <int OP, bool SM>
__device__ __forceinline__ double row_value(const WaveArgs& a, const PassArgs& P, int base, int i, int e,
                                            const double* xs, int* s_dead) {
  constexpr bool FWD = OP == OP_GS_FWD || OP == OP_FACT || OP == OP_ILU_FWD;
  constexpr bool GS = OP == OP_GS_FWD || OP == OP_GS_BWD;
  if (e >= 0) return ld_loc<SM>(xs + e);
  const int j = -(e + 3);
  return !GS || (FWD ? j < i : j > i) ? __longlong_as_double((long long)poll(P.pub, j, s_dead, a.err))
                                      : __ldcg(P.other + j);
}

// The entries of a row that the ELL copy leaves out, from the matrix, eight loads at a time.
template <int OP, bool SM>
__device__ __noinline__ double row_rest(const WaveArgs& a, const PassArgs& P, int base, int i, const double* xs,
                                        int* s_dead, double v) {
  const int k1 = a.rp[i + 1];
  int skip = OP == OP_ILU_BWD ? P.W : 0;  // upper entries lie anywhere in the row
  for (int k = a.rp[i] + (OP == OP_ILU_BWD ? 0 : P.W); k < k1; k += 8) {
    int j[8];
    double w[8], z[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int q = k + t >= k1 ? -1 : OP == OP_ILU_FWD ? a.lord[k + t] : k + t;
      j[t] = q >= 0 ? a.col[q] : -1;
      w[t] = q >= 0 ? a.anb[q] : 0.0;
    }
    if (OP == OP_ILU_BWD) {
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (j[t] <= i || skip-- > 0) j[t] = -1;
    }
#pragma unroll
    for (int t = 0; t < 8; ++t)
      z[t] = j[t] < 0 ? 0.0
                      : row_value<OP, SM>(a, P, base, i, (unsigned)(j[t] - base) < (unsigned)a.B ? j[t] - base : -(j[t] + 3),
                                          xs, s_dead);
#pragma unroll
    for (int t = 0; t < 8; ++t)
      if (j[t] >= 0) v = v - w[t] * z[t];
  }
  return v;
}

// One pass over the CTA's chunk with G warps; `xs`: the chunk's values, and behind them (at offset
// B) the constant 1.0. Entry t of a row contributes w[t] * xs[c[t]] (times w2[t] for the
// factorisation): a coefficient and the place of a value that an earlier row of this pass
// produces, or a finished product (0.0 where the row has no entry) and the place of the 1.0 --
// multiplying by 1.0 and subtracting 0.0 change nothing, and a row's turn has no case
// distinctions. Its instructions are the chain that bounds the sweep. WIDE: 0 rows of at most WP entries,
// 1 a few more, 2 many more, and rows wider than the ELL copy. Ten Gauss-Seidel sweeps of
// 100,000 rows of 60 entries 255 ms with variant 1, 150 ms with variant 2; the small-level kernel on the
// coarse levels of 64^3 (up to 30 entries) 20 ms an iteration and 27 ms, for its spilled registers.
constexpr int kWideRows = 32;  // rows of more entries than this take variant 2
template <int OP, int WP, int G, bool SM, int WIDE>
__device__ __forceinline__ void wave_pass(const WaveArgs& a, const PassArgs& P, int chunk, double* xs,
                                          unsigned long long* turn, int* s_dead) {
  constexpr bool FWD = OP == OP_GS_FWD || OP == OP_FACT || OP == OP_ILU_FWD;
  constexpr bool GS = OP == OP_GS_FWD || OP == OP_GS_BWD;
  constexpr bool FACT = OP == OP_FACT;
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int base = chunk * a.B;
  const int nt = P.ntask[chunk];
  const int* first_pos = P.task + (size_t)chunk * (a.B + 1);
  const size_t n = (size_t)a.n;
  int p0 = g < nt ? first_pos[g] : 0, p1 = g < nt ? first_pos[g + 1] : 0;
  for (int task = g; task < nt; task += G) {
    const int p = p0 + lane;
    const bool on = p < p1;
    if (task + G < nt) { p0 = first_pos[task + G]; p1 = first_pos[task + G + 1]; }
    int i = base, k0 = 0, deg = 0;
    int2 lev = make_int2(0, 0);
    int c[WP];
    double w[WP], w2[FACT ? WP : 1];
    if (on) {
      i = P.rows[p];
      lev = P.plev[p];
    }
#pragma unroll
    for (int t = 0; t < WP; ++t) {
      c[t] = -1;
      w[t] = 0.0;
      if (!FACT && on && t < P.W) {
        c[t] = P.scol[(size_t)t * n + p];
        w[t] = P.sa[(size_t)t * n + p];
      }
    }
    double v = 0.0, d = 1.0, rec = 0.0, x0 = 0.0;
    if (on) {
      if (FACT) {
        k0 = a.rp[i];
        deg = a.rp[i + 1] - k0;
        v = a.ac[i];
      } else if (GS) {
        v = a.bc[i];
        d = a.ac[i];
      } else {
        v = OP == OP_ILU_FWD ? a.res[i] : __ldcg(a.rc + i);
        d = a.dc[i];
        if (OP == OP_ILU_BWD) x0 = a.x[i];
      }
    }
    const int l = i - base;
    if (FACT) {
#pragma unroll
      for (int t = 0; t < WP; ++t) {
        w2[FACT ? t : 0] = 0.0;
        const int q = t < deg ? a.lord[k0 + t] : -1;
        const int tk = q >= 0 ? a.tpos[q] : -1;
        const int j = q >= 0 ? a.col[q] : 0;
        // Q7: the reference's factorisation loop skips row N-1 (1-based), i.e. row n-2
        if (q >= 0 && tk >= 0 && !((a.quirks & UFVM_Q7_ILU_SKIP_ROW) && j == a.n - 2)) {
          c[t] = (unsigned)(j - base) < (unsigned)a.B ? j - base : -(j + 3);
          w[t] = a.anb[q];
          w2[FACT ? t : 0] = a.anb[tk];
        }
      }
    }
    // the task's levels: this row's among them (sub), and the last task that must be complete
    // before the first one (the tasks of one wide level do not wait for one another)
    const int below = __shfl_up_sync(0xffffffffu, lev.x, 1);
    const unsigned edges = __ballot_sync(0xffffffffu, on && lane > 0 && lev.x != below);
    const int sub = on ? __popc(edges & (0xffffffffu >> (31 - lane))) : -1, nsub = 1 + __popc(edges);
    const int after = __shfl_sync(0xffffffffu, lev.y, 0) - 1;
    // values that no row of this chunk before this one produces: those of other chunks, and of
    // rows of this chunk that are later in a Gauss-Seidel pass
    unsigned long long raw[WP];
#pragma unroll
    for (int t = 0; t < WP; ++t) {
      raw[t] = 0;
      if (c[t] <= -3) {
        const int j = -(c[t] + 3);
        const double* src = !GS || (FWD ? j < i : j > i) ? P.pub : P.other;
        raw[t] = ld_relaxed(reinterpret_cast<const unsigned long long*>(src) + j);
      } else if (GS && c[t] >= 0 && (FWD ? c[t] >= l : c[t] <= l)) {
        raw[t] = (unsigned long long)__double_as_longlong(ld_loc<SM>(xs + c[t]));
      }
    }
#pragma unroll
    for (int t = 0; t < WP; ++t) {
      bool ready = GS && c[t] >= 0 && (FWD ? c[t] >= l : c[t] <= l);
      if (c[t] <= -3) {
        const int j = -(c[t] + 3);
        ready = true;
        if (raw[t] == kNotYet && (!GS || (FWD ? j < i : j > i))) raw[t] = poll(P.pub, j, s_dead, a.err);
      }
      if (ready) {
        const double y = __longlong_as_double((long long)raw[t]);
        w[t] = FACT ? w[t] * y * w2[FACT ? t : 0] : w[t] * y;
        c[t] = -1;
      }
    }
    // the leading finished products are subtracted now
    bool lead = true;
#pragma unroll
    for (int t = 0; t < WP; ++t) {
      lead = lead && c[t] < 0;
      if (lead) {
        v = v - w[t];
        w[t] = 0.0;
      }
      if (c[t] < 0) {
        c[t] = a.B;
        if (FACT) w2[FACT ? t : 0] = 1.0;
      }
    }
    if (GS) rec = quotient_rec(d);
    __syncwarp();
    // the turn: everything up to the level before this task's first one is stored
    if (after >= 0 && after > task - G) mb_wait(turn + after % G, (after / G) & 1, s_dead, a.err);
    for (int k = 0; k < nsub; ++k) {
      if (sub == k) {
        double y[WP];
#pragma unroll
        for (int t = 0; t < WP; ++t) y[t] = ld_loc<SM>(xs + c[t]);
#pragma unroll
        for (int t = 0; t < WP; ++t) {
          const double pr = w[t] * y[t];
          v = v - (FACT ? pr * w2[FACT ? t : 0] : pr);
        }
        if (WIDE == 1 || (WIDE && FACT)) {  // entries beyond the registers
          const int more = FACT ? deg : P.W;
          for (int t = WP; t < more; ++t) {
            int e;
            double wt, wt2 = 1.0;
            if (FACT) {
              const int q = a.lord[k0 + t];
              if (q < 0) break;
              const int tk = a.tpos[q], j = a.col[q];
              if (tk < 0 || ((a.quirks & UFVM_Q7_ILU_SKIP_ROW) && j == a.n - 2)) continue;
              e = (unsigned)(j - base) < (unsigned)a.B ? j - base : -(j + 3);
              wt = a.anb[q];
              wt2 = a.anb[tk];
            } else {
              e = P.scol[(size_t)t * n + p];
              if (e == -1) break;
              wt = P.sa[(size_t)t * n + p];
            }
            const double z = row_value<OP, SM>(a, P, base, i, e, xs, s_dead);
            v = v - (FACT ? wt * z * wt2 : wt * z);
          }
        } else if (WIDE == 2) {  // eight at a time, their loads before the first use
          bool end = false;
          for (int t0 = WP; t0 < P.W && !end; t0 += 8) {
            int e[8];
            double wt[8], z[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
              e[t] = t0 + t < P.W ? P.scol[(size_t)(t0 + t) * n + p] : -1;
              wt[t] = t0 + t < P.W ? P.sa[(size_t)(t0 + t) * n + p] : 0.0;
            }
#pragma unroll
            for (int t = 0; t < 8; ++t) z[t] = e[t] == -1 ? 0.0 : row_value<OP, SM>(a, P, base, i, e[t], xs, s_dead);
#pragma unroll
            for (int t = 0; t < 8; ++t)
              if (e[t] != -1) v = v - wt[t] * z[t];
            end = e[7] == -1;
          }
          if (!end) v = row_rest<OP, SM>(a, P, base, i, xs, s_dead, v);
        }
        // what the rows of later levels read of this one
        double out;
        if (GS) out = quotient(v, d, rec);
        else if (FACT) out = 1.0 / v;
        else out = d * v;  // dc_i r_i, the product both substitutions start from
        st_loc<SM>(xs + l, out);
        if (a.chunks > 1) publish(P.pub, i, out);
        if (OP == OP_ILU_FWD) __stcg(a.rc + i, v);
        if (OP == OP_ILU_BWD) a.x[i] = x0 + out;
        if (FACT) a.dc[i] = out;
      }
      __syncwarp();
    }
    // the turn is handed on in task order, once every lane has seen it arrive (a lane that looked
    // later could find the barrier a phase further on and wait for good)
    if (after != task - 1 && task > 0) mb_wait(turn + (task - 1) % G, ((task - 1) / G) & 1, s_dead, a.err);
    __syncwarp();
    if (lane == 0) mb_arrive(turn + task % G);
  }
  __syncthreads();
}

}  // namespace
}  // namespace ufvm
