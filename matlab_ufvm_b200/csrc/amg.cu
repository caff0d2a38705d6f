// amg.cu -- agglomeration AMG: hierarchy build and V/W/F cycles.
//
//   cfdAgglomerate         solve/AMG/cfdAgglomerate.m:7-17
//   cfdAgglomerateLevel    solve/AMG/cfdAgglomerateLevel.m:13-105
//   Galerkin by summation  assemble/assembleAgglomeratedLHS.m:16-30
//   cycles / driver        solve/AMG/cfdApplyVCycle.m, cfdApplyWCycle.m, cfdApplyFCycle.m,
//                          cfdApplyAMG.m:9-57, cfdRestrict.m, cfdProlongate.m
//
// The reference agglomerates with a sequential greedy sweep over seeds in natural order: a seed
// claims itself, its strong unassigned neighbours and their strong unassigned neighbours. It is
// reproduced here exactly, in parallel rounds: every unassigned cell keeps a holder, the
// lowest-index unsettled seed that could still claim it, and a seed takes its step once it holds
// every cell its step can touch. Claims only shrink as cells get assigned, so such a seed's claims
// are the ones it would make in the sequential sweep, and the final `parents` map is identical.
// A holder stands until it is settled, so a cell looks for the next one only a few times in all,
// and a seed away from the front of the sweep costs a round one load (its own cell has another
// holder). Letting every unprocessed seed reserve its claims again in every round took 110 us a
// round on the 64^3 grid.
#include "amg.cuh"

namespace ufvm {

// largest -anb of a row, and which of its entries are strong: -anb / max > 0.5 (bit 0)
__global__ void k_strong(int n, const int* __restrict__ rp, const double* __restrict__ anb, double* maxAnb,
                         signed char* strong) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k0 = rp[i], k1 = rp[i + 1];
  double m = -INFINITY;
  for (int k = k0; k < k1; ++k) m = dmax(m, -anb[k]);
  maxAnb[i] = m;
  for (int k = k0; k < k1; ++k) strong[k] = ((-anb[k]) / m) > 0.5 ? 1 : 0;
}

// bit 1: the transposed entry is strong; *asym is raised where an entry has no transposed one
__global__ void k_strong_back(int n, const int* __restrict__ rp, const int* __restrict__ col, signed char* strong,
                              int* asym) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int k = rp[i]; k < rp[i + 1]; ++k) {
    const int j = col[k];
    int s = -1;
    for (int q = rp[j]; q < rp[j + 1]; ++q)
      if (col[q] == i) s = max(s, strong[q] & 1);
    if (s < 0) *asym = 1;
    else if (s) strong[k] |= 2;  // another thread reads bit 0 of this byte only
  }
}

namespace {

constexpr int kNoHolder = 0x7fffffff;

struct AggArgs {
  int n;
  const int *rp, *col;
  const signed char* strong;
  // each cell's incoming links (bit 1 of istrong) where the pattern is not symmetric; else its own row
  const int *irp, *icol;
  const signed char* istrong;
  int *parents, *hold, *seedflag;
  const int* asym;  // raised: the pattern is not symmetric and these rounds are left out
};

// parents: kOpen, kDone (its step found nothing to claim: it takes no step any more but can still be
// claimed) or the seed it is assigned to. A cell is settled once it is not open.
constexpr int kOpen = -1, kDone = -2;
constexpr int kAggLinks = 8;  // links whose states are loaded before any is looked at

// A round's few working cells lie together (the front of the sweep), and each takes a chain of
// dependent loads, so a block lists the cells that have work and hands them out to groups of G lanes,
// each lane looking after some of the cell's links, kAggLinks at a time. A warp that takes its own
// cells one after another spends up to 32 chains on a round. One level of the 64^3 grid, 272 rounds:
// 14.8 ms; with the lists 6.6; in one launch instead of two a round 5.8; with the links' states
// loaded together instead of one behind the other 3.8 ms. G: 8 for rows of a few entries, 32 for a
// coarse level's (a cell has several hundred second links there, and a round lasts as long as its
// slowest cell).
constexpr int kAggNarrow = 12;  // mean row length up to which groups of 8 lanes are used

template <int G>
struct AggGroup {
  int lane = threadIdx.x & (G - 1), group = threadIdx.x / G, groups = blockDim.x / G;
  unsigned mask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (threadIdx.x & 31 & ~(G - 1));
};

// The lowest unsettled seed that can claim x: x itself, a cell with a strong link to x, or one with
// a strong link to such an unassigned cell. (ONEWAY chosen at run time cost the one-block rounds 22%.)
template <int G, bool ONEWAY>
__device__ __forceinline__ int agg_holder(const AggArgs& a, int x, const AggGroup<G>& gr) {
  const int* irp = ONEWAY ? a.irp : a.rp;
  const int* icol = ONEWAY ? a.icol : a.col;
  const signed char* istrong = ONEWAY ? a.istrong : a.strong;
  int h = gr.lane == 0 && a.parents[x] == kOpen ? x : kNoHolder;
  const int end = irp[x + 1];
  for (int k = irp[x] + gr.lane; k < end; k += G) {
    if (!(istrong[k] & 2)) continue;
    const int d = icol[k], pd = a.parents[d], e = irp[d + 1];
    if (pd >= 0) continue;  // claimed: neither a seed nor a link any more
    if (pd == kOpen) h = min(h, d);
    for (int k0 = irp[d]; k0 < e; k0 += kAggLinks) {
      int t[kAggLinks], p[kAggLinks];
      bool on[kAggLinks];
#pragma unroll
      for (int q = 0; q < kAggLinks; ++q) {
        const int k2 = min(k0 + q, e - 1);
        t[q] = icol[k2];
        on[q] = istrong[k2] & 2;
      }
#pragma unroll
      for (int q = 0; q < kAggLinks; ++q) p[q] = a.parents[t[q]];
#pragma unroll
      for (int q = 0; q < kAggLinks; ++q)
        if (on[q] && p[q] == kOpen) h = min(h, t[q]);
    }
  }
  return __reduce_min_sync(gr.mask, h);
}

// First half of a round: cells whose holder is settled look for the next one.
__device__ __forceinline__ bool agg_needs_holder(const AggArgs& a, int x) {
  const int p = a.parents[x], h = a.hold[x];
  return p < 0 && h != kNoHolder && a.parents[h] != kOpen;
}

// Second half: a seed that holds all it can touch takes the sequential step
// (cfdAgglomerateLevel.m:28-64) on it. Two such seeds share no cell. A cell that another seed is
// claiming at this moment is either seen assigned already or held by that seed, which makes this one
// wait for the next round.
template <int G>
__device__ __forceinline__ void agg_step(const AggArgs& a, int U, const AggGroup<G>& gr) {
  const int lane = gr.lane, u0 = a.rp[U], u1 = a.rp[U + 1];
  bool any = false, lose = false;
  for (int k = u0 + lane; k < u1 && !lose; k += G) {
    if (!(a.strong[k] & 1)) continue;
    const int c = a.col[k], e = a.rp[c + 1];
    const int pc = __ldcg(a.parents + c), hc = a.hold[c];
    if (pc >= 0) continue;
    any = true;
    lose = hc != U;
    for (int k0 = a.rp[c]; k0 < e && !lose; k0 += kAggLinks) {
      int g[kAggLinks], p[kAggLinks], h[kAggLinks];
      bool on[kAggLinks];
#pragma unroll
      for (int q = 0; q < kAggLinks; ++q) {
        const int k2 = min(k0 + q, e - 1);
        g[q] = a.col[k2];
        on[q] = a.strong[k2] & 1;
      }
#pragma unroll
      for (int q = 0; q < kAggLinks; ++q) {
        p[q] = __ldcg(a.parents + g[q]);
        h[q] = a.hold[g[q]];
      }
#pragma unroll
      for (int q = 0; q < kAggLinks; ++q) lose |= on[q] && p[q] < 0 && h[q] != U;
    }
  }
  if (__any_sync(gr.mask, lose)) return;
  if (!__any_sync(gr.mask, any)) {
    if (lane == 0) __stcg(a.parents + U, kDone);  // single-cell aggregate: undone, it stays unassigned
    return;
  }
  if (lane == 0) {
    a.seedflag[U] = 1;
    __stcg(a.parents + U, U);
  }
  for (int k = u0 + lane; k < u1; k += G) {  // first generation
    const int c = a.col[k];
    if ((a.strong[k] & 1) && __ldcg(a.parents + c) < 0) __stcg(a.parents + c, U);
  }
  __syncwarp(gr.mask);
  for (int k = u0 + lane; k < u1; k += G) {  // second generation, from the first
    const int c = a.col[k];
    if (!(a.strong[k] & 1) || c == U || __ldcg(a.parents + c) != U) continue;
    const int e = a.rp[c + 1];
    for (int k0 = a.rp[c]; k0 < e; k0 += kAggLinks) {
      int g[kAggLinks], p[kAggLinks];
      bool on[kAggLinks];
#pragma unroll
      for (int q = 0; q < kAggLinks; ++q) {
        const int k2 = min(k0 + q, e - 1);
        g[q] = a.col[k2];
        on[q] = a.strong[k2] & 1;
      }
#pragma unroll
      for (int q = 0; q < kAggLinks; ++q) p[q] = __ldcg(a.parents + g[q]);
#pragma unroll
      for (int q = 0; q < kAggLinks; ++q)
        if (on[q] && p[q] < 0) __stcg(a.parents + g[q], U);
    }
  }
  __syncwarp(gr.mask);
}

// All rounds of a level in one cooperative launch, two grid barriers a round (about 1.3 us each, where
// a launch is 2.5 us and starts from cold registers). A warp's cells are spread over the grid, 32
// at a time, since the cells with work lie together.
constexpr int kAggBlock = 1024;
constexpr int kAggList = 8192;  // cells of a block listed at a time

struct AggBar { unsigned long long arrived, open; };

// Waits for all blocks; the returned flag says that the wait gave up. `open` is added up before.
__device__ bool agg_barrier(AggBar* bar, unsigned long long target, bool open, int* err) {
  __shared__ int dead;
  __syncthreads();
  if (threadIdx.x == 0) {
    dead = 0;
    if (open) atomicAdd(&bar->open, 1ull);
    __threadfence();
    atomicAdd(&bar->arrived, 1ull);
    const long long t0 = clock64();
    for (unsigned spins = 1; *(volatile unsigned long long*)&bar->arrived < target; ++spins)
      if ((spins & 255u) == 0 && clock64() - t0 > kFlagClocks) {
        atomicExch(err, 1);
        dead = 1;
        break;
      }
    __threadfence();
  }
  __syncthreads();
  return dead != 0;
}

template <int G, bool ONEWAY>
__global__ void __launch_bounds__(kAggBlock) k_agg_grid(AggArgs a, AggBar* bar, int* err) {
  __shared__ int list[kAggList], cnt;
  __shared__ unsigned long long open_sum;
  if (*a.asym) return;
  const AggGroup<G> gr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long per = (long long)kAggBlock * gridDim.x;  // cells of one stride over the grid
  const int strides = (int)((a.n + per - 1) / per);
  constexpr int kAtOnce = kAggList / kAggBlock;
  unsigned long long target = 0, seen = 0;
  for (int round = -1; round < a.n + 2; ++round) {  // round -1: every cell's first holder
    for (int s0 = 0; s0 < strides; s0 += kAtOnce) {
      if (threadIdx.x == 0) cnt = 0;
      __syncthreads();
      for (int s = s0; s < min(strides, s0 + kAtOnce); ++s) {
        const long long x = ((long long)(s * (kAggBlock / 32) + warp) * gridDim.x + blockIdx.x) * 32 + lane;
        if (x < a.n && (round < 0 || agg_needs_holder(a, (int)x))) list[atomicAdd(&cnt, 1)] = (int)x;
      }
      __syncthreads();
      for (int i = gr.group; i < cnt; i += gr.groups) {
        const int X = list[i], h = agg_holder<G, ONEWAY>(a, X, gr);
        if (gr.lane == 0) a.hold[X] = h;
      }
      __syncthreads();
    }
    target += gridDim.x;
    if (agg_barrier(bar, target, false, err)) return;
    bool open = false;
    for (int s0 = 0; s0 < strides; s0 += kAtOnce) {
      if (threadIdx.x == 0) cnt = 0;
      __syncthreads();
      for (int s = s0; s < min(strides, s0 + kAtOnce); ++s) {
        const long long u = ((long long)(s * (kAggBlock / 32) + warp) * gridDim.x + blockIdx.x) * 32 + lane;
        if (u < a.n && a.parents[u] == kOpen) {
          open = true;
          if (a.hold[u] == u) list[atomicAdd(&cnt, 1)] = (int)u;
        }
      }
      __syncthreads();
      for (int i = gr.group; i < cnt; i += gr.groups) agg_step(a, list[i], gr);
      __syncthreads();
    }
    open = __syncthreads_or(open);
    target += gridDim.x;
    if (agg_barrier(bar, target, open, err)) return;
    // no block adds to it again before all have passed the next barrier
    if (threadIdx.x == 0) open_sum = *(volatile unsigned long long*)&bar->open;
    __syncthreads();
    if (open_sum == seen) break;
    seen = open_sum;
    __syncthreads();
  }
}

// All rounds of a level in one block, for levels whose cells are few for the threads of a block:
// bounds of 1024, 2048 and 6000 measure within 1% of one another, 16384 up to 2% more (64^3 cavity).
// Every round settles at least the lowest unsettled seed.
constexpr int kAggOneBlock = 2048;
template <int G, bool ONEWAY>
__global__ void __launch_bounds__(kAggBlock) k_agg_rounds(AggArgs a) {
  __shared__ unsigned short list[kAggOneBlock];
  __shared__ int cnt[2];
  if (*a.asym) return;
  const AggGroup<G> gr;
  for (int x = gr.group; x < a.n; x += gr.groups) {
    const int h = agg_holder<G, ONEWAY>(a, x, gr);
    if (gr.lane == 0) a.hold[x] = h;
  }
  if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
  __syncthreads();
  for (int round = 0; round < a.n + 2; ++round) {
    for (int x = threadIdx.x; x < a.n; x += kAggBlock)
      if (agg_needs_holder(a, x)) list[atomicAdd(&cnt[0], 1)] = (unsigned short)x;
    __syncthreads();
    for (int i = gr.group; i < cnt[0]; i += gr.groups) {
      const int X = list[i], h = agg_holder<G, ONEWAY>(a, X, gr);
      if (gr.lane == 0) a.hold[X] = h;
    }
    __syncthreads();
    bool open = false;
    for (int u = threadIdx.x; u < a.n; u += kAggBlock)
      if (a.parents[u] == kOpen) {
        open = true;
        if (a.hold[u] == u) list[atomicAdd(&cnt[1], 1)] = (unsigned short)u;
      }
    if (threadIdx.x == 0) cnt[0] = 0;
    if (!__syncthreads_or(open)) break;
    for (int i = gr.group; i < cnt[1]; i += gr.groups) agg_step(a, (int)list[i], gr);
    __syncthreads();
    if (threadIdx.x == 0) cnt[1] = 0;  // read again after the next barrier only
  }
}

// A pattern that is not symmetric: a cell does not see in its own row every seed that can claim it, so
// the strong links are listed by the cell they lead to as well (in any order: a holder is a minimum).
// The sweep as it is written, on one thread, took 194 ms for 360,000 rows; this way 13 ms.
__global__ void k_in_count(int n, const int* __restrict__ rp, const int* __restrict__ col,
                           const signed char* __restrict__ strong, int* cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int k = rp[i]; k < rp[i + 1]; ++k)
    if (strong[k] & 1) atomicAdd(cnt + col[k], 1);
}

__global__ void k_in_fill(int n, const int* __restrict__ rp, const int* __restrict__ col,
                          const signed char* __restrict__ strong, const int* __restrict__ irp, int* cnt, int* icol,
                          signed char* istrong) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int k = rp[i]; k < rp[i + 1]; ++k)
    if (strong[k] & 1) {
      const int p = irp[col[k]] + atomicSub(cnt + col[k], 1) - 1;
      icol[p] = i;
      istrong[p] = 2;
    }
}

__global__ void k_unassigned(int n, const int* __restrict__ parents, int* flag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) flag[i] = parents[i] < 0;
}

constexpr int kAggGrid = 64;  // blocks of a level's orphan kernel

}  // namespace

// Orphans (cfdAgglomerateLevel.m:66-83): a cell left unassigned takes the parent of its strongest
// assigned neighbour, in natural order; orphans of lower index among its neighbours go first. An
// orphan's parents entry says that it is settled. orphan: null, or for a pattern that is not symmetric
// the cells that were unassigned at the start.
__global__ void __launch_bounds__(256) k_agg_orphans(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                                     const double* __restrict__ anb,
                                                     const double* __restrict__ maxAnb, int* parents, int* newflag,
                                                     const int* __restrict__ orphan, int* err) {
  const int nth = gridDim.x * blockDim.x;
  int o = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned spins = 0;
  long long t0 = clock64();
  while (__any_sync(0xffffffffu, o < n)) {
    if (o < n) {
      bool wait = false;
      if (ld_flag(parents + o) < 0) {
        for (int k = rp[o]; k < rp[o + 1] && !wait; ++k) wait = col[k] < o && ld_flag(parents + col[k]) < 0;
        if (!wait) {
          double strength = 0.0;
          int par = -1;
          for (int k = rp[o]; k < rp[o + 1]; ++k) {
            const int nb = col[k];
            const int pn = ld_flag(parents + nb);
            // an orphan of higher index has not been attached yet in the sequential sweep either:
            // it waits for this one, if it has the entry for that
            if (pn >= 0 && !(orphan && nb > o && orphan[nb])) {
              const double sv = (-anb[k]) / maxAnb[nb];
              if (strength < sv) { strength = sv; par = pn; }
            }
          }
          if (par == -1) { par = n + o; newflag[o] = 1; }
          st_flag(parents + o, par);
        }
      }
      if (!wait) {
        o += nth;
        t0 = clock64();
      } else if ((++spins & 255u) == 0 && clock64() - t0 > kFlagClocks) {
        atomicExch(err, 1);
        o = n;
      }
    }
    __syncwarp();
  }
}

// id < n: the seed id; id - n: an orphan of its own (rank: exclusive scan of the seeds' flags, then
// the orphans')
__global__ void k_relabel(int n, const int* __restrict__ rank, int* parents) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) parents[i] = rank[parents[i]];
}

__global__ void k_count_children(int n, const int* __restrict__ parents, int* cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicAdd(cnt + parents[i], 1);
}

__global__ void k_fill_children(int n, const int* __restrict__ parents, int* cur, int* child) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) child[atomicAdd(cur + parents[i], 1)] = i;
}

__global__ void k_sort_children(int nc, const int* __restrict__ cs, int* child) {
  const int P = blockIdx.x * blockDim.x + threadIdx.x;
  if (P >= nc) return;
  const int a = cs[P], b = cs[P + 1];
  for (int q = a + 1; q < b; ++q) {
    const int v = child[q];
    int r = q - 1;
    while (r >= a && child[r] > v) { child[r + 1] = child[r]; --r; }
    child[r + 1] = v;
  }
}

__global__ void k_child_nnz(int nc, const int* __restrict__ cs, const int* __restrict__ child,
                            const int* __restrict__ rp, int* cnt) {
  const int P = blockIdx.x * blockDim.x + threadIdx.x;
  if (P >= nc) return;
  int s = 0;
  for (int q = cs[P]; q < cs[P + 1]; ++q) s += rp[child[q] + 1] - rp[child[q]];
  cnt[P] = s;
}

// coarse cconn in discovery order (cfdAgglomerateLevel.m:89-98): a warp per coarse row; the lanes load
// a child's entries together and search the list together, entry by entry in order
__global__ void __launch_bounds__(kBlock) k_coarse_conn(int nc, const int* __restrict__ cs, const int* __restrict__ child,
                                                        const int* __restrict__ rp, const int* __restrict__ col,
                                                        const int* __restrict__ parents,
                                                        const int* __restrict__ estart, int* scratch, int* ccnt) {
  const int P = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (P >= nc) return;
  int* lst = scratch + estart[P];
  int m = 0;
  for (int q = cs[P]; q < cs[P + 1]; ++q) {
    const int k0 = rp[child[q]], k1 = rp[child[q] + 1];
    for (int kb = k0; kb < k1; kb += 32) {
      const int mine = kb + lane < k1 ? parents[col[kb + lane]] : P;
      for (int t = 0; t < min(32, k1 - kb); ++t) {
        const int Q = __shfl_sync(0xffffffffu, mine, t);
        if (Q == P) continue;
        bool seen = false;
        for (int e = lane; e < m && !seen; e += 32) seen = ((volatile int*)lst)[e] == Q;
        if (!__any_sync(0xffffffffu, seen)) {
          if (lane == 0) ((volatile int*)lst)[m] = Q;
          ++m;
          __syncwarp();
        }
      }
    }
  }
  if (lane == 0) ccnt[P] = m;
}

__global__ void k_coarse_copy(int nc, const int* __restrict__ estart, const int* __restrict__ scratch,
                              const int* __restrict__ crp, int* ccol) {
  const int P = blockIdx.x * blockDim.x + threadIdx.x;
  if (P >= nc) return;
  const int* lst = scratch + estart[P];
  for (int t = 0; t < crp[P + 1] - crp[P]; ++t) ccol[crp[P] + t] = lst[t];
}

// Galerkin by summation in fine natural order (assembleAgglomeratedLHS.m:16-30): a warp per coarse
// row. The lanes load a child's entries together; each lane keeps the sum of one coarse entry and
// takes the fine entries that belong to it in order, lane 0 the diagonal too, so every sum is the
// sequential one. Rows of more than 32 coarse entries are done 32 entries at a time.
template <typename T>
__global__ void __launch_bounds__(kBlock) k_galerkin(int nc, const int* __restrict__ cs, const int* __restrict__ child,
                                                     const int* __restrict__ rp, const int* __restrict__ col,
                                                     const int* __restrict__ parents, const T* __restrict__ ac,
                                                     const T* __restrict__ anb, const int* __restrict__ crp,
                                                     const int* __restrict__ ccol, T* cac, T* canb) {
  const int P = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (P >= nc) return;
  const int c0 = crp[P], c1 = crp[P + 1], q0 = cs[P], q1 = cs[P + 1];
  T AC = 0;
  for (int cb = c0; cb == c0 || cb < c1; cb += 32) {
    const int target = cb + lane < c1 ? ccol[cb + lane] : -1;
    T sum = 0;
    for (int q = q0; q < q1; ++q) {
      const int c = child[q], k0 = rp[c], k1 = rp[c + 1];
      if (cb == c0) AC = AC + ac[c];
      for (int kb = k0; kb < k1; kb += 32) {
        const bool in = kb + lane < k1;
        const int mine = in ? parents[col[kb + lane]] : -2;
        const T val = in ? anb[kb + lane] : T(0);
        const int m = min(32, k1 - kb);
        for (int t = 0; t < m; ++t) {
          const int Q = __shfl_sync(0xffffffffu, mine, t);
          const T v = __shfl_sync(0xffffffffu, val, t);
          if (Q == target) sum = sum + v;
          if (cb == c0 && Q == P) AC = AC + v;
        }
      }
    }
    if (cb + lane < c1) canb[cb + lane] = sum;
  }
  if (lane == 0) cac[P] = AC;
}

// ---------------------------------------------------------------------------------
int agglomerate_level(LinCtx& c, AggScratch& w, Level& F, Level& C, int* nCoarse) {
  const int n = F.n;
  UFVM_CHECK(c.ensure(n));
  UFVM_CHECK(dalloc(w.maxAnb, n));
  UFVM_CHECK(dalloc(w.strong, std::max(F.nnz, 1)));
  UFVM_CHECK(dalloc(w.hold, n));
  UFVM_CHECK(dalloc(w.flag, 2 * (size_t)n));
  UFVM_CHECK(dalloc(w.rank, 2 * (size_t)n + 1));
  UFVM_CHECK(dalloc(F.parents, n));
  cudaStream_t st = c.stream;
  k_strong<<<nblocks(n), kBlock, 0, st>>>(n, F.rowptr.p, F.anb.p, w.maxAnb.p, w.strong.p);
  UFVM_LAUNCH_CHECK();
  UFVM_CUDA(cudaMemsetAsync(F.parents.p, 0xff, n * sizeof(int), st));
  UFVM_CUDA(cudaMemsetAsync(w.flag.p, 0, 2 * (size_t)n * sizeof(int), st));
  int h[2] = {0, 0};
  UFVM_CUDA(cudaMemsetAsync(c.iflag.p, 0, 2 * sizeof(int), st));
  k_strong_back<<<nblocks(n), kBlock, 0, st>>>(n, F.rowptr.p, F.col.p, w.strong.p, c.iflag.p + 1);
  UFVM_LAUNCH_CHECK();
  AggArgs a{n, F.rowptr.p, F.col.p, w.strong.p, nullptr, nullptr, nullptr, F.parents.p, w.hold.p, w.flag.p, c.iflag.p + 1};
  const bool narrow = F.nnz <= (long long)kAggNarrow * n;
  auto rounds = [&](bool oneway) -> int {
    if (n <= kAggOneBlock) {
      const auto k = oneway ? (narrow ? k_agg_rounds<8, true> : k_agg_rounds<32, true>)
                            : (narrow ? k_agg_rounds<8, false> : k_agg_rounds<32, false>);
      k<<<1, kAggBlock, 0, st>>>(a);
      UFVM_LAUNCH_CHECK();
      return UFVM_OK;
    }
    UFVM_CHECK(dalloc(w.bar, 2));
    UFVM_CUDA(cudaMemsetAsync(w.bar.p, 0, sizeof(AggBar), st));
    const int blocks = std::min(c.nsm, (n + kAggBlock - 1) / kAggBlock);
    void* args[] = {(void*)&a, (void*)&w.bar.p, (void*)&c.berr.p};
    const auto k = oneway ? (narrow ? k_agg_grid<8, true> : k_agg_grid<32, true>)
                          : (narrow ? k_agg_grid<8, false> : k_agg_grid<32, false>);
    UFVM_CUDA(cudaLaunchCooperativeKernel((const void*)k, dim3(blocks), dim3(kAggBlock), args, 0, st));
    return UFVM_OK;
  };
  UFVM_CHECK(rounds(false));
  UFVM_CUDA(cudaMemcpyAsync(h, c.iflag.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
  UFVM_CUDA(cudaStreamSynchronize(st));
  int* orphan = nullptr;
  if (h[1]) {  // those rounds did nothing: once more, over the links by the cell they lead to
    UFVM_CHECK(dalloc(w.cnt, n));
    UFVM_CHECK(dalloc(w.irp, n + 1));
    UFVM_CHECK(dalloc(w.icol, std::max(F.nnz, 1)));
    UFVM_CHECK(dalloc(w.istrong, std::max(F.nnz, 1)));
    UFVM_CUDA(cudaMemsetAsync(w.cnt.p, 0, n * sizeof(int), st));
    k_in_count<<<nblocks(n), kBlock, 0, st>>>(n, F.rowptr.p, F.col.p, w.strong.p, w.cnt.p);
    UFVM_CHECK(scan_exclusive(c, w.cnt.p, w.irp.p, n, nullptr));
    k_in_fill<<<nblocks(n), kBlock, 0, st>>>(n, F.rowptr.p, F.col.p, w.strong.p, w.irp.p, w.cnt.p, w.icol.p,
                                             w.istrong.p);
    UFVM_LAUNCH_CHECK();
    a.irp = w.irp.p; a.icol = w.icol.p; a.istrong = w.istrong.p;
    a.asym = c.iflag.p;  // not raised
    UFVM_CHECK(rounds(true));
    k_unassigned<<<nblocks(n), kBlock, 0, st>>>(n, F.parents.p, w.hold.p);  // the holders are done with
    UFVM_LAUNCH_CHECK();
    orphan = w.hold.p;
  }
  // orphans wait for one another: a cooperative launch
  const int grid = std::max(1, std::min(kAggGrid, nblocks(n)));
  {
    int* newflag = w.flag.p + n;
    void* args[] = {(void*)&n, (void*)&F.rowptr.p, (void*)&F.col.p, (void*)&F.anb.p, (void*)&w.maxAnb.p,
                    (void*)&F.parents.p, (void*)&newflag, (void*)&orphan, (void*)&c.berr.p};
    UFVM_CUDA(cudaLaunchCooperativeKernel((const void*)k_agg_orphans, dim3(grid), dim3(256), args, 0, st));
  }
  // relabel: seeds' parents in seed order, then orphans' new parents in orphan order
  int nc = 0;
  UFVM_CHECK(scan_exclusive(c, w.flag.p, w.rank.p, 2 * n, &nc));
  UFVM_CHECK(check_barrier(c));
  k_relabel<<<nblocks(n), kBlock, 0, st>>>(n, w.rank.p, F.parents.p);
  UFVM_LAUNCH_CHECK();
  *nCoarse = nc;
  // children of each coarse row, sorted by fine index
  UFVM_CHECK(dalloc(w.cnt, nc + 1));
  UFVM_CHECK(dalloc(F.childStart, nc + 1));
  UFVM_CHECK(dalloc(F.child, n));
  UFVM_CUDA(cudaMemsetAsync(w.cnt.p, 0, (nc + 1) * sizeof(int), st));
  k_count_children<<<nblocks(n), kBlock, 0, st>>>(n, F.parents.p, w.cnt.p);
  UFVM_CHECK(scan_exclusive(c, w.cnt.p, F.childStart.p, nc, nullptr));
  UFVM_CUDA(cudaMemcpyAsync(w.cnt.p, F.childStart.p, nc * sizeof(int), cudaMemcpyDeviceToDevice, st));
  k_fill_children<<<nblocks(n), kBlock, 0, st>>>(n, F.parents.p, w.cnt.p, F.child.p);
  k_sort_children<<<nblocks(nc), kBlock, 0, st>>>(nc, F.childStart.p, F.child.p);
  UFVM_LAUNCH_CHECK();
  // coarse connectivity
  UFVM_CHECK(dalloc(w.estart, nc + 1));
  k_child_nnz<<<nblocks(nc), kBlock, 0, st>>>(nc, F.childStart.p, F.child.p, F.rowptr.p, w.cnt.p);
  UFVM_CHECK(scan_exclusive(c, w.cnt.p, w.estart.p, nc, nullptr));
  UFVM_CHECK(dalloc(w.lists, std::max(F.nnz, 1)));  // every fine row has one parent
  k_coarse_conn<<<nblocks(32ll * nc), kBlock, 0, st>>>(nc, F.childStart.p, F.child.p, F.rowptr.p, F.col.p, F.parents.p,
                                                w.estart.p, w.lists.p, w.cnt.p);
  UFVM_LAUNCH_CHECK();
  C.n = nc;
  UFVM_CHECK(dalloc(C.rowptr, nc + 1));
  int cnnz = 0;
  UFVM_CHECK(scan_exclusive(c, w.cnt.p, C.rowptr.p, nc, &cnnz));
  C.nnz = cnnz;
  UFVM_CHECK(dalloc(C.col, std::max(cnnz, 1)));
  k_coarse_copy<<<nblocks(nc), kBlock, 0, st>>>(nc, w.estart.p, w.lists.p, C.rowptr.p, C.col.p);
  UFVM_LAUNCH_CHECK();
  UFVM_CHECK(dalloc(C.ac, nc));
  UFVM_CHECK(dalloc(C.anb, std::max(cnnz, 1)));
  UFVM_CHECK(dalloc(C.bc, nc));
  UFVM_CHECK(dalloc(C.dphi, nc));
  UFVM_CUDA(cudaMemsetAsync(C.bc.p, 0, nc * sizeof(double), st));
  UFVM_CUDA(cudaMemsetAsync(C.dphi.p, 0, nc * sizeof(double), st));
  C.sched_valid = false;
  C.color_valid = false;
  C.mc_valid = false;
  return galerkin(c, F, C);
}

int galerkin(LinCtx& c, Level& F, Level& C) {
  k_galerkin<double><<<nblocks(32ll * C.n), kBlock, 0, c.stream>>>(C.n, F.childStart.p, F.child.p, F.rowptr.p, F.col.p,
                                                             F.parents.p, F.ac.p, F.anb.p, C.rowptr.p, C.col.p,
                                                             C.ac.p, C.anb.p);
  UFVM_LAUNCH_CHECK();
  return UFVM_OK;
}

int galerkin32(LinCtx& c, Level& F, Level& C) {
  k_galerkin<float><<<nblocks(32ll * C.n), kBlock, 0, c.stream>>>(C.n, F.childStart.p, F.child.p, F.rowptr.p, F.col.p,
                                                            F.parents.p, F.ac32.p, F.anb32.p, C.rowptr.p, C.col.p,
                                                            C.ac32.p, C.anb32.p);
  UFVM_LAUNCH_CHECK();
  return UFVM_OK;
}

void AggScratch::release() {
  dfree(maxAnb); dfree(strong); dfree(hold); dfree(flag); dfree(rank); dfree(cnt); dfree(estart); dfree(lists); dfree(bar);
  dfree(irp); dfree(icol); dfree(istrong);
}

// ---------------------------------------------------------------------------------
// AMG driver on a hierarchy whose level 0 is the assembled p matrix.
// A rebuild (every p solve in the reference, cfdApplyAMG.m:19) keeps the previous hierarchy's
// coarse-level device arrays and hands them to the new levels, whose allocations (dalloc) reuse an
// array that is large enough instead of freeing and allocating it again; every schedule,
// colouring and copy cached on a level is invalidated, since the new level's pattern may differ.
static void reset_level_caches(Level& L) {
  L.sched_valid = false;
  L.dc_epoch = 0;
  L.dc_quirks = 0;
  for (int k = 0; k < 4; ++k) {
    L.sell_valid[k] = false;
    L.sell_epoch[k] = 0;
  }
  L.color_valid = false;
  L.ncolor = 0;
  L.h_colorStart.clear();
  L.mc_valid = false;
  L.mcW = 0;
  L.mc_epoch = 0;
  L.ell_valid = false;
  L.ellW = 0;
}

int AmgSolver::build(std::vector<Level>& lev, int max_coarse, int quirks, int* n_levels) {
  std::vector<Level> pool(lev.begin() + 1, lev.end());
  lev.resize(1);
  size_t next = 0;
  auto release_pool = [&]() {
    for (size_t k = next; k < pool.size(); ++k) free_level(pool[k]);
    pool.clear();
  };
  int il = 0;
  while (il < max_coarse) {
    ++il;
    Level coarse;
    if (next < pool.size()) {
      coarse = pool[next];
      pool[next++] = Level();
      reset_level_caches(coarse);
    }
    int np = 0;
    const int st = agglomerate_level(ctx, agg, lev[il - 1], coarse, &np);
    if (st != UFVM_OK) {
      free_level(coarse);
      release_pool();
      return st;
    }
    if (np == 1 && !(quirks & UFVM_Q16_ONE_CELL_COARSEST)) {
      // repaired: a single aggregate of the pure-Neumann operator has a ~0 diagonal
      free_level(coarse);
      --il;
      break;
    }
    lev.push_back(coarse);
    if (np <= 5) break;
  }
  release_pool();
  *n_levels = il + 1;
  return UFVM_OK;
}

void free_level(Level& L, bool keep_matrix) {
  if (!keep_matrix) { dfree(L.rowptr); dfree(L.col); dfree(L.ac); dfree(L.anb); dfree(L.bc); dfree(L.dphi); }
  dfree(L.parents); dfree(L.tpos); dfree(L.lord); dfree(L.r); dfree(L.dc); dfree(L.rc);
  dfree(L.waveRows); dfree(L.waveLev); dfree(L.waveTask); dfree(L.waveNtask); dfree(L.color); dfree(L.colorRows); dfree(L.colorStart);
  dfree(L.childStart); dfree(L.child); dfree(L.ac32); dfree(L.anb32); dfree(L.bc32); dfree(L.dphi32); dfree(L.r32);
  dfree(L.fr); dfree(L.fp); dfree(L.fq);
  dfree(L.perm); dfree(L.inv); dfree(L.ellCol); dfree(L.parentsP); dfree(L.childP); dfree(L.childStartP); dfree(L.gpos);
  dfree(L.ellAnb); dfree(L.uAnb); dfree(L.uAc); dfree(L.uBc); dfree(L.uX);
  dfree(L.mcRow); dfree(L.mcCol); dfree(L.mcAnb); dfree(L.mcAc); dfree(L.mcBc);
  for (int k = 0; k < 4; ++k) {
    dfree(L.sellCol[k]); dfree(L.sellA[k]);
    L.sell_valid[k] = false;
    L.sell_epoch[k] = 0;
  }
  L.mc_valid = false;
  L.mc_epoch = 0;
  L.ell_valid = false;
  L.sched_valid = false;
  L.color_valid = false;
  L.dc_epoch = 0;
}

// The operations of one cycle, in order. A level's residual r is kept by its smoother call, so the
// restriction that follows starts from it.
int AmgSolver::plan_cycle(int L, std::vector<SmallOp>& ops) const {
  const int down = (quirks & UFVM_Q6_COARSE_DPHI_KEPT) ? SMALL_RESTRICT_KEEP : SMALL_RESTRICT;
  auto S = [&](int l, int n, double f) { ops.push_back(SmallOp{SMALL_SMOOTH, l, n, f}); };
  auto R = [&](int l, int p) {
    if (p >= 0) S(l, p, 0.1);
    ops.push_back(SmallOp{down, l, 0, 0.0});
  };
  auto Pr = [&](int l) {
    ops.push_back(SmallOp{SMALL_PROLONG, l, 0, 0.0});
    S(l - 1, post, rrf);
  };
  auto solveC = [&]() { S(L, post, 0.1); };
  if (cycle_type != UFVM_CYCLE_V && L < 3) {
    set_error("W/F-cycle needs at least 4 AMG levels (the reference indexes level 0)");
    return UFVM_E_AMG_LEVELS;
  }
  for (int l = 0; l < L; ++l) R(l, pre);
  solveC();
  if (cycle_type == UFVM_CYCLE_W || cycle_type == UFVM_CYCLE_F) {
    Pr(L); R(L - 1, -1); solveC();
    Pr(L); Pr(L - 1); R(L - 2, -1); R(L - 1, pre); solveC();
    Pr(L); Pr(L - 1); Pr(L - 2);
    R(L - 3, -1); R(L - 2, pre); R(L - 1, pre); solveC();
    if (cycle_type == UFVM_CYCLE_W) {
      Pr(L); Pr(L - 1); R(L - 2, -1); R(L - 1, pre); solveC();
      Pr(L); R(L - 1, -1); solveC();
    }
  }
  for (int l = L; l >= 1; --l) Pr(l);
  return UFVM_OK;
}

// Runs of operations on small levels are one launch each, the others a few launches each; nothing
// here waits for the device.
int AmgSolver::run_ops(std::vector<Level>& lev, const std::vector<SmallOp>& ops) {
  auto small_op = [&](const SmallOp& o) { return (o.type == SMALL_PROLONG ? o.lev - 1 : o.lev) >= lsmall; };
  for (size_t i = 0; i < ops.size();) {
    const SmallOp& o = ops[i];
    if (small_op(o)) {
      SmallProg p = small_prog();
      for (; i < ops.size() && small_op(ops[i]) && p.nops < kSmallOps; ++i) {
        p.op[p.nops] = ops[i];
        p.op[p.nops++].lev -= lsmall;
      }
      UFVM_CHECK(small_run(ctx, p));
      continue;
    }
    ++i;
    if (o.type == SMALL_SMOOTH) {
      UFVM_CHECK(solve_algebraic_system(ctx, lev[o.lev], smoother, o.iters, o.rrf, quirks, nullptr, nullptr, nullptr));
    } else if (o.type == SMALL_PROLONG) {
      UFVM_CHECK(prolong(ctx, lev[o.lev - 1], lev[o.lev]));
    } else {
      Level& C = lev[o.lev + 1];
      UFVM_CHECK(restrict_residual(ctx, lev[o.lev], C));
      if (o.type == SMALL_RESTRICT) UFVM_CUDA(cudaMemsetAsync(C.dphi.p, 0, C.n * sizeof(double), ctx.stream));
    }
  }
  return UFVM_OK;
}

SmallProg AmgSolver::small_prog() const {
  SmallProg p{};
  p.lev = stab.p;
  p.ctl = ctx.ctl.p;
  p.err = ctx.berr.p;
  p.smoother = smoother;
  p.quirks = quirks;
  return p;
}

int AmgSolver::apply(std::vector<Level>& lev, bool rebuild, int* n_levels, double* r0, double* r1) {
  UFVM_CHECK(ctx.ensure(lev[0].n));
  if (rebuild) UFVM_CHECK(build(lev, max_coarse, quirks, n_levels));
  else {
    for (int l = 1; l < *n_levels; ++l) {
      UFVM_CHECK(galerkin(ctx, lev[l - 1], lev[l]));
      UFVM_CUDA(cudaMemsetAsync(lev[l].bc.p, 0, lev[l].n * sizeof(double), ctx.stream));
      UFVM_CUDA(cudaMemsetAsync(lev[l].dphi.p, 0, lev[l].n * sizeof(double), ctx.stream));
    }
  }
  const int L = *n_levels - 1;
  // the matrices are final from here to the end of this solve: a fresh epoch lets the smoother
  // calls of the cycles share each level's DILU factor and coefficient copies
  EpochScope epoch(ctx);
  std::vector<SmallOp> ops;
  if (cycle_type != UFVM_CYCLE_V && L < 3) {
    // no such cycle exists: an error, unless the start already meets the termination rule
    double init = 0;
    UFVM_CHECK(sum_abs_residual(ctx, lev[0], &init));
    cycles_used = 0;
    *r0 = *r1 = init;
    if (max_cycles < 1 || !(init > rrf * init)) return UFVM_OK;
  }
  UFVM_CHECK(plan_cycle(L, ops));
  // the small levels: their table, and their factorisations as operations of their own
  lsmall = 0;
  while (lsmall <= L && !small_level(lev[lsmall])) ++lsmall;
  SmallProg first = small_prog();
  if (lsmall <= L) {
    std::vector<SmallLev> tab(L + 1 - lsmall);
    for (int l = lsmall; l <= L; ++l)
      UFVM_CHECK(small_describe(ctx, lev[l], l < L ? &lev[l + 1] : nullptr, smoother, tab[l - lsmall]));
    UFVM_CHECK(dalloc(stab, tab.size()));
    UFVM_CUDA(cudaMemcpyAsync(stab.p, tab.data(), tab.size() * sizeof(SmallLev), cudaMemcpyHostToDevice, ctx.stream));
    first = small_prog();
    if (smoother == UFVM_SMOOTHER_ILU)
      for (int l = lsmall; l <= L; ++l) {
        if (first.nops == kSmallOps) {  // the number of levels is the caller's
          UFVM_CHECK(small_run(ctx, first));
          first.nops = 0;
        }
        first.op[first.nops++] = SmallOp{SMALL_FACTOR, l - lsmall, 0, 0.0};
      }
  }
  SmoothCtl h{};
  if (lsmall == 0 && max_cycles > 0 && first.nops + ops.size() <= (size_t)kSmallOps) {
    // every level is small: the whole solve is one launch
    first.pre = first.nops;
    for (const SmallOp& o : ops) first.op[first.nops++] = o;
    first.max_cycles = max_cycles;
    first.rrf = rrf;
    UFVM_CHECK(small_run(ctx, first));
    UFVM_CHECK(read_ctl(ctx, &h));
    cycles_used = h.cycles;
    *r0 = h.init;
    *r1 = h.sum;
    return UFVM_OK;
  }
  if (first.nops) UFVM_CHECK(small_run(ctx, first));
  double init = 0;
  UFVM_CHECK(sum_abs_residual(ctx, lev[0], &init));
  double fin = init;
  int ncyc = 1;
  while (ncyc <= max_cycles && fin > rrf * init) {
    UFVM_CHECK(run_ops(lev, ops));
    UFVM_CHECK(read_ctl(ctx, &h));  // the cycle ends with level 0's smoother call: its last sum |r|
    fin = h.sum;
    ++ncyc;
  }
  cycles_used = ncyc - 1;
  *r0 = init;
  *r1 = fin;
  return UFVM_OK;
}

}  // namespace ufvm
