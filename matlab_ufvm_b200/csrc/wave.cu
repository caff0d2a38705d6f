// wave.cu -- the natural-order sweeps of uFVM's linear solve as chunked wavefronts.
//
//   GS ('SOR')    solve/cfdSolveSOR.m:13-29
//   DILU ('ILU')  solve/cfdFactorizeILU.m:5-47, solve/cfdSolveILU.m:18-93
//
// A row of such a sweep needs the new values of its lower-index neighbours (upper-index ones in
// a backward pass), so the sweep is a chain of dependency levels: 499 of them on a 250 x 250
// grid, 190 on a 64^3 one. The chain's latency bounds it, not the bytes. Two things make a link
// of the chain short here:
//
//  * the rows are cut into contiguous chunks, one CTA each, and a CTA keeps its chunk's values in
//    shared memory, so most links are a shared-memory store, a warp-to-warp hand-off and a
//    shared-memory load. Dependencies between chunks run one way only (from lower to higher row
//    indices, or the other way in a backward pass), so the chunks form a pipeline: a chunk waits
//    for a value of another one only until the other one is far enough ahead. Such a value is
//    published in global memory in an array preset to a NaN pattern that no published value has:
//    the value is its own flag and one polling load is the whole hand-off;
//  * inside a chunk the rows are sorted by dependency level and cut into tasks of 32 rows, taken
//    by the CTA's warps in turn. A warp loads what its next task needs (coefficients, right-hand
//    side, products with values that no earlier row of this pass changes or that come from other
//    chunks) while the other warps run the tasks before it, and when its turn comes it goes
//    through the levels in its task one by one: what is left of a level is a few shared-memory
//    loads, the row's remaining products and subtractions and one store, without a wait for
//    another warp. Tasks of one wide level run side by side.
//
// Every row evaluates the reference's expression in the reference's order, so the results are
// those of the sequential sweep bit for bit, whatever the schedule. That takes more than a row's own
// entries where the pattern is not symmetric: see k_level_relax and wave_gs.
//
// The chunks wait on one another, so every launch whose CTAs wait is cooperative (all CTAs resident), and
// every wait is bounded, by more than the longest chain of the matrix can take: a wait that runs out
// raises the error flag, the CTA stops waiting for values from then on and completes with what it has,
// and the host reports UFVM_E_TIMEOUT.
#include "wave.cuh"

#include "small.cuh"
#include "wave_dev.cuh"

namespace ufvm {

namespace {

constexpr int kSchedBlock = 512, kSchedLocal = 256;  // schedule CTA; its threads that take rows
constexpr size_t kSmemMax = 220 * 1024;

// ---------------------------------------------------------------- schedules
struct SchedArgs {
  int n, nnz, chunks, B, smem_levels, hist_cap, ghist_cap;
  const int *rp, *col;
  int* lvl;        // [2][n], preset to -1
  int* work;       // [2][2][n]: running level and open count of each row, for chunks beyond shared memory
  int2* ext;       // [2][nnz]: (row offset, neighbour) of each neighbour in another chunk
  int* rows;       // [2][n] rows by chunk and level: position -> row
  int2* plev;      // [2][n] position -> (level, first task of that level)
  int* task;       // [2][chunks * (B + 1)] first position of each task
  int* ntask;      // [2][chunks]
  int* ghist;      // [2 * chunks][2 * ghist_cap], or null
  int* flags;      // [0] a wait gave up, [1] a chunk's level range exceeds the histogram, [5] k_wave_pattern,
                   // [6] sum over the chunks of their numbers of levels (forward), [7] progress of all CTAs
  int given;       // the levels are in lvl already
};

// One CTA per (direction, chunk): dependency levels of the chunk's rows (level = 1 + the largest
// level of the lower neighbours, upper ones backward), then the rows sorted by level and cut into
// tasks of at most 32 rows: a wide level is several tasks, consecutive narrow levels that fit share
// one. Every row counts its unresolved neighbours; the first half of the threads look after the
// rows (a row whose count is zero has its level: it is published, and the rows that wait for it are
// told), the second half after the neighbours in other chunks (polled until their level is
// published; a level is its own flag, -1: not known yet). Nothing blocks on one row: a thread
// keeps a bitmask of up to 32 open rows or neighbours and visits each in turn, so a row that is
// ready never waits behind one that is not. (A chunk of more rows than 32 per thread is taken in
// windows, in sweep order: a row's neighbours are in its own window or an earlier one.)
__global__ void __launch_bounds__(kSchedBlock, 2) k_wave_schedule(SchedArgs a) {
  extern __shared__ int sm_i[];
  __shared__ int s_min, s_max, s_next, s_scan[kSchedBlock / 32];
  __shared__ volatile int s_dead;
  const int dir = blockIdx.x / a.chunks, c = blockIdx.x % a.chunks;
  const int base = c * a.B, cnt = min(a.B, a.n - base);
  const int tid = threadIdx.x;
  int* glvl = a.lvl + (size_t)dir * a.n;
  int* lv = a.smem_levels ? sm_i : a.work + (size_t)dir * 2 * a.n + base;
  int* open = a.smem_levels ? sm_i + a.B : a.work + ((size_t)dir * 2 + 1) * a.n + base;
  int2* ext = a.ext + (size_t)dir * a.nnz + a.rp[base];
  if (!a.given && a.flags[5]) return;  // a pattern that is not symmetric: see wave_build
  if (tid == 0) { s_min = 0x7fffffff; s_max = 0; s_dead = 0; s_next = 0; }
  __syncthreads();
  for (int l = tid; l < cnt; l += kSchedBlock) {
    const int i = base + l;
    int o = 0;
    if (a.given) {
      const int level = glvl[i];
      atomicMin(&s_min, level);
      atomicMax(&s_max, level);
      continue;
    }
    for (int k = a.rp[i]; k < a.rp[i + 1]; ++k) {
      const int j = a.col[k];
      if (dir == 0 ? j >= i : j <= i) continue;
      ++o;
      if ((unsigned)(j - base) >= (unsigned)cnt) ext[atomicAdd(&s_next, 1)] = make_int2(l, j);
    }
    lv[l] = 0;
    open[l] = o;
  }
  __syncthreads();
  int lo = 0x7fffffff, hi = 0, seen = 0;
  unsigned spins = 0;
  long long t0 = clock64();
  // a row's level is complete before its count says so (counters in global memory: atomics of one
  // thread are ordered in the L2 only by the wider fence)
  auto fence = [&]() {
    if (a.smem_levels) __threadfence_block();
    else __threadfence();
  };
  // The bound of a wait starts again whenever any CTA resolves something: a chunk at the end of a
  // long chain waits for all the others.
  bool moved = false;
  auto give_up = [&](bool now) {
    moved |= now;
    if ((++spins & 1023u) != 0) return;
    if (moved) atomicAdd(a.flags + 7, 1);
    moved = false;
    const int p = ld_flag(a.flags + 7);
    if (p != seen) {
      seen = p;
      t0 = clock64();
    } else if (clock64() - t0 > kFlagClocks) {
      atomicExch(a.flags, 1);
      s_dead = 1;
    }
  };
  if (a.given) {
  } else if (tid < kSchedLocal) {
    for (int w0 = 0; w0 < cnt; w0 += 32 * kSchedLocal) {
      unsigned pend = 0;
      for (int q = 0; q < 32; ++q)
        if (w0 + q * kSchedLocal + tid < cnt) pend |= 1u << q;
      while (__any_sync(0xffffffffu, pend != 0)) {
        // every lane looks for one ready row; then the warp tells the rows that wait for each of
        // them, a lane per entry
        int l = -1, level = 0;
        for (unsigned m = pend; m && l < 0; m &= m - 1) {
          const int q = __ffs(m) - 1, o = w0 + q * kSchedLocal + tid;
          const int r = dir == 0 ? o : cnt - 1 - o;
          if (*(volatile int*)(open + r) == 0 || s_dead) {
            l = r;
            pend &= ~(1u << q);
          }
        }
        if (l >= 0) {
          fence();
          level = *(volatile int*)(lv + l);
          st_flag(glvl + base + l, level);
          lo = min(lo, level);
          hi = max(hi, level);
        }
        for (unsigned m = __ballot_sync(0xffffffffu, l >= 0); m; m &= m - 1) {
          const int src = __ffs(m) - 1, i = base + __shfl_sync(0xffffffffu, l, src);
          const int up = __shfl_sync(0xffffffffu, level, src) + 1;
          for (int k = a.rp[i] + (tid & 31); k < a.rp[i + 1]; k += 32) {
            const int j = a.col[k];
            if ((dir == 0 ? j <= i : j >= i) || (unsigned)(j - base) >= (unsigned)cnt) continue;
            atomicMax(lv + (j - base), up);
            fence();
            atomicSub(open + (j - base), 1);
          }
        }
        give_up(l >= 0);
        __syncwarp();
      }
    }
  } else {
    const int t = tid - kSchedLocal, np = kSchedBlock - kSchedLocal, ne = s_next;
    for (int w0 = 0; w0 < ne; w0 += 32 * np) {
      unsigned pend = 0;
      for (int q = 0; q < 32; ++q)
        if (w0 + q * np + t < ne) pend |= 1u << q;
      while (__any_sync(0xffffffffu, pend != 0)) {
        const unsigned before = pend;
        unsigned m = pend;
        while (m) {
          int2 e[4];
          int v[4], q[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {  // four polls in flight
            q[u] = m ? __ffs(m) - 1 : -1;
            m &= m - 1;
            if (q[u] >= 0) e[u] = ext[w0 + q[u] * np + t];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = q[u] >= 0 ? ld_flag(glvl + e[u].y) : -1;
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (q[u] >= 0 && (v[u] >= 0 || s_dead)) {
              atomicMax(lv + e[u].x, v[u] + 1);
              fence();
              atomicSub(open + e[u].x, 1);
              pend &= ~(1u << q[u]);
            }
        }
        give_up(pend != before);
        __syncwarp();
      }
    }
  }
  if (lo <= hi) {
    atomicMin(&s_min, lo);
    atomicMax(&s_max, hi);
  }
  __syncthreads();
  const int mn = s_min, range = s_max - s_min + 1;
  int* hist = sm_i + (a.smem_levels ? 2 * a.B : 0);
  if (range > a.hist_cap) {
    if (range > a.ghist_cap) {
      if (tid == 0) atomicExch(a.flags + 1, 1);
      return;
    }
    hist = a.ghist + (size_t)blockIdx.x * 2 * a.ghist_cap;
  }
  int* start = hist + (range > a.hist_cap ? a.ghist_cap : a.hist_cap);
  for (int b = tid; b < range; b += kSchedBlock) hist[b] = 0;
  __syncthreads();
  for (int l = tid; l < cnt; l += kSchedBlock) atomicAdd(hist + (ld_flag(glvl + base + l) - mn), 1);
  __syncthreads();
  // exclusive scan of the levels' rows
  const int per = (range + kSchedBlock - 1) / kSchedBlock;
  const int b0 = min(range, tid * per), b1 = min(range, b0 + per);
  int nr = 0;
  for (int b = b0; b < b1; ++b) nr += hist[b];
  int ir = nr;
  const int lane = tid & 31, w = tid >> 5;
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, ir, o);
    if (lane >= o) ir += x;
  }
  if (lane == 31) s_scan[w] = ir;
  __syncthreads();
  int at = ir - nr;
  for (int v = 0; v < w; ++v) at += s_scan[v];
  for (int b = b0; b < b1; ++b) {
    const int h = hist[b];
    hist[b] = at;
    at += h;
  }
  __syncthreads();
  if (tid == 0) {
    int* task = a.task + ((size_t)dir * a.chunks + c) * (a.B + 1);
    int nt = 0, fill = 0, pos = 0, levels = 0;  // tasks closed; rows in the open task; rows so far
    for (int b = 0; b < range; ++b) {
      const int end = b + 1 < range ? hist[b + 1] : cnt, h = end - pos;
      if (h == 0) continue;
      ++levels;
      if (fill > 0 && fill + h > kTaskRows) {
        ++nt;
        fill = 0;
      }
      start[b] = nt;
      if (fill == 0) task[nt] = base + pos;
      if (h > kTaskRows) {
        for (int r = kTaskRows; r < h; r += kTaskRows) task[++nt] = base + pos + r;
        ++nt;
      } else {
        fill += h;
      }
      pos = end;
    }
    if (fill > 0) ++nt;
    task[nt] = base + cnt;
    a.ntask[dir * a.chunks + c] = nt;
    if (dir == 0) atomicAdd(a.flags + 6, levels);
  }
  __syncthreads();
  int* rows = a.rows + (size_t)dir * a.n;
  int2* plev = a.plev + (size_t)dir * a.n;
  for (int l = tid; l < cnt; l += kSchedBlock) {
    const int level = ld_flag(glvl + base + l);
    const int p = base + atomicAdd(hist + (level - mn), 1);
    rows[p] = base + l;
    plev[p] = make_int2(level, start[level - mn]);
  }
}

// tpos[k]: position of the transposed entry (j, i) for entry k = (i, j).
// lord: for each row, the CSR positions of its lower neighbours in increasing column order
// (the order in which the reference's outer loop over i1 delivers them), then -1 in the row's
// remaining slots. wmax[0..2]: largest number of entries, lower and upper entries of a row;
// wmax[3]: raised if some entry (i, j) is not matched by as many entries (j, i).
__global__ void k_wave_pattern(int n, const int* __restrict__ rp, const int* __restrict__ col, int* tpos, int* lord,
                               int* wmax) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int len = 0, low = 0, up = 0;
  if (i < n) {
    const int k0 = rp[i], k1 = rp[i + 1];
    len = k1 - k0;
    for (int k = k0; k < k1; ++k) {
      const int j = col[k];
      int p = -1, there = 0, here = 1;
      for (int q = rp[j]; q < rp[j + 1]; ++q)
        if (col[q] == i) {
          if (p < 0) p = q;
          ++there;
        }
      // more than one entry (i, j) against a single (j, i) is seen from row j: searching the own
      // row for every entry took 0.25 s for a row of 6,000
      if (there > 1) {
        here = 0;
        for (int q = k0; q < k1; ++q) here += col[q] == j;
      }
      if (here != there) wmax[3] = 1;
      tpos[k] = p;
      up += j > i;
    }
    int t = k0, prev = -1;
    while (true) {
      int best = 0x7fffffff, bk = -1;
      for (int k = k0; k < k1; ++k) {
        const int j = col[k];
        if (j < i && j > prev && j < best) { best = j; bk = k; }
      }
      if (bk < 0) break;
      prev = best;
      lord[t++] = bk;
    }
    low = t - k0;
    for (; t < k1; ++t) lord[t] = -1;
  }
  len = __reduce_max_sync(0xffffffffu, len);
  low = __reduce_max_sync(0xffffffffu, low);
  up = __reduce_max_sync(0xffffffffu, up);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(wmax, len);
    atomicMax(wmax + 1, low);
    atomicMax(wmax + 2, up);
  }
}

// One relaxation pass over the levels: lvl[i] = 1 + max lvl[j] over lower neighbours j < i (upper
// ones for dir 1), from lvl = 0 to the fixed point. For chunks whose levels do not fit in shared
// memory, and (oneway) for a pattern that is not symmetric, where a row cannot tell the rows that wait
// for it: there a row j also comes after the rows before it that read its old value (a Gauss-Seidel
// row i < j with an entry j; in a symmetric pattern j has the entry i itself).
__global__ void k_level_relax(int n, int dir, int oneway, const int* __restrict__ rp, const int* __restrict__ col,
                              int* lvl, int* changed) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int own = __ldcg(lvl + i);
  int m = oneway ? own : 0;
  for (int k = rp[i]; k < rp[i + 1]; ++k) {
    const int j = col[k];
    if (dir == 0 ? j < i : j > i) m = max(m, __ldcg(lvl + j) + 1);
  }
  if (m != own) {
    if (oneway) atomicMax(lvl + i, m);
    else __stcg(lvl + i, m);
    *changed = 1;
  }
  if (!oneway) return;
  for (int k = rp[i]; k < rp[i + 1]; ++k) {
    const int j = col[k];
    if ((dir == 0 ? j > i : j < i) && __ldcg(lvl + j) <= m) {
      atomicMax(lvl + j, m + 1);
      *changed = 1;
    }
  }
}

// *done: whether max_passes were enough (0: as many as the rows can need).
int relax_levels(LinCtx& c, const Level& L, bool oneway, int max_passes, bool* done) {
  const int n = L.n;
  *done = true;
  UFVM_CUDA(cudaMemsetAsync(c.wlvl.p, 0, 2 * (size_t)n * sizeof(int), c.stream));
  for (int dir = 0; dir < 2; ++dir)
    for (int changed = 1, passes = 0; changed; passes += 8) {
      if (max_passes > 0 && passes >= max_passes) {
        *done = false;
        return UFVM_OK;
      }
      if (passes > n + 16) { set_error("level schedule did not converge"); return UFVM_E_INVALID; }
      UFVM_CUDA(cudaMemsetAsync(c.iflag.p, 0, sizeof(int), c.stream));
      for (int k = 0; k < 8; ++k)
        k_level_relax<<<nblocks(n), kBlock, 0, c.stream>>>(n, dir, oneway ? 1 : 0, L.rowptr.p, L.col.p,
                                                           c.wlvl.p + (size_t)dir * n, c.iflag.p);
      UFVM_LAUNCH_CHECK();
      UFVM_CUDA(cudaMemcpyAsync(&changed, c.iflag.p, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
      UFVM_CUDA(cudaStreamSynchronize(c.stream));
    }
  return UFVM_OK;
}

// ---------------------------------------------------------------- position-ordered ELL copies
// Schedule position p (row rows[p]) keeps its entries at [t * n + p], so a step's rows are read
// with unit stride; entries past the copy's width stay in the matrix alone. A column inside the row's own
// chunk is stored as its offset in the chunk, any other column j as -(j + 3); -1 past the row's end.
enum { SELL_GS_FWD = 0, SELL_GS_BWD = 1, SELL_ILU_FWD = 2, SELL_ILU_BWD = 3 };

template <int KIND, bool PATTERN>
__global__ void k_wave_fill(int n, int B, const int* __restrict__ rows, const int* __restrict__ rp,
                            const int* __restrict__ col, const int* __restrict__ lord,
                            const double* __restrict__ anb, int W, int* scol, double* sa) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int i = rows[p], base = i / B * B, k0 = rp[i], k1 = rp[i + 1];
  int t = 0;
  auto put = [&](int q) {
    if (PATTERN) {
      const int j = col[q];
      scol[(size_t)t * n + p] = (unsigned)(j - base) < (unsigned)B ? j - base : -(j + 3);
    }
    sa[(size_t)t * n + p] = anb[q];
    ++t;
  };
  for (int k = k0; k < k1 && t < W; ++k) {
    if (KIND == SELL_GS_FWD || KIND == SELL_GS_BWD) {
      put(k);
    } else if (KIND == SELL_ILU_FWD) {
      const int q = lord[k];
      if (q < 0) break;
      put(q);
    } else if (col[k] > i) {
      put(k);
    }
  }
  for (; PATTERN && t < W; ++t) {
    scol[(size_t)t * n + p] = -1;
    sa[(size_t)t * n + p] = 0.0;
  }
}

// ---------------------------------------------------------------- sweeps
enum { SWEEP_GS = 0, SWEEP_FACT = 1, SWEEP_ILU = 2 };

template <int SWEEP, int WP, int G, bool SM, int WIDE>
__global__ void __launch_bounds__(32 * G) k_wave_sweep(WaveArgs a) {
  if (a.ctl && !a.ctl->active) return;
  extern __shared__ __align__(16) double sm_d[];
  __shared__ unsigned long long turn[2][G];
  __shared__ int s_dead;
  const int chunk = blockIdx.x, base = chunk * a.B, cnt = min(a.B, a.n - base);
  double* xs = SM ? sm_d : a.loc + (size_t)chunk * (a.B + 1);
  if (threadIdx.x < 2 * G) mb_init(&turn[threadIdx.x / G][threadIdx.x % G]);
  if (threadIdx.x == 0) {
    s_dead = 0;
    st_loc<SM>(xs + a.B, 1.0);
  }
  if (SWEEP == SWEEP_GS)
    for (int l = threadIdx.x; l < cnt; l += 32 * G) st_loc<SM>(xs + l, a.x[base + l]);
  __syncthreads();
  if (SWEEP == SWEEP_GS) {
    wave_pass<OP_GS_FWD, WP, G, SM, WIDE>(a, a.f, chunk, xs, turn[0], &s_dead);
    wave_pass<OP_GS_BWD, WP, G, SM, WIDE>(a, a.b, chunk, xs, turn[1], &s_dead);
    for (int l = threadIdx.x; l < cnt; l += 32 * G) a.x[base + l] = ld_loc<SM>(xs + l);
  } else if (SWEEP == SWEEP_FACT) {
    wave_pass<OP_FACT, WP, G, SM, WIDE>(a, a.f, chunk, xs, turn[0], &s_dead);
  } else {
    wave_pass<OP_ILU_FWD, WP, G, SM, WIDE>(a, a.f, chunk, xs, turn[0], &s_dead);
    wave_pass<OP_ILU_BWD, WP, G, SM, WIDE>(a, a.b, chunk, xs, turn[1], &s_dead);
  }
}

// coop: the CTAs wait on one another, so all of them have to be resident
int launch_coop(const void* k, bool coop, int grid, int block, size_t smem, cudaStream_t st, void** args) {
  if (smem > 40 * 1024)  // the default limit of 48 KB includes the kernel's static shared memory
    UFVM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const cudaError_t e = coop ? cudaLaunchCooperativeKernel(k, dim3(grid), dim3(block), args, smem, st)
                             : cudaLaunchKernel(k, dim3(grid), dim3(block), args, smem, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    set_error(std::string("cooperative launch of a wavefront kernel: ") + cudaGetErrorString(e));
    return UFVM_E_CUDA;
  }
  return UFVM_OK;
}

template <int SWEEP, int WP, int G, int WIDE>
int launch_sweep(LinCtx& c, WaveArgs& a, int* fit) {
  const size_t vals = ((size_t)a.B + 1) * sizeof(double);
  void* args[] = {(void*)&a};
  if (fit) {  // only asks how many chunks of this size an SM holds
    const void* k = (const void*)k_wave_sweep<SWEEP, WP, G, true, WIDE>;
    *fit = 0;
    if (vals > kSmemMax) return UFVM_OK;
    if (vals > 40 * 1024) UFVM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)vals));
    UFVM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(fit, k, 32 * G, vals));
    return UFVM_OK;
  }
  if (vals <= kSmemMax)
    return launch_coop((const void*)k_wave_sweep<SWEEP, WP, G, true, WIDE>, a.chunks > 1, a.chunks, 32 * G, vals, c.stream, args);
  UFVM_CHECK(dalloc(c.wloc, (size_t)a.chunks * (a.B + 1)));
  a.loc = c.wloc.p;
  return launch_coop((const void*)k_wave_sweep<SWEEP, WP, G, false, WIDE>, a.chunks > 1, a.chunks, 32 * G, 0, c.stream, args);
}

// Registers for the widest row of the sweep (a row takes as many subtractions one after another as
// it has register entries, so a narrow matrix gets a narrow kernel); rows wider than the widest
// kernel read the rest in their turn (`rest`: some rows go past their ELL copy).
template <int SWEEP>
int sweep_by_width(LinCtx& c, WaveArgs& a, int width, bool rest = false, int* fit = nullptr) {
  if (width <= 2) return launch_sweep<SWEEP, 2, 16, 0>(c, a, fit);
  if (width <= 4) return launch_sweep<SWEEP, 4, 16, 0>(c, a, fit);
  if (width <= 6) return launch_sweep<SWEEP, 6, 16, 0>(c, a, fit);
  if (width <= 10) return launch_sweep<SWEEP, 10, 16, 0>(c, a, fit);
  if (width <= 16) return launch_sweep<SWEEP, 16, 16, 0>(c, a, fit);
  if constexpr (SWEEP != SWEEP_FACT)
    if (rest || width > kWideRows) return launch_sweep<SWEEP, 24, 8, 2>(c, a, fit);
  return launch_sweep<SWEEP, 24, 8, 1>(c, a, fit);
}

int kind_width(const Level& L, int kind) {
  return kind == SELL_ILU_FWD ? L.waveW[1] : (kind == SELL_ILU_BWD ? L.waveW[2] : L.waveW[0]);
}

// The copy's width: the widest row's, unless a few rows are so much wider than the others that the copy
// would be many times the matrix (one row coupled to 20,000 others: 4.8 GB a copy, and a call spent
// 0.2 s on them). Those rows' entries past kEllWide are read from the matrix. The small-level kernel's
// levels are copied whole (2,048 rows: 50 MB at most).
constexpr int kEllWide = 64;
int sell_width(const Level& L, int kind) {
  const int W = kind_width(L, kind);
  const bool whole = W <= kEllWide || small_level(L) || (long long)W * L.n <= 4ll * L.nnz;
  return whole ? W : kEllWide;
}

template <int KIND>
int sell_prepare(LinCtx& c, Level& L) {
  const int n = L.n;
  const int dir = (KIND == SELL_GS_FWD || KIND == SELL_ILU_FWD) ? 0 : 1;
  const int* rows = L.waveRows.p + (size_t)dir * n;
  const int W = sell_width(L, KIND);
  if (!L.sell_valid[KIND]) {
    const size_t cap = std::max<size_t>((size_t)W * n, 1);
    UFVM_CHECK(dalloc(L.sellCol[KIND], cap));
    UFVM_CHECK(dalloc(L.sellA[KIND], cap));
    k_wave_fill<KIND, true><<<nblocks(n), kBlock, 0, c.stream>>>(n, L.waveB, rows, L.rowptr.p, L.col.p, L.lord.p,
                                                                L.anb.p, W, L.sellCol[KIND].p, L.sellA[KIND].p);
    UFVM_LAUNCH_CHECK();
    L.sell_valid[KIND] = true;
    L.sell_epoch[KIND] = c.factor_epoch;
  } else if (c.factor_epoch == 0 || L.sell_epoch[KIND] != c.factor_epoch) {
    // the copied coefficients follow the matrix: once per AMG solve or smoother call, else every time
    k_wave_fill<KIND, false><<<nblocks(n), kBlock, 0, c.stream>>>(n, L.waveB, rows, L.rowptr.p, L.col.p, L.lord.p,
                                                                 L.anb.p, W, L.sellCol[KIND].p, L.sellA[KIND].p);
    UFVM_LAUNCH_CHECK();
    L.sell_epoch[KIND] = c.factor_epoch;
  }
  return UFVM_OK;
}

void pass_args(const Level& L, PassArgs& f, PassArgs& b) {
  f.rows = L.waveRows.p; b.rows = L.waveRows.p + L.n;
  f.plev = L.waveLev.p; b.plev = L.waveLev.p + L.n;
  f.task = L.waveTask.p; b.task = L.waveTask.p + (size_t)L.waveChunks * (L.waveB + 1);
  f.ntask = L.waveNtask.p; b.ntask = L.waveNtask.p + L.waveChunks;
}

// Arguments common to the sweeps; the published arrays are preset to "not yet" when more than
// one chunk uses them.
int wave_args(LinCtx& c, Level& L, WaveArgs& a, int passes) {
  const size_t n = (size_t)L.n;
  UFVM_CHECK(dalloc(c.wpub, L.waveChunks > 1 ? 2 * n : 1));
  if (L.waveChunks > 1) UFVM_CUDA(cudaMemsetAsync(c.wpub.p, 0xff, passes * n * sizeof(double), c.stream));
  a = WaveArgs{};
  a.n = L.n; a.chunks = L.waveChunks; a.B = L.waveB;
  a.rp = L.rowptr.p; a.col = L.col.p; a.tpos = L.tpos.p; a.lord = L.lord.p;
  a.ac = L.ac.p; a.anb = L.anb.p; a.bc = L.bc.p;
  a.x = L.dphi.p; a.dc = L.dc.p; a.rc = L.rc.p;
  a.err = c.berr.p;
  pass_args(L, a.f, a.b);
  a.f.pub = c.wpub.p;
  a.b.pub = L.waveChunks > 1 ? c.wpub.p + n : c.wpub.p;
  return UFVM_OK;
}

void use_sell(const Level& L, PassArgs& P, int kind) {
  P.scol = L.sellCol[kind].p;
  P.sa = L.sellA[kind].p;
  P.W = sell_width(L, kind);
}

}  // namespace

// Chunk sizes. Up to kOneChunk rows one CTA does the whole level: no hop between chunks (about 0.8
// us each, from a store in one CTA to the use of the value in another). Larger levels start from
// chunks of kChunkRows rows, at most one chunk per SM; where such a chunk has few rows per
// dependency level, its warps wait for one another anyway and larger chunks save hops, as long as
// the level keeps some chunks. Measured, forward plus backward Gauss-Seidel / DILU sweep in us, by
// rows per chunk: 250 x 250 grid (8 rows per level in 2048) 427 / 324 at 2048, 346 / 264 at 4096,
// 349 / 266 at 8192; 64^3 grid (21 rows) 639 / 492, 614 / 458, 413 / 321; 136,080 tets (256 rows)
// 294 / 246, 411 / 333, 579 / 463; 127 x 129 grid 194 / 155, 199 / 159, 213 / 185.
// The other way round, a level of more than kChunkRows rows per SM whose chunks have many rows per
// dependency level (256 and more) is cut into up to two chunks per SM, where an SM holds two: 517,000
// tets (452 rows) 853 / 610 with 148 chunks, 619 / 532 with 253; 1,029,000 tets (740 rows) 1713 / 1212
// and 1134 / 850 (a launch per level over all SMs: 1447 / 1346).
constexpr int kOneChunk = 8192, kChunkRows = 2048, kDeepRows = 8192, kDeepWidth = 64, kDeepChunks = 8, kWideWidth = 256;

// Chunks of `rows` rows that an SM holds of every sweep on these widths.
int chunks_per_sm(LinCtx& c, const int* width, int rows, int* fit) {
  WaveArgs a{};
  a.B = rows;
  int f[3];
  UFVM_CHECK(sweep_by_width<SWEEP_GS>(c, a, width[0], false, &f[0]));
  UFVM_CHECK(sweep_by_width<SWEEP_FACT>(c, a, width[1], false, &f[1]));
  UFVM_CHECK(sweep_by_width<SWEEP_ILU>(c, a, std::max(width[1], width[2]), false, &f[2]));
  *fit = std::min(f[0], std::min(f[1], f[2]));
  return UFVM_OK;
}

WaveShape wave_shape(int n, int nsm) {
  WaveShape s;
  if (n > kOneChunk) s.chunks = std::min(std::max(1, nsm), (n + kChunkRows - 1) / kChunkRows);
  s.rows = (n + s.chunks - 1) / s.chunks;
  s.chunks = (n + s.rows - 1) / s.rows;
  return s;
}

// Chunks of more than about 7,000 rows (levels of more than a million) keep their counters in global
// memory while their levels are found, and every look at an open row is a load from the L2 then: the
// 4,000 levels of a 2000 x 2000 grid took more than 4 s, by relaxation a whole Gauss-Seidel call takes
// 0.36 s. Long thin orders turn it round (a pass over all rows for every level), so the relaxation ends
// after this many passes and leaves them to the kernel: 23 s for a chain of 3.2 million rows.
constexpr int kRelaxPasses = 1 << 15;

int wave_build(LinCtx& c, Level& L) {
  if (L.sched_valid) return UFVM_OK;
  const int n = L.n;
  UFVM_CHECK(c.ensure(n));
  UFVM_CHECK(dalloc(c.wlvl, 2 * (size_t)n));
  UFVM_CHECK(dalloc(L.waveRows, 2 * (size_t)n));
  UFVM_CHECK(dalloc(L.waveLev, 2 * (size_t)n));
  UFVM_CHECK(dalloc(L.tpos, std::max(L.nnz, 1)));
  UFVM_CHECK(dalloc(L.lord, std::max(L.nnz, 1)));
  // both directions of all chunks are resident in one launch (two CTAs of 512 threads per SM)
  WaveShape w = wave_shape(n, c.nsm);
  bool pattern = false, sized = false, relaxed = false, oneway = false;
  int given = 0;  // the levels are known (a second pass only sorts them into other chunks)
  for (;;) {
    UFVM_CHECK(dalloc(L.waveTask, 2 * (size_t)w.chunks * (w.rows + 1)));
    UFVM_CHECK(dalloc(L.waveNtask, 2 * (size_t)w.chunks));
    SchedArgs a{};
    a.n = n; a.nnz = L.nnz; a.chunks = w.chunks; a.B = w.rows;
    const size_t room = (w.chunks == 1 ? kSmemMax : kSmemMax / 2) / sizeof(int);
    const size_t want = std::max<size_t>(w.rows, 4096);
    a.smem_levels = 2 * ((size_t)w.rows + want) <= room;
    if (!a.smem_levels && !given && !relaxed) {
      bool done = false;
      UFVM_CHECK(relax_levels(c, L, false, kRelaxPasses, &done));
      relaxed = true;
      given = done;
    }
    a.hist_cap = (int)std::min(room / 2, want);
    a.ghist_cap = 0;
    if (w.chunks == 1 && a.hist_cap < n) {  // one chunk: any range of levels fits n counters
      UFVM_CHECK(dalloc(c.wghist, 4 * (size_t)n));
      a.ghist = c.wghist.p;
      a.ghist_cap = n;
    }
    a.rp = L.rowptr.p; a.col = L.col.p;
    UFVM_CHECK(dalloc(c.wext, 2 * (size_t)std::max(L.nnz, 1)));
    a.ext = c.wext.p;
    if (!a.smem_levels) {
      UFVM_CHECK(dalloc(c.wwork, 4 * (size_t)n));
      a.work = c.wwork.p;
    }
    a.lvl = c.wlvl.p; a.rows = L.waveRows.p; a.plev = L.waveLev.p;
    a.task = L.waveTask.p; a.ntask = L.waveNtask.p;
    a.flags = c.iflag.p + 8;
    a.given = given;
    if (!given) UFVM_CUDA(cudaMemsetAsync(c.wlvl.p, 0xff, 2 * (size_t)n * sizeof(int), c.stream));
    UFVM_CUDA(cudaMemsetAsync(c.iflag.p + 8, 0, (pattern ? 2 : 8) * sizeof(int), c.stream));
    if (pattern) UFVM_CUDA(cudaMemsetAsync(c.iflag.p + 14, 0, 2 * sizeof(int), c.stream));
    if (!pattern) {
      k_wave_pattern<<<nblocks(n), kBlock, 0, c.stream>>>(n, L.rowptr.p, L.col.p, L.tpos.p, L.lord.p, c.iflag.p + 10);
      UFVM_LAUNCH_CHECK();
      pattern = true;
    }
    void* args[] = {(void*)&a};
    const size_t smem = 2 * ((a.smem_levels ? (size_t)w.rows : 0) + (size_t)a.hist_cap) * sizeof(int);
    // (with the levels given the chunks do not wait for one another)
    UFVM_CHECK(launch_coop((const void*)k_wave_schedule, w.chunks > 1 && !given, 2 * w.chunks, kSchedBlock, smem, c.stream,
                           args));
    int h[7] = {0, 0, 0, 0, 0, 0, 0};
    UFVM_CUDA(cudaMemcpyAsync(h, c.iflag.p + 8, sizeof(h), cudaMemcpyDeviceToHost, c.stream));
    UFVM_CUDA(cudaStreamSynchronize(c.stream));
    if (h[0]) {
      set_error("level schedule: a bounded wait gave up");
      return UFVM_E_TIMEOUT;
    }
    for (int k = 0; k < 3; ++k) L.waveW[k] = h[2 + k];
    if (h[5] && !oneway) {  // not structurally symmetric: levels by relaxation, then sort them
      bool done = false;
      oneway = true;
      UFVM_CHECK(relax_levels(c, L, oneway, 0, &done));
      given = 1;
      continue;
    }
    given = 1;
    if (h[1]) {
      // some chunk's rows spread over more levels than its counters: sort the whole level in one
      // chunk instead (a matrix whose natural order mixes unrelated parts)
      w.chunks = 1;
      w.rows = n;
      sized = true;
      continue;
    }
    if (!sized && w.rows > kChunkRows && w.chunks > 1 && n > (long long)kWideWidth * h[6]) {
      sized = true;
      const int chunks = std::min(2 * c.nsm, (n + kChunkRows - 1) / kChunkRows), rows = (n + chunks - 1) / chunks;
      int fit = 0;
      UFVM_CHECK(chunks_per_sm(c, L.waveW, rows, &fit));
      if (fit >= 2) {
        w.rows = rows;
        w.chunks = (n + rows - 1) / rows;
        continue;
      }
    }
    if (!sized && w.chunks > 1 && n <= (long long)kDeepWidth * h[6]) {
      const int rows = std::min(kDeepRows, n / kDeepChunks);
      sized = true;
      if (rows > w.rows) {
        w.chunks = (n + rows - 1) / rows;
        w.rows = (n + w.chunks - 1) / w.chunks;
        w.chunks = (n + w.rows - 1) / w.rows;
        continue;
      }
    }
    break;
  }
  L.waveChunks = w.chunks;
  L.waveB = w.rows;
  L.waveOneway = oneway;
  L.sched_valid = true;
  L.dc_epoch = 0;
  for (int k = 0; k < 4; ++k) L.sell_valid[k] = false;
  return UFVM_OK;
}

int wave_gs(LinCtx& c, Level& L, const SmoothCtl* ctl) {
  UFVM_CHECK(wave_build(c, L));
  UFVM_CHECK(sell_prepare<SELL_GS_FWD>(c, L));
  UFVM_CHECK(sell_prepare<SELL_GS_BWD>(c, L));
  WaveArgs a;
  UFVM_CHECK(wave_args(c, L, a, 2));
  use_sell(L, a.f, SELL_GS_FWD);
  use_sell(L, a.b, SELL_GS_BWD);
  a.f.other = L.dphi.p;  // rows of later chunks keep their old value until the end
  if (L.waveOneway && L.waveChunks > 1) {
    // not for a row that no row of theirs waits for: its chunk reads the old values from a copy
    UFVM_CHECK(dalloc(c.wold, L.n));
    UFVM_CUDA(cudaMemcpyAsync(c.wold.p, L.dphi.p, L.n * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
    a.f.other = c.wold.p;
  }
  a.b.other = a.f.pub;   // rows of earlier chunks as the forward pass left them
  a.ctl = ctl;
  return sweep_by_width<SWEEP_GS>(c, a, L.waveW[0], a.f.W < L.waveW[0]);
}

int wave_ilu_factor(LinCtx& c, Level& L, int quirks) {
  UFVM_CHECK(wave_build(c, L));
  WaveArgs a;
  UFVM_CHECK(wave_args(c, L, a, 1));
  a.quirks = quirks;
  return sweep_by_width<SWEEP_FACT>(c, a, L.waveW[1]);
}

int wave_ilu(LinCtx& c, Level& L, const SmoothCtl* ctl) {
  UFVM_CHECK(wave_build(c, L));
  UFVM_CHECK(sell_prepare<SELL_ILU_FWD>(c, L));
  UFVM_CHECK(sell_prepare<SELL_ILU_BWD>(c, L));
  UFVM_CHECK(dalloc(L.rc, L.n));
  WaveArgs a;
  UFVM_CHECK(wave_args(c, L, a, 2));
  use_sell(L, a.f, SELL_ILU_FWD);
  use_sell(L, a.b, SELL_ILU_BWD);
  a.res = L.r.p;
  a.ctl = ctl;
  return sweep_by_width<SWEEP_ILU>(c, a, std::max(L.waveW[1], L.waveW[2]), a.f.W < L.waveW[1] || a.b.W < L.waveW[2]);
}

int wave_prepare_gs(LinCtx& c, Level& L, PassArgs& f, PassArgs& b) {
  UFVM_CHECK(wave_build(c, L));
  UFVM_CHECK(sell_prepare<SELL_GS_FWD>(c, L));
  UFVM_CHECK(sell_prepare<SELL_GS_BWD>(c, L));
  pass_args(L, f, b);
  use_sell(L, f, SELL_GS_FWD);
  use_sell(L, b, SELL_GS_BWD);
  return UFVM_OK;
}

int wave_prepare_ilu(LinCtx& c, Level& L, PassArgs& f, PassArgs& b) {
  UFVM_CHECK(wave_build(c, L));
  UFVM_CHECK(sell_prepare<SELL_ILU_FWD>(c, L));
  UFVM_CHECK(sell_prepare<SELL_ILU_BWD>(c, L));
  UFVM_CHECK(dalloc(L.rc, L.n));
  UFVM_CHECK(dalloc(L.dc, L.n));
  pass_args(L, f, b);
  use_sell(L, f, SELL_ILU_FWD);
  use_sell(L, b, SELL_ILU_BWD);
  return UFVM_OK;
}

int wave_check(LinCtx& c) {
  int err = 0;
  UFVM_CUDA(cudaMemcpyAsync(&err, c.berr.p, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  UFVM_CUDA(cudaStreamSynchronize(c.stream));
  if (err) {
    UFVM_CUDA(cudaMemsetAsync(c.berr.p, 0, sizeof(int), c.stream));
    set_error("a bounded wait gave up in a natural-order sweep");
    return UFVM_E_TIMEOUT;
  }
  return UFVM_OK;
}

}  // namespace ufvm
