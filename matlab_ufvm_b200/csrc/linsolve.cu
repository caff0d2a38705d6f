// linsolve.cu -- residual, smoothers and grid transfers of uFVM's linear solve.
//
//   residual      compute/cfdComputeResidualsArray.m:9-17
//   GS ('SOR')    solve/cfdSolveSOR.m:13-29   (natural order: chunked wavefronts, wave.cu)
//   DILU ('ILU')  solve/cfdFactorizeILU.m:5-47, solve/cfdSolveILU.m:18-93 (wave.cu)
//   MCGS          multicolour symmetric GS (greedy first-fit colouring in natural order)
//   smoother loop solve/cfdSolveAlgebraicSystem.m:11-66
//   restriction   solve/AMG/cfdUpdateRHS.m:10-17, prolongation cfdCorrectFinerLevelSolution.m:11-14
//
// Roofline: residual / one GS half-sweep are HBM-bound; algorithmic bytes per row =
// 8 (ac) + 8 (bc) + 8 (x) + 8 (r or x write) + 4 (rowptr) + nnz_row * (8 anb + 4 col).
#include <atomic>
#include "linsolve.cuh"
#include "small.cuh"
#include "wave.cuh"

namespace ufvm {

int LinCtx::ensure(int n) {
  const int nb = nblocks(n) + 2;
  UFVM_CHECK(dalloc(part, std::max(nb, 64) * 2));
  UFVM_CHECK(dalloc(iflag, 16));
  if (!ctl.p) {
    UFVM_CHECK(dalloc(ctl, 1));
    UFVM_CUDA(cudaMemsetAsync(ctl.p, 0, sizeof(SmoothCtl), stream));
  }
  UFVM_CHECK(dalloc(iscan, nblocks(n, 1024) * 2 + 64));
  if (nsm <= 0) {
    int dev = 0;
    UFVM_CUDA(cudaGetDevice(&dev));
    UFVM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  }
  if (!berr.p) {
    UFVM_CHECK(dalloc(berr, 2));
    UFVM_CUDA(cudaMemsetAsync(berr.p, 0, 2 * sizeof(int), stream));
    berr_rows = 0;
  }
  if (n > berr_rows) {
    UFVM_CUDA(cudaMemcpyAsync(berr.p + 1, &n, sizeof(int), cudaMemcpyHostToDevice, stream));
    berr_rows = n;
  }
  return UFVM_OK;
}

void LinCtx::release() {
  dfree(part); dfree(ctl); dfree(iflag); dfree(iscan); dfree(berr);
  dfree(wpub); dfree(wloc); dfree(wold); dfree(small); dfree(wlvl); dfree(wghist); dfree(wwork); dfree(wext);
}

EpochScope::EpochScope(LinCtx& ctx) : c(ctx), own(ctx.factor_epoch == 0) {
  static std::atomic<unsigned long long> epochs{0};
  if (own) c.factor_epoch = epochs.fetch_add(1) + 1;
}

// ---------------------------------------------------------------- scan (exclusive, int)
__global__ void k_scan_block(const int* __restrict__ in, int* out, int n, int* bsum) {
  __shared__ int sh[1024];
  const int base = blockIdx.x * 1024;
  for (int t = threadIdx.x; t < 1024; t += blockDim.x) sh[t] = base + t < n ? in[base + t] : 0;
  __syncthreads();
  // Hillis-Steele on 1024 entries with 1024 threads
  for (int o = 1; o < 1024; o <<= 1) {
    int v = 0;
    if (threadIdx.x >= o) v = sh[threadIdx.x - o];
    __syncthreads();
    sh[threadIdx.x] += v;
    __syncthreads();
  }
  const int incl = sh[threadIdx.x];
  const int x = base + threadIdx.x < n ? in[base + threadIdx.x] : 0;
  if (base + threadIdx.x < n) out[base + threadIdx.x] = incl - x;
  if (threadIdx.x == 1023) bsum[blockIdx.x] = incl;
}

__global__ void k_scan_add(int* out, int n, const int* __restrict__ boff) {
  const int i = blockIdx.x * 1024 + threadIdx.x;
  if (i < n) out[i] += boff[blockIdx.x];
}

static int scan_rec(LinCtx& c, const int* in, int* out, int n, int* tmp, size_t tmpcap) {
  const int nb = nblocks(n, 1024);
  if ((size_t)(2 * nb + 2) > tmpcap) { set_error("scan scratch too small"); return UFVM_E_INVALID; }
  int* bsum = tmp;
  int* boff = tmp + nb;
  k_scan_block<<<nb, 1024, 0, c.stream>>>(in, out, n, bsum);
  UFVM_LAUNCH_CHECK();
  if (nb == 1) return UFVM_OK;
  UFVM_CHECK(scan_rec(c, bsum, boff, nb, tmp + 2 * nb, tmpcap - 2 * nb));
  k_scan_add<<<nb, 1024, 0, c.stream>>>(out, n, boff);
  UFVM_LAUNCH_CHECK();
  return UFVM_OK;
}

__global__ void k_scan_total(const int* __restrict__ in, const int* __restrict__ out, int n, int* total_slot) {
  *total_slot = n > 0 ? out[n - 1] + in[n - 1] : 0;
}

// out has n + 1 entries; out[n] = total.
int scan_exclusive(LinCtx& c, const int* in, int* out, int n, int* total_host) {
  size_t need = 0;
  for (int m = n; m > 1; m = nblocks(m, 1024)) need += 2 * (size_t)nblocks(m, 1024) + 2;
  need += 8;
  UFVM_CHECK(dalloc(c.iscan, std::max(need, c.iscan.n)));
  if (n > 0) UFVM_CHECK(scan_rec(c, in, out, n, c.iscan.p, c.iscan.n));
  k_scan_total<<<1, 1, 0, c.stream>>>(in, out, n, out + n);
  UFVM_LAUNCH_CHECK();
  if (total_host) {
    UFVM_CUDA(cudaMemcpyAsync(total_host, out + n, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    UFVM_CUDA(cudaStreamSynchronize(c.stream));
  }
  return UFVM_OK;
}

// ---------------------------------------------------------------- residual
// One row per thread. Everything a row needs apart from the neighbour values (its row
// pointers, bc, ac, x_i) is loaded at once, then its entries kResChunk at a time (the L1
// serves the warp's neighbouring rows from the same sectors), then the neighbour values:
// three dependent memory round trips per row. v = bc - ac x_i, then v = v - anb x_j in cconn
// order, with each product rounded before the subtraction as in the sequential loop.
constexpr int kResChunk = 4;
constexpr int kResBlock = 128;

__device__ __forceinline__ double row_residual(int i, const int* __restrict__ rp, const int* __restrict__ col,
                                               const double* __restrict__ ac, const double* __restrict__ anb,
                                               const double* __restrict__ bc, const double* __restrict__ x) {
  const int k0 = rp[i], k1 = rp[i + 1];
  double v = bc[i] - ac[i] * x[i];
  for (int k = k0; k < k1; k += kResChunk) {
    double p[kResChunk];
#pragma unroll
    for (int t = 0; t < kResChunk; ++t) p[t] = k + t < k1 ? anb[k + t] * x[col[k + t]] : 0.0;
#pragma unroll
    for (int t = 0; t < kResChunk; ++t)
      if (k + t < k1) v = v - p[t];
  }
  return v;
}

__global__ void __launch_bounds__(kResBlock) k_residual(int n, const int* __restrict__ rp,
                                                        const int* __restrict__ col, const double* __restrict__ ac,
                                                        const double* __restrict__ anb,
                                                        const double* __restrict__ bc,
                                                        const double* __restrict__ x, double* __restrict__ r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = row_residual(i, rp, col, ac, anb, bc, x);
}

int residual(LinCtx& c, const Level& L, const double* x, double* r) {
  k_residual<<<nblocks(L.n, kResBlock), kResBlock, 0, c.stream>>>(L.n, L.rowptr.p, L.col.p, L.ac.p, L.anb.p,
                                                                   L.bc.p, x, r);
  UFVM_LAUNCH_CHECK();
  return UFVM_OK;
}

// The stopping test of a smoother call on the device: r = b - A x (kept in r: the DILU substitution
// and the restriction start from it), block sums of |r|, and, in the last block to finish, their sum
// in a fixed order and the reference's rule (solve/cfdSolveAlgebraicSystem.m:38-46). `first`: before
// the first sweep; otherwise after a sweep, and nothing is done once the call has stopped.
__global__ void __launch_bounds__(kBlock) k_smooth_test(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                                        const double* __restrict__ ac, const double* __restrict__ anb,
                                                        const double* __restrict__ bc, const double* __restrict__ x,
                                                        double* r, double* part, SmoothCtl* ctl, int first, int n_iter,
                                                        double rrf) {
  __shared__ double sh[32];
  __shared__ bool s_last;
  if (!first && !*(volatile int*)&ctl->active) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0.0;
  if (i < n) {
    const double ri = row_residual(i, rp, col, ac, anb, bc, x);
    r[i] = ri;
    v = fabs(ri);
  }
  v = block_reduce<0>(v, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = v;
    __threadfence();
    s_last = atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  v = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) v = v + __ldcg(part + k);
  v = block_reduce<0>(v, sh);
  if (threadIdx.x == 0) {
    const double m = v / n;
    ctl->sum = v;
    ctl->r1 = m;
    if (first) {
      ctl->r0 = m;
      ctl->iters = 0;
    } else {
      ctl->iters += 1;
    }
    ctl->active = ctl->iters < n_iter && m > rrf * ctl->r0 ? 1 : 0;
    ctl->ticket = 0;
  }
}

static int smooth_test(LinCtx& c, Level& L, bool first, int n_iter, double rrf) {
  k_smooth_test<<<nblocks(L.n), kBlock, 0, c.stream>>>(L.n, L.rowptr.p, L.col.p, L.ac.p, L.anb.p, L.bc.p, L.dphi.p,
                                                       L.r.p, c.part.p, c.ctl.p, first ? 1 : 0, n_iter, rrf);
  UFVM_LAUNCH_CHECK();
  return UFVM_OK;
}

int read_ctl(LinCtx& c, SmoothCtl* out) {
  int err = 0;
  UFVM_CUDA(cudaMemcpyAsync(out, c.ctl.p, sizeof(SmoothCtl), cudaMemcpyDeviceToHost, c.stream));
  UFVM_CUDA(cudaMemcpyAsync(&err, c.berr.p, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  UFVM_CUDA(cudaStreamSynchronize(c.stream));
  return err ? wave_check(c) : UFVM_OK;
}

int sum_abs_residual(LinCtx& c, Level& L, double* out_host) {
  UFVM_CHECK(c.ensure(L.n));
  UFVM_CHECK(dalloc(L.r, L.n));
  UFVM_CHECK(smooth_test(c, L, true, 0, 0.0));
  SmoothCtl h;
  UFVM_CHECK(read_ctl(c, &h));
  *out_host = h.sum;
  return UFVM_OK;
}

// ---------------------------------------------------------------- natural-order sweeps (wave.cu)
int build_schedule(LinCtx& c, Level& L) { return wave_build(c, L); }
int check_barrier(LinCtx& c) { return wave_check(c); }
int gs_sweep(LinCtx& c, Level& L) {
  UFVM_CHECK(c.ensure(L.n));
  return wave_gs(c, L, nullptr);
}

int ilu_factor(LinCtx& c, Level& L, int quirks) {
  UFVM_CHECK(wave_build(c, L));
  // within one AMG solve the level's matrix is fixed: the factor already computed is the one
  // the reference recomputes on every smoother call (solve/cfdSolveAlgebraicSystem.m:29-33)
  if (c.factor_epoch != 0 && L.dc_epoch == c.factor_epoch && L.dc_quirks == quirks && L.dc.p) return UFVM_OK;
  UFVM_CHECK(dalloc(L.dc, L.n));
  UFVM_CHECK(wave_ilu_factor(c, L, quirks));
  L.dc_epoch = c.factor_epoch;
  L.dc_quirks = quirks;
  return UFVM_OK;
}

int ilu_sweep(LinCtx& c, Level& L) {
  UFVM_CHECK(c.ensure(L.n));
  UFVM_CHECK(dalloc(L.r, L.n));
  UFVM_CHECK(residual(c, L, L.dphi.p, L.r.p));
  return wave_ilu(c, L, nullptr);
}

// ---------------------------------------------------------------- colouring + MCGS
// Greedy first-fit colouring in natural order: a row takes the smallest colour unused by its
// lower-index neighbours once all of them are coloured. A row's colour depends only on its lower
// neighbours' final colours, so the result is the sequential greedy colouring whatever the order in
// which rows are reached. One launch: a thread takes its rows in ascending order and waits at each
// for the lower neighbours that are not coloured yet, so the lowest uncoloured row is always some
// thread's current one, and the launch is cooperative (all blocks resident). A launch per dependency
// round took 7 us a round over all rows. As many threads as the GPU holds: a thread's next row waits
// for its current one, so rows further apart than the threads are not reached side by side, and the
// wavefront of a large grid is wider than that. Smoother calls of one sweep, ms, a launch per round /
// 64 blocks / all: 300 x 300 grid 6.8 / 1.4 / 0.9, 100^3 13.0 / 6.6 / 1.8, 10000 x 100 177 / 202 / 30,
// 2000 x 2000 212 / 316 / 25; a chain of 200,000 rows (latency alone) 1488 / 138 / 141.
// out[0]: number of colours; cnt[c]: rows of colour c; done: rows coloured so far. A wait that has
// reached its bound gives up only if no row was coloured meanwhile: rows of more than 64 colours search
// theirs colour by colour, and 600 rows that are all coupled take 7 s, which the last of them waits for.
constexpr int kColorHist = 256;       // colours counted in shared memory
__global__ void __launch_bounds__(256) k_color_flow(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                                    int* color, int* cnt, int* out, int* done, int* err) {
  __shared__ int hist[kColorHist], top;
  for (int i = threadIdx.x; i < kColorHist; i += blockDim.x) hist[i] = 0;
  if (threadIdx.x == 0) top = 0;
  __syncthreads();
  const int nth = gridDim.x * blockDim.x;
  long long t0 = clock64();
  unsigned spins = 0;
  int i = blockIdx.x * blockDim.x + threadIdx.x, k = 0, e = 0, seen = -1;
  if (i < n) { k = rp[i]; e = rp[i + 1]; }
  unsigned long long used = 0;
  bool big = false;
  while (__any_sync(0xffffffffu, i < n)) {
    if (i < n) {
      bool wait = false;
      for (; k < e; ++k) {
        const int j = col[k];
        if (j >= i) continue;
        const int cj = ld_flag(color + j);
        if (cj < 0) { wait = true; break; }
        if (cj < 64) used |= 1ull << cj;
        else big = true;
      }
      if (!wait) {
        int c = ~used ? __ffsll(~used) - 1 : 64;
        if (c >= 64 && big)
          for (;; ++c) {
            bool hit = false;
            for (k = rp[i]; k < e && !hit; ++k) hit = col[k] < i && ld_flag(color + col[k]) == c;
            if (!hit) break;
          }
        st_flag(color + i, c);
        atomicAdd(c < kColorHist ? hist + c : cnt + c, 1);
        atomicMax(&top, c + 1);
        atomicAdd(done, 1);
        i += nth;
        t0 = clock64();
        used = 0;
        big = false;
        if (i < n) { k = rp[i]; e = rp[i + 1]; }
      } else if ((++spins & 255u) == 0 && clock64() - t0 > kFlagClocks) {
        const int now = ld_flag(done);
        if (now == seen) {
          atomicExch(err, 1);
          i = n;
        }
        seen = now;
        t0 = clock64();
      }
    }
    __syncwarp();
  }
  __syncthreads();
  for (int c = threadIdx.x; c < kColorHist; c += blockDim.x)
    if (hist[c]) atomicAdd(cnt + c, hist[c]);
  if (threadIdx.x == 0) atomicMax(out, top);
}

// The rows of one colour per block, in ascending order
constexpr int kRowsBlock = 1024;
__global__ void __launch_bounds__(kRowsBlock) k_color_rows(int n, const int* __restrict__ color,
                                                           const int* __restrict__ start, int* rows) {
  __shared__ int wsum[kRowsBlock / 32];
  const int c = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = start[c];
  const int end = start[c + 1];
  for (int i0 = 0; i0 < n && base < end; i0 += 4 * kRowsBlock) {
    const int i = i0 + 4 * threadIdx.x;
    int m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) m |= (i + k < n && color[i + k] == c) << k;
    int s = __popc(m);
    const int own = s;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
      const int v = __shfl_up_sync(0xffffffffu, s, d);
      if (lane >= d) s += v;
    }
    if (lane == 31) wsum[warp] = s;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < kRowsBlock / 32; ++w) {
      before += w < warp ? wsum[w] : 0;
      total += wsum[w];
    }
    int p = base + before + s - own;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (m >> k & 1) rows[p++] = i + k;
    base += total;
    __syncthreads();
  }
}

int build_coloring(LinCtx& c, Level& L) {
  if (L.color_valid) return UFVM_OK;
  UFVM_CHECK(c.ensure(L.n));
  int n = L.n;
  UFVM_CHECK(dalloc(L.color, n));
  UFVM_CUDA(cudaMemsetAsync(L.color.p, 0xff, n * sizeof(int), c.stream));
  struct Scratch : DArr<int> {
    ~Scratch() { dfree(*this); }
  } cnt;  // [0]: number of colours; then rows per colour; last: rows coloured
  UFVM_CHECK(dalloc<int>(cnt, (size_t)n + 1 + kColorHist));
  UFVM_CUDA(cudaMemsetAsync(cnt.p, 0, ((size_t)n + 1 + kColorHist) * sizeof(int), c.stream));
  int *hist = cnt.p + 1, *done = cnt.p + n + kColorHist;
  {
    void* args[] = {(void*)&n, (void*)&L.rowptr.p, (void*)&L.col.p, (void*)&L.color.p, (void*)&hist, (void*)&cnt.p,
                    (void*)&done, (void*)&c.berr.p};
    int fit = 0;
    UFVM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_color_flow, 256, 0));
    const int grid = std::max(1, std::min(fit * c.nsm, (n + 255) / 256));
    UFVM_CUDA(cudaLaunchCooperativeKernel((const void*)k_color_flow, dim3(grid), dim3(256), args, 0, c.stream));
  }
  std::vector<int> h(1 + kColorHist);
  UFVM_CUDA(cudaMemcpyAsync(h.data(), cnt.p, h.size() * sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  UFVM_CHECK(check_barrier(c));  // waits for the copy as well
  const int nc = h[0];
  if (nc > kColorHist) {
    h.resize(1 + (size_t)nc);
    UFVM_CUDA(cudaMemcpyAsync(h.data(), cnt.p, h.size() * sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    UFVM_CUDA(cudaStreamSynchronize(c.stream));
  }
  L.ncolor = nc;
  L.h_colorStart.assign(nc + 1, 0);
  for (int q = 0; q < nc; ++q) L.h_colorStart[q + 1] = L.h_colorStart[q] + h[1 + q];
  UFVM_CHECK(dalloc(L.colorStart, nc + 1));
  UFVM_CUDA(cudaMemcpyAsync(L.colorStart.p, L.h_colorStart.data(), (nc + 1) * sizeof(int), cudaMemcpyHostToDevice,
                            c.stream));
  UFVM_CHECK(dalloc(L.colorRows, n));
  k_color_rows<<<nc, kRowsBlock, 0, c.stream>>>(n, L.color.p, L.colorStart.p, L.colorRows.p);
  UFVM_LAUNCH_CHECK();
  UFVM_CUDA(cudaStreamSynchronize(c.stream));
  L.color_valid = true;
  return UFVM_OK;
}

// The plain FP64 multicolour sweep reads a colour-major ELL copy of the matrix: position p
// holds row mcRow[p] (colours ascending, rows ascending inside a colour), entry k of position
// p sits at [k * n + p] (column -1 past the row's end), so a colour's rows are read with
// unit stride. x stays in natural order. Each row evaluates v = bc - sum anb * x in cconn
// order and x = v / ac, the operation order of the CSR sweep: the copy changes no bit.
__global__ void k_row_len_max(int n, const int* __restrict__ rp, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicMax(out, rp[i + 1] - rp[i]);
}

__global__ void k_mc_pattern(int n, int W, const int* __restrict__ mcRow, const int* __restrict__ rp,
                             const int* __restrict__ col, int* mcCol) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int i = mcRow[p], k0 = rp[i], len = rp[i + 1] - k0;
  for (int k = 0; k < W; ++k) mcCol[(size_t)k * n + p] = k < len ? col[k0 + k] : -1;
}

__global__ void k_mc_values(int n, int W, const int* __restrict__ mcRow, const int* __restrict__ rp,
                            const double* __restrict__ ac, const double* __restrict__ anb, double* mcAc,
                            double* mcAnb) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int i = mcRow[p], k0 = rp[i], len = rp[i + 1] - k0;
  mcAc[p] = ac[i];
  for (int k = 0; k < W; ++k) mcAnb[(size_t)k * n + p] = k < len ? anb[k0 + k] : 0.0;
}

__global__ void k_mc_bc(int n, const int* __restrict__ mcRow, const double* __restrict__ bc, double* mcBc) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) mcBc[p] = bc[mcRow[p]];
}

// One colour's rows. The colour kernels of a sweep follow one another as programmatic
// dependent launches: a kernel starts while the previous colour is still running, loads what
// does not depend on x (its rows' positions, bc, ac and the first kMcPre entries, all
// coalesced), and only then waits (griddepcontrol.wait returns once the previous kernel has
// completed and its writes are visible) before it gathers the neighbour values. The entries after
// those are loaded kMcNext at a time: one by one, each behind the test for the row's end, a colour of
// the wider coarse levels took 18 us (136k tetrahedra, mean over the levels), now 8 us.
constexpr int kMcPre = 4, kMcNext = 8;

__global__ void __launch_bounds__(kBlock) k_mc_rows(int cnt, int p0, int n, int W, const int* __restrict__ mcRow,
                                                   const int* __restrict__ mcCol, const double* __restrict__ mcAnb,
                                                   const double* __restrict__ mcAc,
                                                   const double* __restrict__ mcBc, double* x,
                                                   const SmoothCtl* ctl) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (ctl && !ctl->active) {  // no kernel of the sweep changes it
    asm volatile("griddepcontrol.wait;" ::: "memory");  // not to complete before the kernel it follows
    return;
  }
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= cnt) return;
  const int p = p0 + t;
  const int i = mcRow[p];
  const double b = mcBc[p], a = mcAc[p];
  int j[kMcPre];
  double w[kMcPre];
#pragma unroll
  for (int k = 0; k < kMcPre; ++k) {
    j[k] = k < W ? mcCol[(size_t)k * n + p] : -1;
    w[k] = k < W ? mcAnb[(size_t)k * n + p] : 0.0;
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  double xv[kMcPre];
#pragma unroll
  for (int k = 0; k < kMcPre; ++k) xv[k] = j[k] >= 0 ? x[j[k]] : 0.0;
  double v = b;
  bool end = false;
#pragma unroll
  for (int k = 0; k < kMcPre; ++k) {
    end |= j[k] < 0;
    if (!end) v = v - w[k] * xv[k];
  }
  for (int k0 = kMcPre; k0 < W && !end; k0 += kMcNext) {  // kMcNext entries' loads before the first use
    int jn[kMcNext];
    double wn[kMcNext], xn[kMcNext];
#pragma unroll
    for (int k = 0; k < kMcNext; ++k) {
      jn[k] = k0 + k < W ? mcCol[(size_t)(k0 + k) * n + p] : -1;
      wn[k] = k0 + k < W ? mcAnb[(size_t)(k0 + k) * n + p] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kMcNext; ++k) xn[k] = jn[k] >= 0 ? x[jn[k]] : 0.0;
#pragma unroll
    for (int k = 0; k < kMcNext; ++k) {
      end |= jn[k] < 0;
      if (!end) v = v - wn[k] * xn[k];
    }
  }
  x[i] = v / a;
}

static int build_mc_pattern(LinCtx& c, Level& L) {
  if (L.mc_valid) return UFVM_OK;
  UFVM_CHECK(build_coloring(c, L));
  const int n = L.n;
  UFVM_CHECK(dalloc(L.mcRow, n));
  UFVM_CUDA(cudaMemcpyAsync(L.mcRow.p, L.colorRows.p, n * sizeof(int), cudaMemcpyDeviceToDevice, c.stream));
  UFVM_CUDA(cudaMemsetAsync(c.iflag.p + 4, 0, sizeof(int), c.stream));
  k_row_len_max<<<nblocks(n), kBlock, 0, c.stream>>>(n, L.rowptr.p, c.iflag.p + 4);
  UFVM_LAUNCH_CHECK();
  int W = 0;
  UFVM_CUDA(cudaMemcpyAsync(&W, c.iflag.p + 4, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  UFVM_CUDA(cudaStreamSynchronize(c.stream));
  L.mcW = W;
  const size_t cap = std::max<size_t>((size_t)W * n, 1);
  UFVM_CHECK(dalloc(L.mcCol, cap));
  UFVM_CHECK(dalloc(L.mcAnb, cap));
  UFVM_CHECK(dalloc(L.mcAc, n));
  UFVM_CHECK(dalloc(L.mcBc, n));
  k_mc_pattern<<<nblocks(n), kBlock, 0, c.stream>>>(n, W, L.mcRow.p, L.rowptr.p, L.col.p, L.mcCol.p);
  UFVM_LAUNCH_CHECK();
  L.mc_valid = true;
  L.mc_epoch = 0;
  return UFVM_OK;
}

// Copies the matrix (once per AMG solve, or per smoother call outside one) and the right-hand
// side (every call) into the colour-major layout.
int mcgs_prepare(LinCtx& c, Level& L) {
  UFVM_CHECK(c.ensure(L.n));
  UFVM_CHECK(build_mc_pattern(c, L));
  if (c.factor_epoch == 0 || L.mc_epoch != c.factor_epoch) {
    k_mc_values<<<nblocks(L.n), kBlock, 0, c.stream>>>(L.n, L.mcW, L.mcRow.p, L.rowptr.p, L.ac.p, L.anb.p, L.mcAc.p,
                                                       L.mcAnb.p);
    L.mc_epoch = c.factor_epoch;
  }
  k_mc_bc<<<nblocks(L.n), kBlock, 0, c.stream>>>(L.n, L.mcRow.p, L.bc.p, L.mcBc.p);
  UFVM_LAUNCH_CHECK();
  return UFVM_OK;
}

int mcgs_sweep(LinCtx& c, Level& L, const SmoothCtl* ctl) {
  if (!L.mc_valid) { set_error("mcgs_sweep: layout not prepared"); return UFVM_E_INVALID; }
  // the first colour kernel of the sweep waits for all earlier work the ordinary way; the
  // later ones are programmatic dependents of the colour before them
  int launched = 0;
  // the backward pass starts one colour in: its first colour would repeat the forward pass's
  // last update from the same neighbour values (same bits), so it is skipped
  for (int pass = 0; pass < 2; ++pass) {
    for (int q = pass; q < L.ncolor; ++q) {
      const int col_ = pass == 0 ? q : L.ncolor - 1 - q;
      const int s = L.h_colorStart[col_], cnt = L.h_colorStart[col_ + 1] - s;
      if (cnt <= 0) continue;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(nblocks(cnt));
      cfg.blockDim = dim3(kBlock);
      cfg.stream = c.stream;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[0].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr;
      cfg.numAttrs = launched > 0 ? 1 : 0;
      UFVM_CUDA(cudaLaunchKernelEx(&cfg, k_mc_rows, cnt, s, L.n, L.mcW, (const int*)L.mcRow.p,
                                   (const int*)L.mcCol.p, (const double*)L.mcAnb.p, (const double*)L.mcAc.p,
                                   (const double*)L.mcBc.p, L.dphi.p, ctl));
      ++launched;
    }
  }
  return UFVM_OK;
}

// ---------------------------------------------------------------- smoother loop
// Sweeps are queued ahead of the stopping test, which runs on the device; a sweep queued after the
// call has stopped returns at once. The host reads the result only when its caller wants it, or
// after kAhead sweeps, so that a long call does not queue many empty ones.
constexpr int kAhead = 4, kAheadRead = 2;

int solve_algebraic_system(LinCtx& c, Level& L, int smoother, int n_iter, double rrf, int quirks, double* r0out,
                           double* r1out, int* iters) {
  // the matrix stays the same for the length of the call: its sweeps share the coefficient copies
  // (refilled before every sweep they made 50 sweeps of a million tetrahedra 92.8 ms instead of 90.8)
  EpochScope epoch(c);
  UFVM_CHECK(c.ensure(L.n));
  UFVM_CHECK(dalloc(L.r, L.n));
  const bool want = r0out || r1out || iters;
  SmoothCtl h{};
  bool have = false;
  if (small_level(L)) {
    UFVM_CHECK(small_smooth(c, L, smoother, n_iter, rrf, quirks));
  } else {
    UFVM_CHECK(smooth_test(c, L, true, n_iter, rrf));
    if (smoother == UFVM_SMOOTHER_ILU) UFVM_CHECK(ilu_factor(c, L, quirks));
    else if (smoother != UFVM_SMOOTHER_SOR) UFVM_CHECK(mcgs_prepare(c, L));
    for (int it = 0; it < n_iter;) {
      const int m = std::min(n_iter - it, want ? kAheadRead : kAhead);
      for (int k = 0; k < m; ++k, ++it) {
        if (smoother == UFVM_SMOOTHER_ILU) UFVM_CHECK(wave_ilu(c, L, c.ctl.p));
        else if (smoother == UFVM_SMOOTHER_SOR) UFVM_CHECK(wave_gs(c, L, c.ctl.p));
        else UFVM_CHECK(mcgs_sweep(c, L, c.ctl.p));
        UFVM_CHECK(smooth_test(c, L, false, n_iter, rrf));
      }
      if (it < n_iter || want) {
        UFVM_CHECK(read_ctl(c, &h));
        have = true;
        if (!h.active) break;
      }
    }
  }
  if (want && !have) UFVM_CHECK(read_ctl(c, &h));
  if (r0out) *r0out = h.r0;
  if (r1out) *r1out = h.r1;
  if (iters) *iters = h.iters;
  return UFVM_OK;
}

// ---------------------------------------------------------------- transfers
__global__ void k_restrict(int nc, const int* __restrict__ cs, const int* __restrict__ ch,
                           const double* __restrict__ r, double* bcC) {
  const int P = blockIdx.x * blockDim.x + threadIdx.x;
  if (P >= nc) return;
  double v = 0.0;
  for (int q = cs[P]; q < cs[P + 1]; ++q) v = v + r[ch[q]];
  bcC[P] = v;
}

__global__ void k_prolong(int n, const int* __restrict__ parents, const double* __restrict__ dC, double* dF) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dF[i] = dF[i] + dC[parents[i]];
}

int restrict_residual(LinCtx& c, Level& F, Level& C) {
  k_restrict<<<nblocks(C.n), kBlock, 0, c.stream>>>(C.n, F.childStart.p, F.child.p, F.r.p, C.bc.p);
  UFVM_LAUNCH_CHECK();
  return UFVM_OK;
}

int prolong(LinCtx& c, Level& F, const Level& C) {
  k_prolong<<<nblocks(F.n), kBlock, 0, c.stream>>>(F.n, F.parents.p, C.dphi.p, F.dphi.p);
  UFVM_LAUNCH_CHECK();
  return UFVM_OK;
}

}  // namespace ufvm
