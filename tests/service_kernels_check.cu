// Runs kernels of the batched service on hand-made levels and compares them with plain loops, bit for
// bit: the Galerkin product (8 and 32 lanes a coarse row, coarse rows of more than 16, 32 and 64 entries)
// and one colour of the FP32 Gauss-Seidel sweep (rows at and past the entries loaded before the wait).
#include "fast.cu"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

using namespace ufvm;

template <typename T>
static T* dev(const std::vector<T>& h) {
  T* p = nullptr;
  cudaMalloc((void**)&p, std::max<size_t>(h.size(), 1) * sizeof(T));
  cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
  return p;
}
template <typename T>
static std::vector<T> host(const T* p, size_t n) {
  std::vector<T> h(n);
  cudaMemcpy(h.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost);
  return h;
}
template <typename T>
static size_t differ(const std::vector<T>& a, const std::vector<T>& b) {
  size_t d = 0;
  for (size_t i = 0; i < a.size(); ++i) d += std::memcmp(&a[i], &b[i], sizeof(T)) != 0;
  return d;
}

// n fine rows of `deg` random entries, nc aggregates; every aggregate has a row
static int check_galerkin(int n, int nc, int deg, int G, unsigned seed) {
  std::mt19937 rng(seed);
  std::uniform_real_distribution<double> val(-1.0, 1.0);
  std::vector<int> parents(n), rp(n + 1, 0), col, cs(nc + 1, 0), child, crp(nc + 1, 0), ccol, gpos;
  for (int i = 0; i < n; ++i) parents[i] = i < nc ? i : (int)(rng() % nc);
  for (int i = 0; i < n; ++i) {
    const int d = (int)(rng() % (2 * deg + 1));
    for (int k = 0; k < d; ++k) col.push_back((int)(rng() % n));
    rp[i + 1] = (int)col.size();
  }
  std::vector<double> ac(n), anb(col.size());
  for (auto& v : ac) v = val(rng);
  for (auto& v : anb) v = val(rng);
  gpos.assign(col.size(), -1);
  std::vector<double> want_ac(nc), want;
  size_t widest = 0;
  for (int P = 0; P < nc; ++P) {
    double AC = 0.0;
    for (int i = 0; i < n; ++i) {
      if (parents[i] != P) continue;
      child.push_back(i);
      AC = AC + ac[i];
      for (int k = rp[i]; k < rp[i + 1]; ++k) {
        const int Q = parents[col[k]];
        if (Q == P) {
          AC = AC + anb[k];
          continue;
        }
        size_t t = crp[P];
        while (t < ccol.size() && ccol[t] != Q) ++t;
        if (t == ccol.size()) {
          ccol.push_back(Q);
          want.push_back(0.0);
        }
        want[t] = want[t] + anb[k];
        gpos[k] = (int)t;
      }
    }
    want_ac[P] = AC;
    cs[P + 1] = (int)child.size();
    crp[P + 1] = (int)ccol.size();
    widest = std::max(widest, ccol.size() - crp[P]);
  }
  LevDesc lev[2] = {};
  lev[0].n = n;
  lev[0].rowptr = dev(rp);
  lev[0].childStart = dev(cs);
  lev[0].child = dev(child);
  lev[0].ac64 = dev(ac);
  lev[0].anb64 = dev(anb);
  lev[0].gpos = dev(gpos);
  lev[1].n = nc;
  lev[1].galG = G;
  lev[1].rowptr = dev(crp);
  lev[1].ac64 = dev(std::vector<double>(nc, 7.0));
  lev[1].anb64 = dev(std::vector<double>(std::max<size_t>(want.size(), 1), 7.0));
  const int blocks = (int)(((long long)nc * G + kBlock - 1) / kBlock);
  std::vector<int2> work(blocks);
  for (int b = 0; b < blocks; ++b) work[b] = make_int2(0, b);
  SolveCtl ctl{};
  ctl.active = 1;
  k_galerkin_b<<<blocks, kBlock>>>(dev(std::vector<LevDesc>(lev, lev + 2)), 1, 0, dev(work), dev(std::vector<SolveCtl>{ctl}));
  const cudaError_t e = cudaDeviceSynchronize();
  const size_t bad = differ(host(lev[1].ac64, nc), want_ac) + differ(host(lev[1].anb64, want.size()), want);
  printf("galerkin n %d nc %d widest coarse row %zu lanes %d: %zu differ (%s)\n", n, nc, widest, G, bad, cudaGetErrorString(e));
  return e != cudaSuccess || bad ? 1 : 0;
}

// one colour: rows p0 .. p0 + cnt - 1 of n, reading x elsewhere
template <int PRE>
static int check_colour(int n, int p0, int cnt, int W, unsigned seed) {
  std::mt19937 rng(seed);
  std::uniform_real_distribution<float> val(-1.0f, 1.0f);
  std::vector<float> x(n), bc(n), ac(n), a((size_t)W * n, 0.0f);
  std::vector<int> col((size_t)W * n, -1);
  for (int i = 0; i < n; ++i) {
    x[i] = val(rng);
    bc[i] = val(rng);
    ac[i] = 2.0f + val(rng);
  }
  for (int p = 0; p < n; ++p) {
    const int d = p % 3 == 0 ? W : (int)(rng() % (W + 1));
    for (int k = 0; k < d; ++k) {
      int j = (int)(rng() % (n - cnt));
      if (j >= p0) j += cnt;  // not a row of this colour
      col[(size_t)k * n + p] = j;
      a[(size_t)k * n + p] = val(rng);
    }
  }
  std::vector<float> want = x;
  for (int p = p0; p < p0 + cnt; ++p) {
    volatile float v = bc[p];
    for (int k = 0; k < W && col[(size_t)k * n + p] >= 0; ++k) {
      volatile float pr = a[(size_t)k * n + p] * x[col[(size_t)k * n + p]];
      v = v - pr;
    }
    want[p] = v / ac[p];
  }
  GsItem it{};
  std::vector<GsItem> items;
  it.n = n; it.W = W;
  it.x = dev(x); it.bc = dev(bc); it.ac = dev(ac); it.ellCol = dev(col); it.ellAnb = dev(a);
  for (int q = 0; q < cnt; q += kBlock) {
    it.p0 = p0 + q;
    it.cnt = std::min(kBlock, cnt - q);
    items.push_back(it);
  }
  SolveCtl ctl{};
  ctl.active = 1;
  k_mc32_items<PRE><<<(int)items.size(), kBlock>>>(dev(items), dev(std::vector<SolveCtl>{ctl}));
  const cudaError_t e = cudaDeviceSynchronize();
  const size_t bad = differ(host(it.x, n), want);
  printf("colour n %d rows %d..%d width %d loaded %d: %zu differ (%s)\n", n, p0, p0 + cnt - 1, W, PRE, bad, cudaGetErrorString(e));
  return e != cudaSuccess || bad ? 1 : 0;
}

int main() {
  int bad = 0;
  bad += check_galerkin(40, 13, 3, 8, 1);       // rows at the ends of the 8 and 16 entries of a pass
  bad += check_galerkin(1000, 300, 4, 8, 2);
  bad += check_galerkin(1000, 17, 2, 8, 3);     // rows of all 16 others: one full pass
  bad += check_galerkin(1000, 18, 6, 8, 4);     // 17: a second pass
  bad += check_galerkin(900, 33, 6, 32, 5);     // 32
  bad += check_galerkin(900, 65, 20, 32, 6);    // 64: one full pass of 32 lanes
  bad += check_galerkin(900, 66, 20, 32, 7);    // 65: a second pass
  bad += check_galerkin(3000, 300, 30, 32, 8);  // about 200 entries
  bad += check_galerkin(5, 5, 0, 8, 9);         // no entries at all
  bad += check_galerkin(1, 1, 0, 32, 10);
  for (int W : {1, 7, 8}) bad += check_colour<8>(1000, 300, 257, W, W);
  for (int W : {9, 15, 16}) bad += check_colour<16>(700, 0, 256, W, W);
  for (int W : {17, 31, 32, 33, 40, 41, 72}) bad += check_colour<32>(900, 611, 289, W, W);
  printf(bad ? "FAILED\n" : "OK\n");
  return bad ? 1 : 0;
}
