// Host-side check of the on-chip BBPGD solver's dispatch and shapes
// (pcc_resident.cu, built by nvcc, run on the CPU).  Reads lines
//   <real: f or d> <3d: 0 or 1> <phases> <cells n> <constraints m> <gi gj> x m
// (constraints in the order of their detection) and prints for each the form
// that the solver takes for them, its blocks and how many groups of 16 cells
// find no room in their block's shared memory, after checking the bounds that
// the kernel relies on: cells per block, entries covered once, warps' worths
// per block, slots for the constraints past a chunk's first 256.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "pcc_resident.cu"

using namespace pcc;

static int bad(const char* what) { return printf("%s\n", what), 1; }

template <class Real, bool k3D>
static int check(int phases, int n, int m, const std::vector<int>& gi, const std::vector<int>& gj) {
  Shape sh;
  bool cluster = false;
  if (!pick_shape<Real, k3D>(m, n, phases, 148, kMaxCluster, &sh, &cluster)) return printf("streaming 0 0\n"), 0;
  if (sh.smem > kSmemMost || sh.nb < 1) return bad("the shape does not fit");
  const int nch = (int)chunk_count(m);
  std::vector<int> off(n + 1, 0);
  for (int c = 0; c < m; ++c) ++off[gi[c] + 1], ++off[gj[c] + 1];
  for (int i = 0; i < n; ++i) off[i + 1] += off[i];
  int without = 0, entries = 0;
  for (int b = 0; b < sh.nb; ++b) {
    const int lo = first_cell(off.data(), n, sh.kappa, b, sh.nb), hi = first_cell(off.data(), n, sh.kappa, b + 1, sh.nb);
    if (b == 0 && lo != 0) return bad("cells before the first block's");
    if (hi - lo > sh.cells_max) return bad("more cells in a block than it has room for");
    entries += off[hi] - off[lo];
    std::vector<int> degree;
    for (int i = lo; i < hi; ++i) degree.push_back(off[i + 1] - off[i]);
    std::sort(degree.begin(), degree.end(), [](int x, int y) { return x > y; });
    int run = 0;
    for (size_t g = 0; g < degree.size(); g += kGroup) {
      run += 32 * ((degree[g] + kLanes - 1) / kLanes);
      without += run > sh.cap;
    }
  }
  if (entries != 2 * m) return bad("entries missing");
  if (cluster) {
    std::vector<int> key(sh.nvw), order(sh.nvw);
    for (int id = 0; id < sh.nvw; ++id) {
      const long long c = chunk_lo(id >> 3, m, nch) + 32 * (id & 7);
      key[id] = c < chunk_lo((id >> 3) + 1, m, nch) ? gi[c] : 0x7fffffff;
      order[id] = id;
    }
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return key[x] < key[y]; });
    for (int r = 0; r < sh.nb; ++r) {
      const int b = (int)((long long)r * sh.nvw / sh.nb), e = (int)((long long)(r + 1) * sh.nvw / sh.nb);
      int first = 0;
      for (int p = b; p < e; ++p) first += (order[p] & 7) == 0;
      if (e - b > sh.lvw) return bad("more warps' worths in a block than it has room for");
      if (first > sh.extra) return bad("more chunks start in a block than it has room for");
    }
    for (int ch = 0; ch < nch; ++ch)
      if (chunk_lo(ch + 1, m, nch) - chunk_lo(ch, m, nch) > kBlock + 32) return bad("a chunk past its slots");
  } else {
    for (int ch = 0; ch < nch; ++ch)
      if (chunk_lo(ch + 1, m, nch) - chunk_lo(ch, m, nch) > sh.cstride) return bad("a chunk past its slots");
  }
  printf("%s %d %d\n", cluster ? "cluster" : "grid", sh.nb, without);
  return 0;
}

int main() {
  char real;
  int full, phases, n, m;
  while (scanf(" %c %d %d %d %d", &real, &full, &phases, &n, &m) == 5) {
    std::vector<int> gi(m), gj(m);
    for (int c = 0; c < m; ++c)
      if (scanf("%d %d", &gi[c], &gj[c]) != 2) return bad("input ends early");
    if (full ? check<double, true>(phases, n, m, gi, gj)
             : real == 'f' ? check<float, false>(phases, n, m, gi, gj) : check<double, false>(phases, n, m, gi, gj))
      return 1;
  }
  return 0;
}
