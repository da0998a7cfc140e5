// k_projgr_noalloc (noalloc.cu) on the host, block by block, with l, u and x on pages that
// cannot be read wherever nbd says that the variable has no such bound: the kernel may read
// x, l and u only where projgr (culbfgsb/lbfgsbcpu.cpp:1390-1415) can use them.
//   projgr_reads_check {1|4|16}: elements a thread
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <string>
#include <vector>

#include "projgr_slice.cuh"

using namespace lbfgsb_b200;

static double* unreadable(size_t n) {
  void* p = mmap(nullptr, n * 8, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  return p == MAP_FAILED ? nullptr : static_cast<double*>(p);
}

template <int kPer>
static int check() {
  const int n = 2 * kPer * kNoAllocThreads + 77, rows = (n + kPer * kNoAllocThreads - 1) / (kPer * kNoAllocThreads);
  std::vector<double> x(n), g(n), l(n), u(n);
  for (int i = 0; i < n; i++) {
    x[i] = 0.001 * (i % 1000), g[i] = ((i * 37) % 101 - 50) * 0.01;
    l[i] = x[i] - 0.003 * (i % 7), u[i] = x[i] + 0.002 * (i % 5);
  }
  double* none = unreadable((size_t)n);
  if (!none) return 2;
  int bad = 0;
  for (int kind = 0; kind < 4; kind++) {
    const std::vector<int> nbd(n, kind);
    const bool lo = kind == 1 || kind == 2, up = kind >= 2;
    double want = 0;
    for (int i = 0; i < n; i++) {
      double pg = g[i];
      if (pg < 0 && up) pg = x[i] - u[i] > pg ? x[i] - u[i] : pg;
      if (g[i] >= 0 && lo) pg = x[i] - l[i] < pg ? x[i] - l[i] : pg;
      want = fabs(pg) > want ? fabs(pg) : want;
    }
    double out = -1;
    for (int b = 0; b < rows; b++)
      if (!emu::run_block(kNoAllocThreads, b, rows, [&] {
            k_projgr_noalloc<kPer>(n, kind ? x.data() : none, g.data(), nbd.data(), lo ? l.data() : none,
                                   up ? u.data() : none, g_projgr_scratch, &out);
          }))
        bad++;
    if (out != want || g_projgr_scratch[0] != 0) {
      fprintf(stderr, "nbd %d: %.17g, not %.17g\n", kind, out, want);
      bad++;
    }
  }
  return bad;
}

int main(int argc, char** argv) {
  const int per = argc == 2 ? atoi(argv[1]) : 0;
  return per == 1 ? check<1>() : per == 4 ? check<4>() : per == 16 ? check<16>() : 2;
}
