// Host-only check of the block -> work layout of the chained passes
// (simulation_gb300/csrc/fd2d_chain.cuh), built by tests/test_chain_mapping.py and
// run on the CPU (it makes no CUDA call).
//
// A block marches down one segment of rows of one stripe of columns; the stripes
// that the absorbing layer or the grid's edge makes general get shorter segments
// (chain_layout, chain_work).  With the header's own functions, over grid shapes,
// layer widths, block counts and cost factors, in the shapes that are launched: every
// (stripe, row) belongs to exactly one block, the stripes' columns cover the grid, and
// a block's shared memory fits.
#include <cstdio>
#include <vector>

#include "fd2d_chain.cuh"

namespace {

int g_fail = 0;

void check(int K, int nx, int ny, long want, int P, float G) {
  fdtd::ChainArgs a{};
  a.nx = nx;
  a.ny = ny;
  const long blocks = fdtd::chain_layout(a, K, want, P, G);
  const int outw = fdtd::kChainCols - 2 * fdtd::chain_halo(K, 1);
  std::vector<int> cover((size_t)a.n_stripes * nx, 0);
  bool ok = (long)a.n_stripes * outw >= ny && (long)(a.n_stripes - 1) * outw < ny && blocks > 0 && blocks < (1L << 31) &&
            a.n_gen_lo + a.n_gen_hi <= a.n_stripes;
  for (long b = 0; ok && b < blocks + 64; ++b) {
    int stripe, i_s, i_e;
    if (!fdtd::chain_work(a, (int)b, stripe, i_s, i_e)) continue;
    ok = b < blocks && stripe >= 0 && stripe < a.n_stripes && i_s >= 0 && i_e <= nx;
    for (int r = i_s; ok && r < i_e; ++r) ++cover[(size_t)stripe * nx + r];
  }
  for (int c : cover) ok = ok && c == 1;
  if (!ok && g_fail++ < 20) std::printf("FAIL K=%d nx=%d ny=%d blocks=%ld P=%d G=%g\n", K, nx, ny, want, P, G);
}

}  // namespace

int main() {
  for (int K : {4, 8})
    for (int nx : {64, 65, 130, 301, 1024, 1501, 4099})
      for (int ny : {128, 129, 223, 225, 1003, 1204, 8192})
        for (long want : {1L, 152L, 608L, 1216L, 4864L})
          for (int P : {0, 1, 9, 33, 400})
            for (float G : {0.f, 1.f, 1.5f, 2.5f, 4.f, 16.f}) check(K, nx, ny, want, P, G);
  const int shapes[][2] = {{2, 2}, {2, 4}, {4, 2}};
  for (auto& s : shapes)
    for (int lossy = 0; lossy < 2; ++lossy)
      for (int pml = 0; pml < 2; ++pml)
        if (fdtd::chain_smem_bytes(s[0], s[1], lossy, pml) > 227u * 1024 && g_fail++ < 20) std::printf("FAIL shared memory\n");
  if (g_fail) return 1;
  std::printf("ok\n");
  return 0;
}
