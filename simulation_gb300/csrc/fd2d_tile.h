// Host side of the on-chip 2D time loop (fd2d_tile.cuh): its layout for a grid
// and its launch.
#pragma once

#include "fd2d_internal.cuh"

namespace fdtd {

constexpr int kTileWarps = 16;   // of a block; V rows each
constexpr int kTileCols = 128;   // of a tile
constexpr int kTileMinSteps = 4;  // shorter runs march: loading and storing the tiles takes longer than the steps
struct TilePlan {
  int V = 0, T = 0, hc = 0, n_ti = 0, n_tj = 0, own_r = 0, own_c = 0;
};
constexpr int kTileMaxBlocks = 152;                       // one per SM
constexpr size_t kTileFlagBytes = kTileMaxBlocks * 128;  // flags of the largest launch

// What the adjoint's runs record and read besides the fields
constexpr int kTileFwd = 0;  // the time loop
constexpr int kTileRec = 1;  // and dz' - iz of the design box after each step
constexpr int kTileRev = 2;  // steps t0, t0-1, .. undone on the adjoint fields
constexpr int kTileExt = 3;  // the time loop with TF/SF box and record of ez
struct TileExt {
  int np = 0;                      // TF/SF box, 0: none
  const float* inc_e = nullptr;    // of the run's steps, as in MarchExt
  const float* inc_h = nullptr;
  float* ez_rec = nullptr;         // ez of step t0+s+1 at s*rec_slot, or null
  size_t rec_slot = 0;
};
struct TileAdj {
  fdtd2d_box box{};
  int jb = 0, njp = 0;   // the box's columns in whole groups of four: first column, how many
  float* rec = nullptr;  // [step of the run][box row][njp]
  float probe_w = 0.f;
  float* grad_naz = nullptr;
  float* grad_nbz = nullptr;
};

// The layout with the shortest modelled step among those whose tiles fit the
// SMs, one block each; false when none does (the caller marches).  max_V: the
// largest strip to consider.  The model, in us, fitted to measured layouts with an
// absorbing layer (the general steps, on which all tiles wait): a step takes 0.35 + 0.27 V (V = 1: 0.58,
// 2: 0.75, 5: 1.7), loss adds 0.1 V; an exchange 2.1 + 0.52 V (fence, flag and
// read latencies, and the halo's traffic), once in T steps.  100^2 runs 1.2 a
// step with V = 1, T = 4 (6.2 marching), 1024^2 3.3 with V = 5, T = 4 (10.5).
inline bool tile_plan(int nx, int ny, bool lossy, bool pml, int max_blocks, TilePlan& best, int max_V = 5) {
  double best_cost = 1e30;
  for (int V = 1; V <= max_V; ++V)
    for (int T = 2; T <= 8; ++T) {
      TilePlan pl;
      pl.V = V;
      pl.T = T;
      pl.hc = ny <= kTileCols ? 0 : (T + 3) / 4 * 4;  // whole lanes
      pl.own_r = kTileWarps * V - 2 * T;
      pl.own_c = kTileCols - 2 * pl.hc;
      if (pl.own_r < T) continue;
      // (64 bits: extents near 2^31 would wrap to a small or negative count)
      const long long ti = ((long long)nx + pl.own_r - 1) / pl.own_r, tj = ((long long)ny + pl.own_c - 1) / pl.own_c;
      const long long blocks = ti * tj;
      if (blocks > max_blocks) continue;
      pl.n_ti = (int)ti;
      pl.n_tj = (int)tj;
      const double step = 0.35 + V * ((pml ? 0.27 : 0.2) + (lossy ? 0.1 : 0.0));
      const double cost = step + (blocks > 1 ? (2.1 + 0.52 * V) / T : 0.0);
      if (cost < best_cost) {
        best_cost = cost;
        best = pl;
      }
    }
  return best_cost < 1e30;
}

constexpr int tile_rev_max_V(bool lossy) { return lossy ? 4 : 5; }  // the gradients' shared memory
// defined in fd2d_tile.cu.  Every launch that can wait gets a status word
// (FDTD_STATUS_TIMEOUT where a wait ran out, after which the fields are wrong);
// check_finite: it also tests the fields it stores
int launch_tile(const fdtd2d_params& p, const FieldSet& in, const FieldSet& out, const FieldSet& x0, const FieldSet& x1,
                float* ez, int t0, int nsteps, int* status, float* probe_ez, unsigned* flags, const TilePlan& pl,
                cudaStream_t st, int mode = kTileFwd, const TileAdj* adj = nullptr,
                const TileExt* ext = nullptr, bool check_finite = true);

}  // namespace fdtd
