// Host side of the on-chip 2D time loop (fd2d_tile.cuh): its layout for a grid
// and its launch.
#pragma once

#include "fd2d_internal.cuh"

namespace fdtd {

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

// defined in fd2d_tile.cu.  max_V: the largest strip to consider.  Every launch that
// can wait gets a status word (FDTD_STATUS_TIMEOUT where a wait ran out, after which the
// fields are wrong); check_finite: it also tests the fields it stores
bool tile_plan(int nx, int ny, bool lossy, bool pml, int max_blocks, TilePlan& best, int max_V = 5);
constexpr int tile_rev_max_V(bool lossy) { return lossy ? 4 : 5; }  // the gradients' shared memory
int launch_tile(const fdtd2d_params& p, const FieldSet& in, const FieldSet& out, const FieldSet& x0, const FieldSet& x1,
                float* ez, int t0, int nsteps, int* status, float* probe_ez, unsigned* flags, const TilePlan& pl,
                cudaStream_t st, int mode = kTileFwd, const TileAdj* adj = nullptr,
                const TileExt* ext = nullptr, bool check_finite = true);

}  // namespace fdtd
