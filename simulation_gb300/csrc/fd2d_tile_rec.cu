// The on-chip 2D time loop that records the design box (fd2d_tile.cuh).
#include "fd2d_tile.cuh"

namespace fdtd {

int launch_tile_rec(const TileArgs& a, int V, bool lossy, cudaStream_t st) {
  switch (V) {
    case 1: return lossy ? launch_t<1, true, true, kTileRec>(a, st) : launch_t<1, false, true, kTileRec>(a, st);
    case 2: return lossy ? launch_t<2, true, true, kTileRec>(a, st) : launch_t<2, false, true, kTileRec>(a, st);
    case 3: return lossy ? launch_t<3, true, true, kTileRec>(a, st) : launch_t<3, false, true, kTileRec>(a, st);
    case 4: return lossy ? launch_t<4, true, true, kTileRec>(a, st) : launch_t<4, false, true, kTileRec>(a, st);
    case 5: return lossy ? launch_t<5, true, true, kTileRec>(a, st) : launch_t<5, false, true, kTileRec>(a, st);
    default: return FDTD_ERR_ARG;
  }
}

}  // namespace fdtd
