// The on-chip 2D time loop with plane wave and record of ez, lossless media (fd2d_tile.cuh).
#include "fd2d_tile.cuh"

namespace fdtd {

int launch_tile_ext(const TileArgs& a, int V, bool lossy, bool pml, cudaStream_t st) {
  if (lossy) return launch_tile_ext_lossy(a, V, pml, st);
  switch (V) {
    case 1: return pml ? launch_t<1, false, true, kTileExt>(a, st) : launch_t<1, false, false, kTileExt>(a, st);
    case 2: return pml ? launch_t<2, false, true, kTileExt>(a, st) : launch_t<2, false, false, kTileExt>(a, st);
    case 3: return pml ? launch_t<3, false, true, kTileExt>(a, st) : launch_t<3, false, false, kTileExt>(a, st);
    case 4: return pml ? launch_t<4, false, true, kTileExt>(a, st) : launch_t<4, false, false, kTileExt>(a, st);
    case 5: return pml ? launch_t<5, false, true, kTileExt>(a, st) : launch_t<5, false, false, kTileExt>(a, st);
    default: return FDTD_ERR_ARG;
  }
}

}  // namespace fdtd
