// The on-chip 2D time loop with plane wave and record of ez, lossy media (fd2d_tile.cuh).
#include "fd2d_tile.cuh"

namespace fdtd {

int launch_tile_ext_lossy(const TileArgs& a, int V, bool pml, cudaStream_t st) {
  switch (V) {
    case 1: return pml ? launch_t<1, true, true, kTileExt>(a, st) : launch_t<1, true, false, kTileExt>(a, st);
    case 2: return pml ? launch_t<2, true, true, kTileExt>(a, st) : launch_t<2, true, false, kTileExt>(a, st);
    case 3: return pml ? launch_t<3, true, true, kTileExt>(a, st) : launch_t<3, true, false, kTileExt>(a, st);
    case 4: return pml ? launch_t<4, true, true, kTileExt>(a, st) : launch_t<4, true, false, kTileExt>(a, st);
    case 5: return pml ? launch_t<5, true, true, kTileExt>(a, st) : launch_t<5, true, false, kTileExt>(a, st);
    default: return FDTD_ERR_ARG;
  }
}

}  // namespace fdtd
