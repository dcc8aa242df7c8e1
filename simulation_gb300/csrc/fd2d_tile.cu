// Launch of the on-chip 2D time loop (fd2d_tile.cuh).
#include "fd2d_tile.cuh"

#include <type_traits>

namespace fdtd {

namespace {

template <int V>
int launch_v(const TileArgs& a, bool lossy, bool pml, cudaStream_t st) {
  if (lossy) return pml ? launch_t<V, true, true, kTileFwd>(a, st) : launch_t<V, true, false, kTileFwd>(a, st);
  return pml ? launch_t<V, false, true, kTileFwd>(a, st) : launch_t<V, false, false, kTileFwd>(a, st);
}

bool al16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

}  // namespace

int launch_tile(const fdtd2d_params& p, const FieldSet& in, const FieldSet& out, const FieldSet& x0, const FieldSet& x1,
                float* ez, int t0, int nsteps, int* status, float* probe_ez, unsigned* flags, const TilePlan& pl,
                cudaStream_t st, int mode, const TileAdj* adj, const TileExt* ext, bool check_finite) {
  TileArgs a{};
  a.nx = p.nx;
  a.ny = p.ny;
  a.in = in;
  a.out = out;
  a.x[0] = x0;
  a.x[1] = x1;
  a.ez = ez;
  a.naz = p.naz;
  a.nbz = p.nbz;
  a.pml = p.pml;
  a.src_kind = p.src.kind;
  a.src_i = p.src.i;
  a.src_j = p.src.j;
  a.src_table = p.src.table;
  a.t0 = t0;
  a.nsteps = nsteps;
  a.status = status;
  a.check_finite = status && check_finite;
  a.probe_i = p.probe_i;
  a.probe_j = p.probe_j;
  a.probe_ez = probe_ez;
  a.flags = flags;
  if (adj) a.adj = *adj;
  if (ext) a.ext = *ext;
  a.T = pl.T;
  a.hc = pl.hc;
  a.n_ti = pl.n_ti;
  a.n_tj = pl.n_tj;
  a.own_r = pl.own_r;
  a.own_c = pl.own_c;
  const bool lossy = p.nbz != nullptr, pml = has_pml(p);
  bool v = p.ny % 4 == 0 && al16(p.naz) && al16(ez) && (!lossy || al16(p.nbz));
  for (const FieldSet* f : {&in, &out, &x0, &x1})
    v = v && al16(f->dz) && al16(f->hx) && al16(f->hy) && (!lossy || al16(f->iz)) &&
        (!pml || (al16(f->ihx) && al16(f->ihy)));
  a.vec = v;
  if (pl.n_ti * pl.n_tj > 1) {
    const cudaError_t e = cudaMemsetAsync(flags, 0, (size_t)pl.n_ti * pl.n_tj * 128, st);
    if (e != cudaSuccess) {
      fdtd_host::note_cuda_error(e);
      return FDTD_ERR_CUDA;
    }
  }
  if (mode == kTileExt) {
    a.vec = v && al16(a.ext.ez_rec) && a.ext.rec_slot % 4 == 0;
    return launch_tile_ext(a, pl.V, lossy, pml, st);
  }
  if (mode != kTileFwd) {
    if (!pml || !v || !adj) return FDTD_ERR_ARG;
    return mode == kTileRec ? launch_tile_rec(a, pl.V, lossy, st) : launch_tile_rev(a, pl.V, lossy, st);
  }
  switch (pl.V) {
    case 1: return launch_v<1>(a, lossy, pml, st);
    case 2: return launch_v<2>(a, lossy, pml, st);
    case 3: return launch_v<3>(a, lossy, pml, st);
    case 4: return launch_v<4>(a, lossy, pml, st);
    case 5: return launch_v<5>(a, lossy, pml, st);
    default: return FDTD_ERR_ARG;
  }
}

}  // namespace fdtd
