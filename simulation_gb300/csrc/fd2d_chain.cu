// Launch of the chained passes (fd2d_chain.cuh).
#include "fd2d_chain.cuh"

namespace fdtd {
namespace {

template <int LV, int NC>
int launch_nc(const ChainArgs& a, bool lossy, bool pml, int pml_cells, double waves, float g, cudaStream_t st) {
  if (lossy)
    return pml ? launch_t<LV, NC, true, true, false>(a, pml_cells, waves, g, st)
               : launch_t<LV, NC, true, false, false>(a, 0, waves, g, st);
  return pml ? launch_t<LV, NC, false, true, false>(a, pml_cells, waves, g, st)
             : launch_t<LV, NC, false, false, false>(a, 0, waves, g, st);
}

}  // namespace

int launch_chain(const fdtd2d_params& p, int pitch, const float* naz, const float* nbz, const FieldSet& in,
                 const FieldSet& out, float* ez, int t0, int k, int* status, float gen_cost, cudaStream_t st) {
  const ChainArgs a = chain_args(p, pitch, naz, nbz, in, out, ez, t0, status);
  const bool lossy = nbz != nullptr, pml = has_pml(p);
  const long long cells = (long long)p.nx * p.ny;
  auto cost = [&](float g) { return gen_cost > 0.f ? gen_cost : g; };
  // general over interior time per row: 2.5 with the layer at 2 steps a warp
  // (4096^2: 594 against 520 at 1.5 and 553 at 4), 4 at 4 steps; 1.5 without it
  if (k == 4) return launch_nc<2, 2>(a, lossy, pml, p.pml_cells, 1.0, cost(pml ? 2.5f : 1.5f), st);
  if (k != 8) return FDTD_ERR_ARG;
  if (!pml) {
    // (no layer: 3072^2 971 against 767 with 2 steps a warp; 2048^2 lies between)
    if (cells >= (1LL << 23)) return launch_nc<4, 2>(a, lossy, pml, 0, 1.0, cost(1.5f), st);
  } else if (cells >= (1LL << 25)) {
    return launch_nc<4, 2>(a, lossy, pml, p.pml_cells, 4.0, cost(4.0f), st);
  }
  return launch_nc<2, 4>(a, lossy, pml, p.pml_cells, 1.0, cost(pml ? 2.5f : 1.5f), st);
}

}  // namespace fdtd
