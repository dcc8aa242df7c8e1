// Launch of the chained passes (fd2d_chain.cuh).
#include "fd2d_chain.cuh"

namespace fdtd {
namespace {

// waves: blocks launched over those resident.  One wave ends with its slowest
// block (SMs idle for 16% of a 2 x 4 pass at 6144^2); four short ones, the
// general stripes first, balance themselves, at the price of more recomputed
// rows: 8192^2 lossy with layer 580 -> 717 Gcell-updates/s, but 4096^2 521 -> 451.
template <int LV, int NC, bool LOSSY, bool PML>
int launch_t(ChainArgs a, int pml_cells, double waves, float gen_cost, cudaStream_t st) {
  auto kern = k_chain<LV, NC, LOSSY, PML>;
  const size_t smem = chain_smem_bytes(LV, NC, LOSSY, PML);
  int dev = 0, nsm = 0, per_sm = 0;
  cudaError_t e = cudaSuccess;
  if (smem > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * NC, smem);
  if (e != cudaSuccess) {
    fdtd_host::note_cuda_error(e);
    return FDTD_ERR_CUDA;
  }
  const long blocks = chain_layout(a, LV * NC, (long)(nsm * std::max(per_sm, 1) * waves), pml_cells, gen_cost);
  kern<<<(unsigned)blocks, 32 * NC, smem, st>>>(a);
  return fdtd_host::check_launch();
}

template <int LV, int NC>
int launch_nc(const ChainArgs& a, bool lossy, bool pml, int pml_cells, double waves, float g, cudaStream_t st) {
  if (lossy)
    return pml ? launch_t<LV, NC, true, true>(a, pml_cells, waves, g, st)
               : launch_t<LV, NC, true, false>(a, 0, waves, g, st);
  return pml ? launch_t<LV, NC, false, true>(a, pml_cells, waves, g, st)
             : launch_t<LV, NC, false, false>(a, 0, waves, g, st);
}

}  // namespace

int launch_chain(const fdtd2d_params& p, int pitch, const float* naz, const float* nbz, const FieldSet& in,
                 const FieldSet& out, float* ez, int t0, int k, int* status, float gen_cost, cudaStream_t st) {
  ChainArgs a{};
  a.nx = p.nx;
  a.ny = p.ny;
  a.pitch = pitch;
  a.in = in;
  a.out = out;
  a.ez = ez;
  a.naz = naz;
  a.nbz = nbz;
  a.pml = p.pml;
  a.src_kind = p.src.kind;
  a.src_i = p.src.i;
  a.src_j = p.src.j;
  a.src_table = p.src.table;
  a.t0 = t0;
  a.status = status;
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
