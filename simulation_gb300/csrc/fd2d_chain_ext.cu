// Chained passes (fd2d_chain.cuh) with the fd2d_3_4 extras
// (fd2d/python/fd2d_3_4.py:90-170): the TF/SF box's corrections in the pass, the
// running DFT of Ez after it.
//
// The march carries the DFT's accumulators with each row through its levels: 2
// loads and stores of shared memory per cell, step and frequency, 3 blocks an
// SM, 148 us for 4 steps at 2048^2 with 3 frequencies.  Here the pass stores
// the ez of each of its steps (coalesced, 4 bytes a cell and step), and every
// 16 steps k_dft_rec adds them to the accumulators in the order of the steps,
// so the sums are bitwise the same: 113 us for 8 steps and 41 for their DFT.
#include "fd2d_chain.cuh"

namespace fdtd {
namespace {

template <int NC>
int launch_k(const ChainArgs& a, bool lossy, bool pml, int pml_cells, float g, cudaStream_t st) {
  if (lossy)
    return pml ? launch_t<2, NC, true, true, true>(a, pml_cells, 1.0, g, st)
               : launch_t<2, NC, true, false, true>(a, 0, 1.0, g, st);
  return pml ? launch_t<2, NC, false, true, true>(a, pml_cells, 1.0, g, st)
             : launch_t<2, NC, false, false, true>(a, 0, 1.0, g, st);
}

}  // namespace

int launch_chain_ext(const fdtd2d_params& p, int pitch, const float* naz, const float* nbz, const FieldSet& in,
                     const FieldSet& out, float* ez, int t0, int k, int* status, float gen_cost, const MarchExt& ext,
                     float* ez_rec, size_t rec_slot, cudaStream_t st) {
  if (k != 4 && k != 8) return FDTD_ERR_ARG;
  ChainArgs a = chain_args(p, pitch, naz, nbz, in, out, ez, t0, status);
  a.np = ext.tfsf_npml;
  a.inc_e = ext.inc_e;
  a.inc_h = ext.inc_h;
  a.ez_rec = ext.nf > 0 ? ez_rec : nullptr;
  a.rec_slot = rec_slot;
  const bool lossy = p.nbz != nullptr, pml = has_pml(p);
  // the box's edge columns lie in the stripes of the layer, or make the first and last general
  const int edge = std::max(pml ? p.pml_cells : 0, ext.tfsf_npml > 0 ? ext.tfsf_npml + 1 : 0);
  // general over interior time per row: 3.5 (2048^2, 96 steps, no DFT: 1323 us against 1500 at 2.5 and 1344 at 5)
  const float g = gen_cost > 0.f ? gen_cost : pml ? 3.5f : 1.5f;
  return k == 8 ? launch_k<4>(a, lossy, pml, edge, g, st) : launch_k<2>(a, lossy, pml, edge, g, st);
}

}  // namespace fdtd
