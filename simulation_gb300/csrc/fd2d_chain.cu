// Launch of the chained passes (fd2d_chain.cuh).
#include "fd2d_chain.cuh"

namespace fdtd {
namespace {

template <int NC, bool LOSSY, bool PML>
int launch_t(ChainArgs a, int pml_cells, float gen_cost, cudaStream_t st) {
  auto kern = k_chain<NC, LOSSY, PML>;
  const size_t smem = chain_smem_bytes(NC, LOSSY, PML);
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
  const long blocks = chain_layout(a, kChainLv * NC, (long)nsm * std::max(per_sm, 1), pml_cells, gen_cost > 0.f ? gen_cost : 2.5f);
  kern<<<(unsigned)blocks, 32 * NC, smem, st>>>(a);
  return fdtd_host::check_launch();
}

template <int NC>
int launch_nc(const ChainArgs& a, bool lossy, bool pml, int pml_cells, float gen_cost, cudaStream_t st) {
  if (lossy) return pml ? launch_t<NC, true, true>(a, pml_cells, gen_cost, st) : launch_t<NC, true, false>(a, 0, gen_cost, st);
  return pml ? launch_t<NC, false, true>(a, pml_cells, gen_cost, st) : launch_t<NC, false, false>(a, 0, gen_cost, st);
}

}  // namespace

int launch_chain(const fdtd2d_params& p, const FieldSet& in, const FieldSet& out, float* ez, int t0, int nc, int* status,
                 float gen_cost, cudaStream_t st) {
  ChainArgs a{};
  a.nx = p.nx;
  a.ny = p.ny;
  a.in = in;
  a.out = out;
  a.ez = ez;
  a.naz = p.naz;
  a.nbz = p.nbz;
  a.pml = p.pml;
  a.src_kind = p.src.kind;
  a.src_i = p.src.i;
  a.src_j = p.src.j;
  a.src_table = p.src.table;
  a.t0 = t0;
  a.status = status;
  const bool lossy = p.nbz != nullptr, pml = has_pml(p);
  if (nc == 2) return launch_nc<2>(a, lossy, pml, p.pml_cells, gen_cost, st);
  if (nc == 4) return launch_nc<4>(a, lossy, pml, p.pml_cells, gen_cost, st);
  return FDTD_ERR_ARG;
}

}  // namespace fdtd
