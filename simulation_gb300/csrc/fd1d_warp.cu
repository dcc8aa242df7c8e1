// Single-warp fused 1D run (lines of up to 512 cells without the running DFT).
#include "fd1d_warp.cuh"

namespace fdtd {

int launch_fd1d_warp(const fdtd1d_params& p, const fdtd1d_state& s, int t0, int nsteps, cudaStream_t st) {
  const int nx = p.nx;
  if (nx > 32 * 16) return FDTD_ERR_SIZE;
  // fewest cells per lane that cover the line with 32 lanes
  const int cpt = nx <= 64 ? 2 : nx <= 128 ? 4 : nx <= 256 ? 8 : 16;
  const Warp1DArgs a{p, s, t0, nsteps};
  const bool hi_end = nx % cpt == 0, soft = p.src_kind == FDTD_SRC_SOFT;
  auto go = [&](auto kern) -> int {
    kern<<<1, 32, 0, st>>>(a);
    return fdtd_host::check_launch();
  };
#define FDTD_WARP_CASE(F, C)                                                                    \
  if (p.form == F && cpt == C) {                                                                \
    if (soft) return hi_end ? go(k_fd1d_warp<F, C, true, true>) : go(k_fd1d_warp<F, C, false, true>); \
    return hi_end ? go(k_fd1d_warp<F, C, true, false>) : go(k_fd1d_warp<F, C, false, false>);   \
  }
#define FDTD_WARP_FORM(F) \
  FDTD_WARP_CASE(F, 2) FDTD_WARP_CASE(F, 4) FDTD_WARP_CASE(F, 8) FDTD_WARP_CASE(F, 16)
  FDTD_WARP_FORM(FDTD1D_FORM_CB)
  FDTD_WARP_FORM(FDTD1D_FORM_CACB)
  FDTD_WARP_FORM(FDTD1D_FORM_DFORM)
  FDTD_WARP_FORM(FDTD1D_FORM_DEBYE)
#undef FDTD_WARP_FORM
#undef FDTD_WARP_CASE
  return FDTD_ERR_ARG;
}

}  // namespace fdtd
