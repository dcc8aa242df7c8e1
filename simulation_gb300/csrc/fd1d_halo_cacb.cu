// Fused 1D runs of any length, cacb form (one translation unit per form, so the build compiles them in parallel).
#include "fd1d_halo.cuh"

namespace fdtd {

int launch_fd1d_halo_cacb(const Halo1DArgs& a, const HaloPlan& pl, int nfm, cudaStream_t st) {
  return launch_fd1d_halo_form<FDTD1D_FORM_CACB>(a, pl, nfm, st);
}

}  // namespace fdtd
