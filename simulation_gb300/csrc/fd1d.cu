// 1D Ex/Hy FDTD (fd1d): per-function kernels and the fused single-run kernel.
//
// Per-function kernels (fdtd1d_efield / fdtd1d_hfield / fdtd1d_fourier) update
// the caller's arrays in place with one launch per reference function.
//
// The fused runs (fdtd1d_step_n) take a whole time loop in ONE launch: lines of
// up to 512 cells without the DFT in one warp (fd1d_warp.cuh), all others as
// overlapping chunks, one warp each, in a block or a thread-block cluster
// (fd1d_halo.cuh).  Both keep the reference's serial order E -> source -> DFT
// -> ABC -> H exactly; the reference's own CUDA kernels race on ex[1] and
// ex[nx-1] (fd1d/cuda/fd1d_1_3.cu:25-28, :35-39).
#include <algorithm>

#include "fd1d_halo.cuh"
#include "fd1d_warp.cuh"
#include "fdtd_common.cuh"

namespace fdtd {

// ============================================================ per-function
// E stage, one thread per cell (fd1d/program/fd1d_1_3.py:55-57,
// fd1d/program/fd1d_1_5.py:65-67, fd1d/program/fd1d_2_2.py:74-84)
template <int FORM>
__global__ void k_fd1d_efield(fdtd1d_params p, fdtd1d_state s, int t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 1 || i >= p.nx) return;
  const float v = (p.src_kind != FDTD_SRC_NONE && i == p.src_k) ? p.src_table[t - 1] : 0.f;
  if (FORM == FDTD1D_FORM_CB || FORM == FDTD1D_FORM_CACB) {
    float e = (FORM == FDTD1D_FORM_CB) ? ex_update_cb(s.ex[i], s.hy[i - 1], s.hy[i], p.cb[i])
                                        : ex_update_cacb(s.ex[i], s.hy[i - 1], s.hy[i], p.ca[i], p.cb[i]);
    if (p.src_kind != FDTD_SRC_NONE && i == p.src_k) e = (p.src_kind == FDTD_SRC_HARD) ? v : __fadd_rn(e, v);
    s.ex[i] = e;
  } else {
    float d = dx_update(s.dx[i], s.hy[i - 1], s.hy[i]);
    if (p.src_kind != FDTD_SRC_NONE && i == p.src_k) d = (p.src_kind == FDTD_SRC_HARD) ? v : __fadd_rn(d, v);
    s.dx[i] = d;
    float ixv = s.ix[i];
    if (FORM == FDTD1D_FORM_DFORM) {
      s.ex[i] = ex_from_dx(d, ixv, p.nax[i], p.nbx[i]);
    } else {
      float sxv = s.sx[i];
      s.ex[i] = ex_from_dx_debye(d, ixv, sxv, p.nax[i], p.nbx[i], p.ncx[i], p.ndx[i]);
      s.sx[i] = sxv;
    }
    s.ix[i] = ixv;
  }
}

// source at cell 0 (never updated by the E loop, which starts at 1)
__global__ void k_fd1d_src0(fdtd1d_params p, fdtd1d_state s, int t) {
  const float v = p.src_table[t - 1];
  float* f = (p.form == FDTD1D_FORM_CB || p.form == FDTD1D_FORM_CACB) ? s.ex : s.dx;
  f[0] = (p.src_kind == FDTD_SRC_HARD) ? v : __fadd_rn(f[0], v);
  if (p.form >= FDTD1D_FORM_DFORM) {
    // ex[0] is not recomputed from dx[0] by the reference (exfield covers 1..nx-1)
  }
}

// ABC then H (fd1d/program/fd1d_2_2.py:87-92).  Thread 0 owns the low-side
// ABC and hy[0]; the thread of cell nx-2 owns the high-side ABC and hy[nx-2],
// so each boundary value is set before the only H update that reads it.
__global__ void k_fd1d_hfield(fdtd1d_params p, fdtd1d_state s) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int nx = p.nx;
  if (i > nx - 2) return;
  float e0, e1;
  if (p.abc && i == 0) {
    const float b0 = s.bc[0], b1 = s.bc[1];
    e1 = s.ex[1];
    s.ex[0] = b0;
    s.bc[0] = b1;
    s.bc[1] = e1;
    e0 = b0;
  } else {
    e0 = s.ex[i];
    e1 = s.ex[i + 1];
  }
  if (p.abc && i == nx - 2) {
    const float b2 = s.bc[2], b3 = s.bc[3];
    // ex[nx-2] (e0, nx >= 4 so i > 0) is final for this step; ex[nx-1] becomes bc[3]
    s.ex[nx - 1] = b3;
    s.bc[3] = b2;
    s.bc[2] = e0;
    e1 = b3;
  }
  s.hy[i] = hy_update(s.hy[i], e0, e1);
}

// running DFT (fd1d/program/fd1d_2_2.py:65-71): probes and, optionally, every cell
__global__ void k_fd1d_fourier(fdtd1d_params p, fdtd1d_state s, int t) {
  const float* cs = p.dft_cos + (size_t)(t - 1) * p.nf;
  const float* sn = p.dft_sin + (size_t)(t - 1) * p.nf;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (p.full_dft && i < p.nx) {
    const float e = s.ex[i];
    for (int f = 0; f < p.nf; ++f) {
      const size_t m = (size_t)f * p.nx + i;
      s.r_pt[m] = __fmaf_rn(cs[f], e, s.r_pt[m]);
      s.i_pt[m] = __fmaf_rn(-sn[f], e, s.i_pt[m]);
    }
  }
  if (i < p.nf) {
    for (int q = 0; q < p.nprobe; ++q) {
      const float e = s.ex[p.probe_k[q]];
      const size_t m = (size_t)q * p.nf + i;
      s.r_pr[m] = __fmaf_rn(cs[i], e, s.r_pr[m]);
      s.i_pr[m] = __fmaf_rn(-sn[i], e, s.i_pr[m]);
    }
  }
}

// ============================================================ fused run
int launch_fd1d_efield(int t, const fdtd1d_params& p, const fdtd1d_state& s, cudaStream_t st);
int launch_fd1d_fourier(int t, const fdtd1d_params& p, const fdtd1d_state& s, cudaStream_t st);
int launch_fd1d_hfield(const fdtd1d_params& p, const fdtd1d_state& s, cudaStream_t st);

int launch_fd1d_run(const fdtd1d_params& p, const fdtd1d_state& s, int t0, int nsteps, cudaStream_t st) {
  // a line of up to 512 cells without the DFT runs in ONE warp (47 ns a step
  // at 200 cells, 65 in overlapping chunks); with the DFT the chunks' several
  // warps are the faster layout (512 cells, 3 frequencies at every cell: 180
  // ns a step against 6000 in one warp)
  if (p.nf == 0 && p.nx <= 32 * 16) return launch_fd1d_warp(p, s, t0, nsteps, st);
  const int nfm = !(p.nf > 0 && p.full_dft) ? 0 : p.nf <= 4 ? 4 : p.nf <= 8 ? 8 : 1;
  for (int max_cluster = 16; max_cluster >= 8; max_cluster /= 2) {
    HaloPlan pl;
    int use = nfm;
    bool have = halo_plan(p.form, p.nx, use, p.nf, p.nprobe, max_cluster, pl);
    if (!have && nfm >= 4) {  // too long for accumulators in registers
      use = 1;
      have = halo_plan(p.form, p.nx, use, p.nf, p.nprobe, max_cluster, pl);
    }
    if (!have) break;
    const Halo1DArgs a{p, s, t0, nsteps, pl.n, pl.L};
    int rc = FDTD_ERR_ARG;
    switch (p.form) {
      case FDTD1D_FORM_CB: rc = launch_fd1d_halo_cb(a, pl, use, st); break;
      case FDTD1D_FORM_CACB: rc = launch_fd1d_halo_cacb(a, pl, use, st); break;
      case FDTD1D_FORM_DFORM: rc = launch_fd1d_halo_dform(a, pl, use, st); break;
      case FDTD1D_FORM_DEBYE: rc = launch_fd1d_halo_debye(a, pl, use, st); break;
    }
    if (rc != FDTD_ERR_UNSUPPORTED) return rc;
  }
  // a device that takes no 16-block cluster, and a line that 8 blocks do not hold
  for (int t = t0 + 1; t <= t0 + nsteps; ++t) {
    int rc = launch_fd1d_efield(t, p, s, st);
    if (!rc && p.nf > 0) rc = launch_fd1d_fourier(t, p, s, st);
    if (!rc) rc = launch_fd1d_hfield(p, s, st);
    if (rc) return rc;
  }
  return FDTD_OK;
}

int launch_fd1d_efield(int t, const fdtd1d_params& p, const fdtd1d_state& s, cudaStream_t st) {
  const int blocks = (p.nx + 255) / 256;
  switch (p.form) {
    case FDTD1D_FORM_CB: k_fd1d_efield<FDTD1D_FORM_CB><<<blocks, 256, 0, st>>>(p, s, t); break;
    case FDTD1D_FORM_CACB: k_fd1d_efield<FDTD1D_FORM_CACB><<<blocks, 256, 0, st>>>(p, s, t); break;
    case FDTD1D_FORM_DFORM: k_fd1d_efield<FDTD1D_FORM_DFORM><<<blocks, 256, 0, st>>>(p, s, t); break;
    case FDTD1D_FORM_DEBYE: k_fd1d_efield<FDTD1D_FORM_DEBYE><<<blocks, 256, 0, st>>>(p, s, t); break;
    default: return FDTD_ERR_ARG;
  }
  int rc = fdtd_host::check_launch();
  if (rc) return rc;
  if (p.src_kind != FDTD_SRC_NONE && p.src_k == 0) {
    k_fd1d_src0<<<1, 1, 0, st>>>(p, s, t);
    rc = fdtd_host::check_launch();
  }
  return rc;
}

int launch_fd1d_hfield(const fdtd1d_params& p, const fdtd1d_state& s, cudaStream_t st) {
  k_fd1d_hfield<<<(p.nx + 255) / 256, 256, 0, st>>>(p, s);
  return fdtd_host::check_launch();
}

int launch_fd1d_fourier(int t, const fdtd1d_params& p, const fdtd1d_state& s, cudaStream_t st) {
  const int n = std::max(p.full_dft ? p.nx : 0, p.nf);
  k_fd1d_fourier<<<(n + 255) / 256, 256, 0, st>>>(p, s, t);
  return fdtd_host::check_launch();
}

}  // namespace fdtd

// ============================================================ C-ABI
namespace {

int check1d(const fdtd1d_params* p, const fdtd1d_state* s, int t_last) {
  if (!p || !s) return FDTD_ERR_NULL;
  if (p->nx < 4) return FDTD_ERR_SIZE;
  if (!s->ex || !s->hy) return FDTD_ERR_NULL;
  switch (p->form) {
    case FDTD1D_FORM_CB:
      if (!p->cb) return FDTD_ERR_NULL;
      break;
    case FDTD1D_FORM_CACB:
      if (!p->ca || !p->cb) return FDTD_ERR_NULL;
      break;
    case FDTD1D_FORM_DFORM:
      if (!p->nax || !p->nbx || !s->dx || !s->ix) return FDTD_ERR_NULL;
      break;
    case FDTD1D_FORM_DEBYE:
      if (!p->nax || !p->nbx || !p->ncx || !p->ndx || !s->dx || !s->ix || !s->sx) return FDTD_ERR_NULL;
      break;
    default: return FDTD_ERR_ARG;
  }
  if (p->src_kind < FDTD_SRC_NONE || p->src_kind > FDTD_SRC_SOFT) return FDTD_ERR_ARG;
  if (p->src_kind != FDTD_SRC_NONE) {
    if (p->src_k < 0 || p->src_k >= p->nx) return FDTD_ERR_ARG;
    if (!p->src_table) return FDTD_ERR_NULL;
    if (t_last > p->src_table_len) return FDTD_ERR_SIZE;
  }
  if (p->abc && !s->bc) return FDTD_ERR_NULL;
  if (p->nf < 0 || p->nf > 1024) return FDTD_ERR_SIZE;
  if (p->nprobe < 0 || p->nprobe > FDTD1D_MAX_PROBES) return FDTD_ERR_SIZE;
  if (p->nf > 0) {
    if (!p->dft_cos || !p->dft_sin) return FDTD_ERR_NULL;
    if (t_last > p->dft_table_len) return FDTD_ERR_SIZE;
    if (p->full_dft && (!s->r_pt || !s->i_pt)) return FDTD_ERR_NULL;
    if (p->nprobe > 0 && (!s->r_pr || !s->i_pr)) return FDTD_ERR_NULL;
    for (int q = 0; q < p->nprobe; ++q)
      if (p->probe_k[q] < 0 || p->probe_k[q] >= p->nx) return FDTD_ERR_ARG;
  }
  return FDTD_OK;
}

}  // namespace

extern "C" {

int fdtd1d_efield(int t, const fdtd1d_params* p, fdtd1d_state* s, fdtd_stream_t stream) {
  int rc = check1d(p, s, t);
  if (rc) return rc;
  if (t < 1) return FDTD_ERR_ARG;
  return fdtd::launch_fd1d_efield(t, *p, *s, (cudaStream_t)stream);
}

int fdtd1d_hfield(const fdtd1d_params* p, fdtd1d_state* s, fdtd_stream_t stream) {
  int rc = check1d(p, s, 0);
  if (rc) return rc;
  return fdtd::launch_fd1d_hfield(*p, *s, (cudaStream_t)stream);
}

int fdtd1d_fourier(int t, const fdtd1d_params* p, fdtd1d_state* s, fdtd_stream_t stream) {
  int rc = check1d(p, s, t);
  if (rc) return rc;
  if (t < 1 || p->nf <= 0) return FDTD_ERR_ARG;
  return fdtd::launch_fd1d_fourier(t, *p, *s, (cudaStream_t)stream);
}

int fdtd1d_step_n(const fdtd1d_params* p, fdtd1d_state* s, int t0, int nsteps, fdtd_stream_t stream) {
  if (t0 < 0 || nsteps < 0) return FDTD_ERR_ARG;
  int rc = check1d(p, s, t0 + nsteps);
  if (rc) return rc;
  if (nsteps == 0) return FDTD_OK;
  if (p->nx > FDTD1D_MAX_FUSED_NX) return FDTD_ERR_SIZE;
  return fdtd::launch_fd1d_run(*p, *s, t0, nsteps, (cudaStream_t)stream);
}

}  // extern "C"
