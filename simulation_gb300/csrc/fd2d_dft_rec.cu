// The running DFT of Ez from a record of its values: what fourier
// (fd2d/python/fd2d_3_4.py:90-99) adds step by step, over many steps at once.
#include "fd2d_internal.cuh"

namespace fdtd {
namespace {

struct DftRecArgs {
  size_t n;        // items of V cells
  int steps, nf, f0;
  const float* ez;  // step s at ez + s*slot
  size_t slot;
  int ny, pitch;   // columns of a row of the accumulators, and of the record (V = 1 where they differ)
  const float* cs;  // [step][nf]
  const float* sn;
  float *re, *im;   // [nf][n*V]
};

// Bound by HBM or L2: each recorded value is read once for the NF frequencies of
// the launch, each accumulator read and written once; a thread keeps V cells'
// accumulators in registers over the steps, whose reads are in flight eight at a
// time.  One fma per value and accumulator, in the order of the steps.
template <int NF, int V>
__global__ void __launch_bounds__(256) k_dft_rec(const DftRecArgs a) {
  const size_t n = blockIdx.x * (size_t)256 + threadIdx.x;
  if (n >= a.n) return;
  const size_t c = n * V;
  const size_t ce = V == 1 && a.pitch != a.ny ? c / a.ny * a.pitch + c % a.ny : c;
  auto ld = [](const float* p, float (&v)[V]) {
    if constexpr (V == 4) {
      const float4 x = __ldcs(reinterpret_cast<const float4*>(p));
      v[0] = x.x;
      v[1] = x.y;
      v[2] = x.z;
      v[3] = x.w;
    } else {
      v[0] = __ldcs(p);
    }
  };
  auto st = [](float* p, const float (&v)[V]) {
    if constexpr (V == 4) __stcs(reinterpret_cast<float4*>(p), make_float4(v[0], v[1], v[2], v[3]));
    else __stcs(p, v[0]);
  };
  float re[NF][V], im[NF][V];
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    ld(a.re + (size_t)(a.f0 + f) * a.n * V + c, re[f]);
    ld(a.im + (size_t)(a.f0 + f) * a.n * V + c, im[f]);
  }
  const float* cs = a.cs + a.f0;
  const float* sn = a.sn + a.f0;
  auto add = [&](int s, const float (&e)[V]) {
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const float x = __ldg(cs + (size_t)s * a.nf + f), y = -__ldg(sn + (size_t)s * a.nf + f);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        re[f][k] = __fmaf_rn(x, e[k], re[f][k]);
        im[f][k] = __fmaf_rn(y, e[k], im[f][k]);
      }
    }
  };
  int s = 0;
  for (; s + 8 <= a.steps; s += 8) {
    float e[8][V];
#pragma unroll
    for (int q = 0; q < 8; ++q) ld(a.ez + (s + q) * a.slot + ce, e[q]);
#pragma unroll
    for (int q = 0; q < 8; ++q) add(s + q, e[q]);
  }
  for (; s < a.steps; ++s) {
    float e[V];
    ld(a.ez + s * a.slot + ce, e);
    add(s, e);
  }
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    st(a.re + (size_t)(a.f0 + f) * a.n * V + c, re[f]);
    st(a.im + (size_t)(a.f0 + f) * a.n * V + c, im[f]);
  }
}

template <int V>
int launch_v(DftRecArgs a, cudaStream_t st) {
  const unsigned blocks = (unsigned)((a.n + 255) / 256);
  for (; a.f0 < a.nf; a.f0 += 4) {
    switch (std::min(a.nf - a.f0, 4)) {
      case 1: k_dft_rec<1, V><<<blocks, 256, 0, st>>>(a); break;
      case 2: k_dft_rec<2, V><<<blocks, 256, 0, st>>>(a); break;
      case 3: k_dft_rec<3, V><<<blocks, 256, 0, st>>>(a); break;
      default: k_dft_rec<4, V><<<blocks, 256, 0, st>>>(a); break;
    }
    const int rc = fdtd_host::check_launch();
    if (rc) return rc;
  }
  return FDTD_OK;
}

}  // namespace

int launch_dft_rec(int nx, int ny, int pitch, int t0, int steps, int nf, const float* dft_cos, const float* dft_sin, const float* ez,
                   size_t slot, float* r_pt, float* i_pt, cudaStream_t st) {
  // table row t-1 = t0+s of step t0+s+1
  const size_t ncell = (size_t)nx * ny;
  DftRecArgs a{ncell, steps, nf, 0, ez, slot, ny, pitch, dft_cos + (size_t)t0 * nf, dft_sin + (size_t)t0 * nf, r_pt, i_pt};
  if (pitch == ny && ncell % 4 == 0 && slot % 4 == 0 && (((uintptr_t)ez | (uintptr_t)r_pt | (uintptr_t)i_pt) & 15u) == 0) {
    a.n = ncell / 4;
    return launch_v<4>(a, st);
  }
  return launch_v<1>(a, st);
}

}  // namespace fdtd
