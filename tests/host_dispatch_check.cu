// Host-only check of what the 2D entry points launch (simulation_gb300/csrc/
// capi_2d.cu, or with -DADJOINT adjoint_run.cu), built by tests/test_host_dispatch.py
// and run on the CPU: the CUDA runtime calls and the kernel launchers that the file uses
// are replaced by fakes that record their arguments, on a pretended device of 152
// SMs.  Pointers are never dereferenced.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#ifndef ADJOINT
#include "fd2d_chain.cuh"
#endif
#include "fd2d_internal.cuh"
#include "fd2d_tile.h"

namespace fake {

struct Launch {
  std::string name;
  int* status = nullptr;
  bool finite = false;  // the launch tests the fields for Inf/NaN
  int t0 = 0, n = 0;
};
struct Clear {
  char* p;
  size_t bytes;
};
std::vector<Launch> launches;
std::vector<Clear> clears;
bool march_set = false;  // the caller has set a march shape

cudaError_t get_device(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t attribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
  return cudaSuccess;
}
cudaError_t memset_async(void* p, int, size_t n, cudaStream_t) {
  clears.push_back({(char*)p, n});
  return cudaSuccess;
}
cudaError_t memcpy_async(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t stream_create(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)0x100;
  return cudaSuccess;
}
cudaError_t event_create(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t)0x100;
  return cudaSuccess;
}
cudaError_t event_record(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t wait_event(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }

}  // namespace fake

namespace fdtd_host {
void note_cuda_error(cudaError_t) {}
int check_launch() {
  (void)cudaGetLastError();
  return FDTD_OK;
}
}  // namespace fdtd_host

namespace fdtd {

static int log(const char* name, int* status, bool finite, int t0, int n) {
  fake::launches.push_back({name, status, finite, t0, n});
  return FDTD_OK;
}
using P = const fdtd2d_params&;
using S = const fdtd2d_state&;
using FS = const FieldSet&;
using St = cudaStream_t;

int launch_dfield(int, P, S, St) { return log("dfield", nullptr, false, 0, 0); }
int launch_efield(P, S, St) { return log("efield", nullptr, false, 0, 0); }
int launch_hfield(P, S, St) { return log("hfield", nullptr, false, 0, 0); }
int launch_ezinct(P, S, St) { return log("ezinct", nullptr, false, 0, 0); }
int launch_inctdz(P, S, St) { return log("inctdz", nullptr, false, 0, 0); }
int launch_hxinct(P, S, St) { return log("hxinct", nullptr, false, 0, 0); }
int launch_incth(P, S, St) { return log("incth", nullptr, false, 0, 0); }
int launch_fourier(int, P, S, St) { return log("fourier", nullptr, false, 0, 0); }
int launch_step3(int t, P, S, St) { return log("step3", nullptr, false, t - 1, 1); }
int launch_dielectric(int, int, int, double, double, double, double, float*, float*, St) { return FDTD_OK; }
int launch_pad(FS, FS, const float*, float*, const float*, float*, int, int, int, St) {
  return log("pad", nullptr, false, 0, 0);
}
int launch_unpad(FS, FS, const float*, float*, int, int, int, St) { return log("unpad", nullptr, false, 0, 0); }
int launch_check_finite(const float*, size_t, int* status, St) { return log("check_finite", status, true, 0, 0); }
int launch_march(P, FS, FS, float*, int t0, int k, int* status, float*, St) {
  return log("march", status, status != nullptr, t0, k);
}
int launch_march_record(P, FS, FS, float*, int t0, int k, const RecSet*, St) {
  return log("march_record", nullptr, false, t0, k);
}
int launch_march_ext(P, FS, FS, float*, int t0, int k, int* status, const MarchExt&, St) {
  return log("march_ext", status, status != nullptr, t0, k);
}
int launch_dft_rec(int, int, int, int t0, int n, int, const float*, const float*, const float*, size_t, float*, float*,
                   St) {
  return log("dft_rec", nullptr, false, t0, n);
}
int launch_inc_line(P, S, int t0, int n, float*, float*, St) { return log("inc_line", nullptr, false, t0, n); }
int launch_chain(P, int, const float*, const float*, FS, FS, float*, int t0, int k, int* status, float, St) {
  return log("chain", status, status != nullptr, t0, k);
}
int launch_chain_ext(P, int, const float*, const float*, FS, FS, float*, int t0, int k, int* status, float,
                     const MarchExt&, float*, size_t, St) {
  return log("chain_ext", status, status != nullptr, t0, k);
}
int launch_tile(P, FS, FS, FS, FS, float*, int t0, int n, int* status, float*, unsigned*, const TilePlan&, St, int mode,
                const TileAdj*, const TileExt*, bool finite) {
  static const char* const kName[] = {"tile", "tile_rec", "tile_rev", "tile_ext"};
  return log(kName[mode], status, finite && status, t0, n);
}
int launch_adjoint_fused(P, int t, const fdtd2d_fields&, const fdtd2d_fields&, const fdtd2d_fields&, int, int, float,
                         const fdtd2d_box&, float*, float*, St) {
  return log("adjoint_fused", nullptr, false, t, 1);
}
int launch_adjoint_fused2(P, int t, const fdtd2d_fields&, const fdtd2d_fields&, const fdtd2d_fields&,
                          const fdtd2d_fields&, int, int, float, const fdtd2d_box&, float*, float*, St) {
  return log("adjoint_fused2", nullptr, false, t, 2);
}
int march_max_steps_per_pass() { return 4; }
int march_default_steps(int, int) { return 2; }
float march_gen_cost() { return 0.f; }
bool march_shape_set() { return fake::march_set; }
bool chain_better(int nx, int ny) { return !fake::march_set && (long long)nx * ny > (1 << 20); }
bool chain_ext_better(int nx, int ny) { return chain_better(nx, ny); }
bool march_ext_supported(P p) { return p.nf <= kMarchMaxNf; }

}  // namespace fdtd

#define cudaGetDevice fake::get_device
#define cudaDeviceGetAttribute fake::attribute
#define cudaMemsetAsync fake::memset_async
#define cudaMemcpyAsync fake::memcpy_async
#define cudaStreamCreateWithFlags fake::stream_create
#define cudaEventCreateWithFlags fake::event_create
#define cudaEventRecord fake::event_record
#define cudaStreamWaitEvent fake::wait_event
#ifdef ADJOINT
#include "adjoint_run.cu"
#else
#include "capi_2d.cu"
#endif

namespace {

int g_fail = 0;
void expect(bool ok, const char* what) {
  if (!ok) std::printf("FAIL %s\n", what);
  g_fail += !ok;
}

float* const F = (float*)0x100000;  // an aligned address
char* const WS = (char*)0x40000000;

fdtd2d_params params(int nx, int ny) {
  fdtd2d_params p{};
  p.nx = nx;
  p.ny = ny;
  p.naz = F;
  p.pml = {F, F, F, F, F, F, F, F, F, F};
  return p;
}
[[maybe_unused]] fdtd2d_state state() {
  fdtd2d_state s{};
  s.dz = s.ez = s.iz = s.hx = s.hy = s.ihx = s.ihy = s.ezi = s.hxi = s.bc = s.r_pt = s.i_pt = s.r_in = s.i_in = F;
  s.status = (int*)0x2000;
  return s;
}
[[maybe_unused]] int count(const char* name) {
  int n = 0;
  for (const fake::Launch& l : fake::launches) n += l.name == name;
  return n;
}
void reset() {
  fake::launches.clear();
  fake::clears.clear();
}

#ifndef ADJOINT
// every launch of the on-chip loop, whose blocks wait on one another, can report a
// wait that runs out; the Inf/NaN test is the last one's alone
void check_ext_status() {
  fdtd2d_params p = params(100, 96);
  p.tfsf_npml = 8;
  p.tfsf_table = F;
  p.tfsf_table_len = 1000;
  fdtd2d_state s = state();
  reset();
  const size_t n = fdtd2d_fast_workspace_size(&p, 0);
  expect(fdtd2d_step_n(&p, &s, 0, 150, 0, WS, n, nullptr) == FDTD_OK, "step_n with a plane wave");
  expect(count("tile_ext") == 3, "three launches of 64, 64 and 22 steps");
  int seen = 0;
  for (const fake::Launch& l : fake::launches)
    if (l.name == "tile_ext") {
      ++seen;
      expect(l.status == s.status, "plane wave: the launch has the caller's status word");
      expect(l.finite == (seen == 3), "plane wave: the last launch alone tests for Inf/NaN");
    }
}

// a march shape that the caller has set is used where the library would otherwise
// take the loop on the chip, as it is on larger grids
void check_march_shape() {
  for (bool ext : {false, true}) {
    fdtd2d_params p = params(100, 96);
    if (ext) {
      p.nf = 2;
      p.dft_cos = p.dft_sin = F;
      p.dft_table_len = 1000;
    }
    fdtd2d_state s = state();
    const size_t n = fdtd2d_fast_workspace_size(&p, 0);
    for (bool set : {false, true}) {
      reset();
      fake::march_set = set;
      expect(fdtd2d_step_n(&p, &s, 0, 24, 0, WS, n, nullptr) == FDTD_OK, "step_n");
      expect((count(ext ? "tile_ext" : "tile") > 0) == !set, "on the chip unless a march shape is set");
      expect((count(ext ? "march_ext" : "march") > 0) == set, "marching where a march shape is set");
    }
    fake::march_set = false;
  }
}
// no layout for grids far beyond the chip, up to the largest extents that are taken
void check_plan_extents() {
  for (int n : {2000, 1 << 20, 2147483647 - 100, 2147483647})
    for (bool lossy : {false, true})
      for (bool pml : {false, true}) {
        TilePlan pl;
        expect(!tile_plan(n, n == 2000 ? n : 4000, lossy, pml, 152, pl), "no layout");
        expect(!tile_plan(n == 2000 ? n : 4000, n, lossy, pml, 152, pl), "no layout");
        if (n > 2000) expect(!tile_plan(n, 3, lossy, pml, 152, pl) && !tile_plan(3, n, lossy, pml, 152, pl), "no layout");
      }
  for (int nx : {3, 100, 1024, 1080})
    for (int ny : {3, 100, 960, 1024}) {
      TilePlan pl;
      expect(tile_plan(nx, ny, true, true, 152, pl), "a layout");
      expect((long long)pl.n_ti * pl.own_r >= nx && (long long)pl.n_tj * pl.own_c >= ny && pl.n_ti * pl.n_tj <= 152,
             "the layout covers the grid");
    }
  fdtd2d_params p = params(2147483647 - 10, 3);
  fdtd2d_state s = state();
  reset();
  expect(fdtd2d_step_n(&p, &s, 0, 8, 0, WS, ~(size_t)0, nullptr) == FDTD_OK && count("step3") == 8,
         "a grid of 2^31 rows steps in three launches");
}
#else
// the adjoint's launches report into words of the workspace that the call clears first
void check_adjoint_status() {
  fdtd2d_params p = params(64, 64);
  for (int checkpoint : {16, 64}) {
    fdtd2d_adjoint_params a{100, checkpoint, 40, 32, 2.f, {20, 20, 16, 16}};
    const size_t n = fdtd2d_tm_adjoint_workspace_size(&p, &a);
    const size_t off = fdtd2d_tm_adjoint_status_offset(&p, &a);
    expect(off > 0 && off % 4 == 0 && off + 8 <= n, "adjoint: the status words are in the workspace");
    using Run = int (*)(const fdtd2d_params*, const fdtd2d_adjoint_params*, size_t);
    const Run runs[] = {
        [](const fdtd2d_params* p, const fdtd2d_adjoint_params* a, size_t n) {
          return fdtd2d_tm_adjoint_forward(p, a, F, nullptr, WS, n, nullptr);
        },
        [](const fdtd2d_params* p, const fdtd2d_adjoint_params* a, size_t n) {
          return fdtd2d_tm_adjoint_forward_rec(p, a, F, nullptr, WS, n, nullptr);
        },
        [](const fdtd2d_params* p, const fdtd2d_adjoint_params* a, size_t n) {
          return fdtd2d_tm_adjoint_reverse(p, a, F, nullptr, WS, n, nullptr);
        },
        [](const fdtd2d_params* p, const fdtd2d_adjoint_params* a, size_t n) {
          return fdtd2d_tm_adjoint_reverse_rec(p, a, F, nullptr, WS, n, nullptr);
        }};
    for (int k = 0; k < 4; ++k) {
      reset();
      expect(runs[k](&p, &a, n) == FDTD_OK, "adjoint call");
      const bool forward = k < 2;
      char* const word = WS + off + (forward ? 0 : 4);
      int tiles = 0;
      for (const fake::Launch& l : fake::launches) {
        if (l.name.compare(0, 4, "tile")) continue;
        ++tiles;
        expect((char*)l.status == word, "adjoint: the launch has its half's status word");
        expect(!l.finite, "adjoint: no Inf/NaN test");
      }
      expect(tiles > 0, "adjoint: on the chip");
      bool cleared = false, other = false;
      for (const fake::Clear& c : fake::clears) {
        cleared |= c.p <= word && word + 4 <= c.p + c.bytes;
        other |= !forward && c.p <= word - 4 && word <= c.p + c.bytes;  // the forward's outcome, still to be read
      }
      expect(cleared && !other, "adjoint: the half clears its own status word");
    }
  }
}

#endif

}  // namespace

int main() {
#ifdef ADJOINT
  check_adjoint_status();
#else
  check_ext_status();
  check_march_shape();
  check_plan_extents();
#endif
  if (g_fail) return 1;
  std::printf("ok\n");
  return 0;
}
