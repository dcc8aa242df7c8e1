// Batched uneven 1D runs (thousands of independent lossy-slab simulations in
// one persistent launch), with the running-DFT probes fused in.
//
// Each run is the ca/cb lossy 1D program of fd1d/program/fd1d_1_5.py:63-72
// (E update, soft Gaussian source, two-step-back ABC, H update) with per-run
// layered coefficients and two DFT probes accumulated as in
// fd1d/program/fd1d_2_2.py:65-71 (after E, before the ABC).  The reference has
// no batched form; this is the library's extension for spectra sweeps.
//
// Execution model:
//   * a run is executed by a TEAM of warps inside a thread block: each lane
//     holds CPT consecutive cells (ex, hy) in registers and warp shuffles carry
//     the neighbour values inside a warp;
//   * neighbouring warps overlap by one lane: lane 31 of a warp and lane 0 of
//     the next hold the same CPT cells, the first half owned by the former, the
//     second by the latter, and each advances the other's half redundantly.
//     Wrong values creep in by one cell a step, so the warps exchange their
//     halves once in H = CPT/2 steps, with ONE team barrier (a named barrier
//     `bar.sync id, n`), instead of two barriers in every step;
//   * the cells' updates are packed two to an instruction (f32x2: the same
//     rounding), 3.5 instructions per cell-step.  A warp whose lanes each lie
//     in one material reads its (ca, cb) from two registers; only warps that
//     hold a material boundary read per-cell pairs from shared memory, where
//     they are expanded from the layer table once per run;
//   * the probe cells are sampled into shared memory and the team adds the
//     samples to its DFT accumulators once per exchange, spread over its warps;
//   * the host planner (fdtd1d_batch_plan, C++ below) sizes each team as
//     ceil(ke / cells_per_thread) rounded up to whole warps, so every run costs
//     about the same per step, and packs teams into "bundles" that fill a block
//     (first-fit decreasing, <= 15 multi-warp teams per block).  A lane holds
//     two cells more than the plan's cells_per_thread, which more than pays for
//     the overlaps, so every run that the plan admits fits its team;
//   * persistent blocks take bundles from a device counter (atomicAdd); there
//     is no spin-wait anywhere.  An optional clock budget stops a block from
//     taking new bundles and raises FDTD_STATUS_TIMEOUT; per-run `done` flags
//     say which runs finished.
// What bounds it: the FP32 pipe and issue slots (5 FP32 operations and 3.5
// instructions per cell-step, four warps per scheduler).
#include <algorithm>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <utility>
#include <vector>

#include "fdtd_common.cuh"

namespace fdtd {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int MAX_WARPS = 32;
constexpr int ENTRY_INTS = 4;  // run, threads, thread offset, barrier id (0 = single warp)

struct BatchArgs {
  fdtd1d_batch_params p;
  fdtd1d_batch_out o;
  const int* plan;  // device copy of the plan
  int nbundles;
  const int* bstart;  // [nbundles+1] entry offsets (into plan)
  const int* entries;
  long long max_cycles;
};

__device__ __forceinline__ void team_sync(int bar_id, int nthreads) {
  if (bar_id == 0) {
    __syncwarp();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(nthreads) : "memory");
  }
}

// body(K) for each of the up to 7 cells K around the runtime cell c, which is
// the same in the whole warp: a tree of uniform branches to a short run of
// straight-line code, in which the body selects its lane and cell by
// predicates.  (An indexed branch to one of 42 cases took more than the whole
// step: 44 ms against 20 without any special cell, for 4096 runs of 2000
// steps.)
template <int LO, class F, int... K>
__device__ __forceinline__ void cell_each(F& body, std::integer_sequence<int, K...>) {
  (body(std::integral_constant<int, LO + K>{}), ...);
}
template <int LO, int HI, class F>
__device__ __forceinline__ void cell_at(int c, F&& body) {
  if constexpr (HI - LO <= 7) {
    cell_each<LO>(body, std::make_integer_sequence<int, HI - LO>{});
  } else {
    constexpr int MID = (LO + HI) / 2;
    if (c < MID) cell_at<LO, MID>(c, body);
    else cell_at<MID, HI>(c, body);
  }
}
// cell K of a packed register array
template <int K, int N>
__device__ __forceinline__ float& cell(float2 (&a)[N]) {
  if constexpr (K % 2 == 0) return a[K / 2].x;
  else return a[K / 2].y;
}
// cells [LO, LO+N) to or from consecutive floats, in pairs where they are aligned (p: pairs start at even offsets)
template <int LO, int N, int M>
__device__ __forceinline__ void cells_put(float2 (&a)[M], float* p) {
  if constexpr (LO % 2) *p = cell<LO>(a);
#pragma unroll
  for (int k = (LO + 1) / 2; k < (LO + N) / 2; ++k) *reinterpret_cast<float2*>(p + 2 * k - LO / 2 * 2) = a[k];
  if constexpr ((LO + N) % 2) p[LO + N - 1 - LO / 2 * 2] = cell<LO + N - 1>(a);
}
template <int LO, int N, int M>
__device__ __forceinline__ void cells_get(float2 (&a)[M], const float* p) {
  if constexpr (LO % 2) cell<LO>(a) = *p;
#pragma unroll
  for (int k = (LO + 1) / 2; k < (LO + N) / 2; ++k) a[k] = *reinterpret_cast<const float2*>(p + 2 * k - LO / 2 * 2);
  if constexpr ((LO + N) % 2) cell<LO + N - 1>(a) = p[LO + N - 1 - LO / 2 * 2];
}

// a 16-byte shared-memory read that stays where it is written (the compiler
// would sink it to its use, which then waits for it)
__device__ __forceinline__ float4 lds4(const float4* p) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"((unsigned)__cvta_generic_to_shared(p)));
  return v;
}

// floats of one warp's edge buffer (ex and hy of half a lane, padded to pairs) and of one team's probe samples
__host__ __device__ constexpr int edge_floats(int cpt) { return 2 * ((cpt / 2 + 2) / 2 * 2); }
__host__ __device__ constexpr int sample_floats(int cpt) { return 2 * (cpt / 2 + 1); }

template <int CPT>
__device__ void run_team(const BatchArgs& A, int run, int T, int tt, int bar_id, int wb, float4* coef, float* edges,
                         float* samples, float* acc) {
  static_assert(CPT / 2 <= 32, "one lane per source value of an epoch");
  constexpr int H = CPT / 2, NP = CPT / 2, EF = edge_floats(CPT), HF = EF / 2, SF = sample_floats(CPT);
  const fdtd1d_batch_params& p = A.p;
  const int lane = threadIdx.x & 31;
  const int w = tt >> 5;  // warp index inside the team
  const int nx = p.ke[run];
  // warps that hold cells: cell 31*CPT*w is the first of warp w
  const int nw = nx <= 32 * CPT ? 1 : ((nx + CPT - 1) / CPT - 1 + 30) / 31;
  const int g0 = (31 * w + lane) * CPT;  // first cell of this lane
  const bool active = w < nw;

  // expand the layer table: background ca=1, cb=0.5 (free space of fd1d_1_5).
  // Cells past the run's end are free space too, so the cell loops need no
  // range test: nothing flows back from them, since ex[nx-1] is set by the ABC
  // after every E update (nor from hy[nx-1], which only that update reads; it
  // is kept at 0, as the reference never updates it, where a probe sees the
  // updated ex[nx-1] before the ABC).
  const int l0 = p.layer_off[run], l1 = p.layer_off[run + 1];
  float2 ca = make_float2(1.f, 1.f), cb = make_float2(0.5f, 0.5f);  // of a lane in one material
  bool one = true;
  if (active) {
    float4* const mine = coef + (size_t)w * NP * 32 + lane;  // [pair][lane]: 16-byte reads without bank conflicts
#pragma unroll 1
    for (int k = 0; k < NP; ++k) {
      float a2[2], b2[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = g0 + 2 * k + h;
        a2[h] = 1.f;
        b2[h] = 0.5f;
        if (i < nx)
          for (int l = l0; l < l1; ++l)
            if (i >= p.layer_start[l] && i < p.layer_end[l]) {
              a2[h] = p.layer_ca[l];
              b2[h] = p.layer_cb[l];
            }
        if (k == 0 && h == 0) {
          ca = make_float2(a2[0], a2[0]);
          cb = make_float2(b2[0], b2[0]);
        }
        one &= a2[h] == ca.x && b2[h] == cb.x;
      }
      mine[k * 32] = make_float4(a2[0], a2[1], b2[0], b2[1]);
    }
  }
  const bool uniform = __all_sync(FULL, one);
  const float4* const my_coef = coef + (size_t)w * NP * 32 + lane;  // read by the lane that wrote it
  const int pin = p.probe_in[run], pout = p.probe_out[run];
  const int nf = p.nf;
  // DFT accumulators of the team in shared memory: acc[4][nf] (re/im at the
  // entry probe, re/im at the exit probe)
  for (int f = tt; f < 4 * nf; f += T) acc[f] = 0.f;

  float2 ex[NP], hy[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) ex[k] = hy[k] = make_float2(0.f, 0.f);
  // the lanes (and their cells) that differ: cell 0 and 1, nx-1, the source
  // (in both copies of an overlap), the probes (in their owner)
  const bool owned = active && !(lane == 0 && w > 0) && !(lane == 31 && w < nw - 1);
  auto holds = [&](int k) { return active && k / CPT == g0 / CPT; };
  // the owner of a cell in an overlap holds it in its half of the lane
  auto owns = [&](int k) {
    return holds(k) && (owned || (lane == 31 ? k - g0 < H : k - g0 >= H));
  };
  // the cell (in its lane) of a special cell that this warp holds, in the whole
  // warp, or -1; and the same in the one lane that holds it, -1 in the others
  auto in_warp = [&](bool mine, int k) { return __any_sync(FULL, mine) ? k % CPT : -1; };
  const bool src_l = holds(p.src_k), pin_l = owns(pin), pout_l = owns(pout), hi_l = w == nw - 1 && holds(nx - 1);
  const int src_c = in_warp(src_l, p.src_k), pin_c = in_warp(pin_l, pin), pout_c = in_warp(pout_l, pout),
            hi_c = in_warp(hi_l, nx - 1);
  const bool end_probe = pin == nx - 1 || pout == nx - 1;
  const bool lo_warp = w == 0;
  const bool special = lo_warp || src_c >= 0 || pin_c >= 0 || pout_c >= 0 || hi_c >= 0;
  float bc0 = 0.f, bc1 = 0.f, bc2 = 0.f, bc3 = 0.f;
  const float2 half = make_float2(0.5f, 0.5f);

  // steps i0 .. i1-1 of an epoch, samples into smp, the epoch's source values vs in lane order;
  // UNI: every lane in one material; SPEC: the warp holds cells that differ
  auto steps = [&](auto uni_tag, auto spec_tag, const int i0, const int i1, float* smp, const float vs) {
    constexpr int PFD = 4;
    constexpr bool UNI = decltype(uni_tag)::value, SPEC = decltype(spec_tag)::value;
#pragma unroll 1
    for (int i = i0; i < i1; ++i) {
      // ---------------- E stage: ex = ca*ex + cb*(hy[i-1]-hy[i])
      float4 kc[UNI ? 1 : PFD];  // coefficients of the next PFD pairs, on their way from shared memory
      if constexpr (!UNI) {
#pragma unroll
        for (int k = 0; k < PFD; ++k) kc[k] = lds4(my_coef + k * 32);
      }
      const float hy_left = __shfl_up_sync(FULL, hy[NP - 1].y, 1);
      const float ex0 = ex[0].x;
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        const float hym = (k == 0) ? hy_left : hy[k - 1].y;
        const float2 d = make_float2(__fsub_rn(hym, hy[k].x), __fsub_rn(hy[k].x, hy[k].y));
        if constexpr (UNI) {
          ex[k] = __ffma2_rn(ca, ex[k], __fmul2_rn(cb, d));
        } else {
          const float4 c = kc[k % PFD];
          if (k + PFD < NP) kc[k % PFD] = lds4(my_coef + (k + PFD) * 32);
          ex[k] = __ffma2_rn(make_float2(c.x, c.y), ex[k], __fmul2_rn(make_float2(c.z, c.w), d));
        }
      }
      if constexpr (SPEC) {
        if (lo_warp) ex[0].x = lane == 0 ? ex0 : ex[0].x;  // cell 0 is not E-updated
        // soft source, fd1d/program/fd1d_1_5.py:67 (a pulse that has passed adds
        // exact zeros: skipped), then the probes read their cells
        const float v = __shfl_sync(FULL, vs, i);
        if (src_c >= 0 && v != 0.f)
          cell_at<0, CPT>(src_c, [&](auto K) {
            float& e = cell<decltype(K)::value>(ex);
            if (src_l && src_c == K) e = __fadd_rn(e, v);
          });
        if (pin_c >= 0) {
          float e = 0.f;
          cell_at<0, CPT>(pin_c, [&](auto K) { e = pin_c == K ? cell<decltype(K)::value>(ex) : e; });
          if (pin_l) smp[i] = e;
        }
        if (pout_c >= 0) {
          float e = 0.f;
          cell_at<0, CPT>(pout_c, [&](auto K) { e = pout_c == K ? cell<decltype(K)::value>(ex) : e; });
          if (pout_l) smp[H + i] = e;
        }
        // two-step-back ABC (fd1d/program/fd1d_1_2.py:47-48); the state moves
        // in every lane, only lane 0 and the lane of nx-1 use theirs
        if (lo_warp) {
          const float e1 = ex[0].y;
          ex[0].x = lane == 0 ? bc0 : ex[0].x;
          bc0 = bc1;
          bc1 = e1;
        }
        if (hi_c >= 0) {
          float e2 = __shfl_up_sync(FULL, ex[NP - 1].y, 1);  // nx-2 when nx-1 is its lane's first cell
          cell_at<0, CPT>(hi_c, [&](auto K) {
            constexpr int k = decltype(K)::value;
            float& e = cell<k>(ex);
            if constexpr (k > 0) e2 = hi_c == k ? cell<(k > 0 ? k - 1 : 0)>(ex) : e2;
            e = hi_l && hi_c == k ? bc3 : e;
          });
          bc3 = bc2;
          bc2 = e2;
        }
      }
      // ---------------- H stage
      float ex_right = __shfl_down_sync(FULL, ex[0].x, 1);
      if (SPEC && lane == 31) ex_right = 0.f;  // behind the run's end: keeps the cells there bounded
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        const float er = (k == NP - 1) ? ex_right : ex[k + 1].x;
        hy[k] = __ffma2_rn(half, make_float2(__fsub_rn(ex[k].x, ex[k].y), __fsub_rn(ex[k].y, er)), hy[k]);
      }
      if (SPEC && end_probe && hi_c >= 0)
        cell_at<0, CPT>(hi_c, [&](auto K) {
          float& h = cell<decltype(K)::value>(hy);
          if (hi_l && hi_c == K) h = 0.f;
        });
    }
  };

  // running DFT of an epoch's m samples (steps t+1 ..), in step order: item q =
  // (frequency, probe), spread evenly over the team's warps
  auto dft = [&](const float* smp, const int t, const int m) {
    const int tw = T >> 5;
    for (int q = lane * tw + w; q < 2 * nf; q += T) {
      const int f = q >> 1, pr = q & 1;
      const float* const e = smp + pr * H;
      const float* const dc = p.dft_cos + (size_t)t * nf + f;
      const float* const ds = p.dft_sin + (size_t)t * nf + f;
      float* const a = acc + 2 * pr * nf + f;
      float re = a[0], im = a[nf];
#pragma unroll 7
      for (int i = 0; i < m; ++i) {
        re = __fmaf_rn(__ldg(dc + (size_t)i * nf), e[i], re);
        im = __fmaf_rn(-__ldg(ds + (size_t)i * nf), e[i], im);
      }
      a[0] = re;
      a[nf] = im;
    }
  };

  team_sync(bar_id, T);  // the accumulators are cleared
  float vnext = lane < p.nsteps ? __ldg(p.src_table + lane) : 0.f;
  for (int t = 0, b = 0; t < p.nsteps; t += H, b ^= 1) {
    const int m = min(H, p.nsteps - t);
    float* const smp = samples + b * SF;
    const float vs = vnext;  // the next epoch's source values are on their way while this one runs
    if (special) vnext = t + H + lane < p.nsteps ? __ldg(p.src_table + t + H + lane) : 0.f;
    // the DFT of the epoch before is added part-way through this one, at another
    // step in each of a scheduler's warps: its table reads (L2) are then waited
    // for while the other warps compute (100 ns of a step's 1150 when all did it
    // behind the barrier)
    const int mid = min(m, (wb + w) / 4 * (H / 4));
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
      const int i0 = part ? mid : 0, i1 = part ? m : mid;
      if (active) {
        if (special) steps(std::false_type{}, std::true_type{}, i0, i1, smp, vs);
        else if (uniform) steps(std::true_type{}, std::false_type{}, i0, i1, smp, 0.f);
        else steps(std::false_type{}, std::false_type{}, i0, i1, smp, 0.f);
      }
      if (part == 0 && t > 0) dft(samples + (b ^ 1) * SF, t - H, H);
    }
    // exchange of the overlaps' halves; the two buffers alternate, so one
    // barrier orders both this exchange's reads and the next but one's writes
    float* const mine = edges + ((size_t)b * MAX_WARPS + wb + w) * 2 * EF;  // [left edge][right edge]
    if (active) {
      if (lane == 31 && w < nw - 1) {
        cells_put<0, H>(ex, mine + EF);
        cells_put<0, H>(hy, mine + EF + HF);
      }
      if (lane == 0 && w > 0) {
        cells_put<H, H>(ex, mine);
        cells_put<H, H>(hy, mine + HF);
      }
    }
    team_sync(bar_id, T);
    if (active) {
      if (lane == 0 && w > 0) {
        cells_get<0, H>(ex, mine - EF);  // warp w-1's right edge
        cells_get<0, H>(hy, mine - EF + HF);
      }
      if (lane == 31 && w < nw - 1) {
        cells_get<H, H>(ex, mine + 2 * EF);  // warp w+1's left edge
        cells_get<H, H>(hy, mine + 2 * EF + HF);
      }
    }
    if (t + H >= p.nsteps) dft(smp, t, m);  // the last epoch's
  }
  team_sync(bar_id, T);
  bool fin = true;
  float* sp = A.o.spec + (size_t)run * 4 * nf;
  for (int f = tt; f < 4 * nf; f += T) {
    sp[f] = acc[f];
    fin &= isfinite(acc[f]);
  }
  if (!fin) raise_status(A.o.status, ST_NONFINITE);
  if (tt == 0 && A.o.done) A.o.done[run] = 1;
}

template <int CPT, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1) k_batch(const BatchArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* coef = reinterpret_cast<float4*>(smem_raw);  // [blockDim * CPT / 2]
  const int nwarps = blockDim.x >> 5;
  float* edges = reinterpret_cast<float*>(coef + (size_t)blockDim.x * (CPT / 2));  // [2][MAX_WARPS][2][edge]
  float* x_smp = edges + (size_t)2 * MAX_WARPS * 2 * edge_floats(CPT);  // [warps][2][samples] (per team, by its first warp)
  float* x_acc = x_smp + (size_t)nwarps * 2 * sample_floats(CPT);       // [warps][4*64] DFT accumulators (per team)
  __shared__ int s_bundle;
  const long long t_start = clock64();
  for (;;) {
    if (threadIdx.x == 0) {
      int b = -1;
      if (A.max_cycles > 0 && clock64() - t_start > A.max_cycles) {
        // budget spent: take nothing more; report if work was left
        if (*(volatile unsigned*)A.o.queue < (unsigned)A.nbundles) raise_status(A.o.status, ST_TIMEOUT);
      } else {
        b = (int)atomicAdd(A.o.queue, 1u);
      }
      s_bundle = b;
    }
    __syncthreads();
    const int b = s_bundle;
    if (b < 0 || b >= A.nbundles) break;
    for (int e = A.bstart[b]; e < A.bstart[b + 1]; ++e) {
      const int* en = A.entries + (size_t)e * ENTRY_INTS;
      const int off = en[2], T = en[1];
      if ((int)threadIdx.x >= off && (int)threadIdx.x < off + T) {
        run_team<CPT>(A, en[0], T, threadIdx.x - off, en[3], off >> 5, coef + (size_t)(off >> 5) * 32 * (CPT / 2), edges,
                      x_smp + (size_t)(off >> 5) * 2 * sample_floats(CPT), x_acc + (size_t)256 * (off >> 5));
      }
    }
    __syncthreads();
  }
}

}  // namespace

// smem bytes of one block
static size_t batch_smem(int threads, int cpt) {
  const size_t warps = threads / 32;
  return (size_t)threads * (cpt / 2) * sizeof(float4) +
         sizeof(float) * ((size_t)2 * MAX_WARPS * 2 * edge_floats(cpt) + warps * (2 * sample_floats(cpt) + 256));
}

template <int CPT, int BLOCK>
static int launch_batch_t(const BatchArgs& A, int threads, int ctas_per_sm, cudaStream_t st) {
  if (threads > BLOCK) return FDTD_ERR_ARG;
  auto kern = k_batch<CPT, BLOCK>;
  const size_t smem = batch_smem(threads, CPT);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) {
    fdtd_host::note_cuda_error(e);
    return FDTD_ERR_CUDA;
  }
  int dev = 0, nsm = 0, occ = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem);
  if (occ < 1) return FDTD_ERR_UNSUPPORTED;
  if (ctas_per_sm > 0) occ = std::min(occ, ctas_per_sm);
  const int grid = std::max(1, std::min(nsm * occ, A.nbundles));
  kern<<<grid, threads, smem, st>>>(A);
  return fdtd_host::check_launch();
}

}  // namespace fdtd

// ======================================================================= C-ABI
extern "C" {

int fdtd1d_batch_plan(const int* ke_host, int nruns, int cells_per_thread, int block_threads, int* plan,
                      size_t plan_ints, int* plan_len) {
  using fdtd::ENTRY_INTS;
  if (!ke_host || !plan_len) return FDTD_ERR_NULL;
  if (nruns <= 0) return FDTD_ERR_SIZE;
  if (cells_per_thread <= 1 || block_threads < 32 || block_threads > 1024 || block_threads % 32) return FDTD_ERR_ARG;
  std::vector<int> team(nruns);
  for (int r = 0; r < nruns; ++r) {
    if (ke_host[r] < 4) return FDTD_ERR_SIZE;
    const int thr = (ke_host[r] + cells_per_thread - 1) / cells_per_thread;
    team[r] = ((thr + 31) / 32) * 32;
    if (team[r] > block_threads) return FDTD_ERR_SIZE;
  }
  // first-fit decreasing by team size into blocks of block_threads threads,
  // at most 15 multi-warp teams (named barriers 1..15) per block
  std::vector<int> order(nruns);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return team[a] > team[b]; });
  struct Bin {
    int used = 0, named = 0;
    std::vector<int> runs;
  };
  std::vector<Bin> bins;
  for (int r : order) {
    const bool multi = team[r] > 32;
    bool placed = false;
    for (Bin& b : bins) {
      if (b.used + team[r] <= block_threads && (!multi || b.named < 15)) {
        b.runs.push_back(r);
        b.used += team[r];
        b.named += multi;
        placed = true;
        break;
      }
    }
    if (!placed) {
      Bin b;
      b.runs.push_back(r);
      b.used = team[r];
      b.named = multi;
      bins.push_back(b);
    }
  }
  const int nb = (int)bins.size();
  // layout: [0] nbundles, [1] cells_per_thread, [2] block_threads, [3] reserved,
  //         [4 .. 4+nb] bundle start (entry index), then entries (ENTRY_INTS each)
  const size_t need = 4 + (size_t)(nb + 1) + (size_t)nruns * ENTRY_INTS;
  *plan_len = (int)need;
  if (!plan) return FDTD_OK;  // size query
  if (plan_ints < need) return FDTD_ERR_WORKSPACE;
  plan[0] = nb;
  plan[1] = cells_per_thread;
  plan[2] = block_threads;
  plan[3] = 0;
  int* bstart = plan + 4;
  int* ent = plan + 4 + nb + 1;
  int e = 0;
  for (int b = 0; b < nb; ++b) {
    bstart[b] = e;
    int off = 0, bar = 1;
    for (int r : bins[b].runs) {
      ent[e * ENTRY_INTS + 0] = r;
      ent[e * ENTRY_INTS + 1] = team[r];
      ent[e * ENTRY_INTS + 2] = off;
      ent[e * ENTRY_INTS + 3] = team[r] > 32 ? bar++ : 0;
      off += team[r];
      ++e;
    }
  }
  bstart[nb] = e;
  return FDTD_OK;
}

int fdtd1d_batch_run(const fdtd1d_batch_params* p, fdtd1d_batch_out* o, const int* plan_device, int plan_len,
                     int nbundles, int cells_per_thread, int block_threads, int ctas_per_sm, long long max_cycles,
                     fdtd_stream_t stream) {
  if (!p || !o || !plan_device) return FDTD_ERR_NULL;
  if (p->nruns <= 0 || p->nsteps < 0 || nbundles <= 0 || plan_len < 4 + nbundles + 1) return FDTD_ERR_SIZE;
  if (!p->ke || !p->layer_off || !p->probe_in || !p->probe_out || !p->src_table || !o->spec || !o->queue)
    return FDTD_ERR_NULL;
  if (p->nf < 1 || p->nf > 64 || !p->dft_cos || !p->dft_sin) return FDTD_ERR_SIZE;
  if (p->nlayers > 0 && (!p->layer_start || !p->layer_end || !p->layer_ca || !p->layer_cb)) return FDTD_ERR_NULL;
  if (p->src_k < 1) return FDTD_ERR_ARG;
  if (block_threads < 32 || block_threads > 1024 || block_threads % 32) return FDTD_ERR_ARG;
  if (p->nsteps == 0) return FDTD_OK;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(o->queue, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) {
    fdtd_host::note_cuda_error(e);
    return FDTD_ERR_CUDA;
  }
  // done[] is not cleared here: a plan may cover only some of the runs (one
  // call per tuning group), and clearing all nruns flags would erase the
  // flags an earlier group's launch set.  The caller zeroes done[] once.
  fdtd::BatchArgs A{};
  A.p = *p;
  A.o = *o;
  A.plan = plan_device;
  A.nbundles = nbundles;
  A.bstart = plan_device + 4;
  A.entries = plan_device + 4 + nbundles + 1;
  A.max_cycles = max_cycles;
  // the plan's cells per thread, two more in the kernel's lanes, and the
  // largest block each supports (register budget: 64 per thread for
  // 1024-thread blocks, 128 for 512)
  switch (cells_per_thread) {
    // (blocks of up to 512 threads get 128 registers a thread here too: at 64,
    // the 18-cell lanes spill, 5.7 us a step against 4.6 before at 1500 runs)
    case 8:
      return block_threads <= 512 ? fdtd::launch_batch_t<10, 512>(A, block_threads, ctas_per_sm, st)
                                  : fdtd::launch_batch_t<10, 1024>(A, block_threads, ctas_per_sm, st);
    case 16:
      return block_threads <= 512 ? fdtd::launch_batch_t<18, 512>(A, block_threads, ctas_per_sm, st)
                                  : fdtd::launch_batch_t<18, 1024>(A, block_threads, ctas_per_sm, st);
    case 24: return fdtd::launch_batch_t<26, 512>(A, block_threads, ctas_per_sm, st);
    case 32: return fdtd::launch_batch_t<34, 512>(A, block_threads, ctas_per_sm, st);
    case 40: return fdtd::launch_batch_t<42, 512>(A, block_threads, ctas_per_sm, st);
    default: return FDTD_ERR_ARG;
  }
}

}  // extern "C"
