// Fused 2D pass of 4 or 8 time steps for large grids: the streaming march
// (fd2d_march.cuh) in chains of warps.
//
// A pass moves 56 bytes per cell (6 evolving fields in and out, two
// materials; ez only in a call's last pass) whatever its number of steps K,
// so large grids are bound by 56/K bytes per cell-update: the K = 4 march ran
// at 85% of the copy bandwidth and could only gain by more steps per pass,
// whose state does not fit one warp's registers.  K = 8 is a chain of warps,
// each of which does LV steps and hands its rows through a ring in shared
// memory to the next; the last stores them.
//
// A block is one chain: it owns a stripe of 128 columns (4 per lane, K on each
// side recomputed by the neighbours) and marches down a segment of rows.  At
// iteration r level s of a warp (s = 0 .. LV-1) does D and E of row r-s and H
// of row r-s-1.  A row's values stay in the same registers through all levels:
// RF = LV+1 rows are in flight, row r in register set r mod RF, and the loop is
// unrolled by RF rows, so no value ever moves (the march's register shifts were
// a third of its instructions).  Updates are packed two cells to an
// instruction.  Input rows arrive by cp.async RF-1 rows ahead.  One block
// barrier per row keeps the chain in step.
//
// Two shapes, measured in Gcell-updates/s (lossy with absorbing layer /
// lossless with / lossy without; the march: 373 at 8192^2):
//   2 warps x 4 steps: 717 / 866 / 1212 at 8192^2, 521 / 651 / 1015 at 4096^2,
//     291 / 349 at 2048^2: fewer rows pass through shared memory, but a body of
//     20 levels (fetching its code costs 0.6 cycles an issue) and 2 warps per
//     scheduler;
//   4 warps x 2 steps: 643 / 742 / 995, 594 / 689 / 907, 417 / 479.
// The choice is in fd2d_chain.cu.
//
// Blocks of RF rows run in one of two forms, as in the march: interior (unit
// coefficients, nothing that the reference's loops leave out, no source) or
// general, decided on the coefficient vectors themselves.  Same per-cell
// formulas and order as the per-function kernels: bitwise equal results.
#pragma once

#include <type_traits>

#include "fd2d_internal.cuh"
#include "fd2d_pack.cuh"

namespace fdtd {

constexpr int kChainCols = 128;
// LV: time steps (levels) per warp; NC: warps in the chain
__host__ __device__ constexpr int chain_rf(int lv) { return lv + 1; }              // rows in flight in a warp's registers
__host__ __device__ constexpr int chain_lag(int lv) { return lv + chain_rf(lv); }  // rows a warp is behind the one before
// rows of the material ring: from the row being fetched (RF-1 ahead) to the last
// level of the last warp, and one for the warps' skew within an iteration
__host__ __device__ constexpr int chain_mat(int lv, int nc) { return chain_rf(lv) + chain_lag(lv) * (nc - 1) + lv + 1; }
// halo columns on each side of a stripe: whole lanes
__host__ __device__ constexpr int chain_halo(int lv, int nc) { return (lv * nc + 3) / 4 * 4; }

struct ChainArgs {
  int nx, ny;
  int pitch;  // columns from one row of every array to the next, a multiple of 4, >= ny
  FieldSet in, out;
  float* ez;  // null: not stored by this pass
  const float* naz;
  const float* nbz;
  fdtd2d_pml pml;
  int src_kind, src_i, src_j;
  const float* src_table;
  int t0;
  int* status;  // null: no Inf/NaN test
  // blocks 0 .. n_gen*n_segs_g-1: the general stripes at either edge, in shorter
  // segments; then the other stripes
  int n_stripes, n_gen_lo, n_gen_hi, n_segs, seg_first, seg_rows, n_segs_g, seg_rows_g;
  // the EXT builds' plane wave and record of ez
  int np;              // TF/SF box, 0: none
  const float* inc_e;  // as in MarchExt
  const float* inc_h;
  float* ez_rec;       // ez of each of the pass's steps, for the running DFT; null: not wanted
  size_t rec_slot;     // floats from one step's to the next
};

// floats of a block's shared memory: an input ring and a hand-over ring per
// link [RF rows][fields][128], the material ring [rows][1 or 2][128], column
// coefficients [5][128]
__host__ __device__ constexpr int chain_fields(bool lossy, bool pml) { return 3 + (lossy ? 1 : 0) + (pml ? 2 : 0); }
__host__ __device__ constexpr size_t chain_smem_bytes(int lv, int nc, bool lossy, bool pml) {
  return sizeof(float) * kChainCols *
         ((size_t)nc * chain_rf(lv) * chain_fields(lossy, pml) + chain_mat(lv, nc) * (lossy ? 2 : 1) + (pml ? 5 : 0));
}

// block -> stripe and rows; false: no work
__host__ __device__ inline bool chain_work(const ChainArgs& a, int b, int& stripe, int& i_s, int& i_e) {
  const int n_gen = a.n_gen_lo + a.n_gen_hi, n_int = a.n_stripes - n_gen, n_first = n_gen * a.n_segs_g;
  if (b < n_first) {
    const int g = b % n_gen, seg = b / n_gen;
    stripe = g < a.n_gen_lo ? g : a.n_stripes - n_gen + g;
    i_s = seg * a.seg_rows_g;
    i_e = i_s + a.seg_rows_g;
  } else {
    const int k = b - n_first;
    if (n_int == 0 || k >= n_int * a.n_segs) return false;
    stripe = a.n_gen_lo + k % n_int;
    // the first and last segments of a stripe, which hold general rows, before the others
    const int q = k / n_int, seg = q == 0 ? 0 : q == 1 ? a.n_segs - 1 : q - 1;
    i_s = seg == 0 ? 0 : a.seg_first + (seg - 1) * a.seg_rows;
    i_e = seg == a.n_segs - 1 ? a.nx : seg == 0 ? a.seg_first : i_s + a.seg_rows;
  }
  i_e = i_e < a.nx ? i_e : a.nx;
  return i_s < i_e;
}

// About `blocks` blocks over the grid: the stripes that the absorbing layer (P
// cells, 0: unknown) or the grid's edge makes general get gen_cost times as
// many segments, and the other stripes' first and last segments are shortened
// by the time of their general rows.  Returns the number of blocks.
inline long chain_layout(ChainArgs& a, int K, long blocks, int P, float gen_cost) {
  const int hb = chain_halo(K, 1), outw = kChainCols - 2 * hb;
  a.n_stripes = (a.ny + outw - 1) / outw;
  auto general = [&](int s) {
    const int lo = s * outw - hb, hi = lo + kChainCols - 1;
    return lo < std::max(P, 1) || hi > a.ny - 2 - P;
  };
  int glo = 0, ghi = 0;
  while (glo < a.n_stripes && general(glo)) ++glo;
  while (ghi < a.n_stripes - glo && general(a.n_stripes - 1 - ghi)) ++ghi;
  const int n_int = a.n_stripes - glo - ghi, n_gen = glo + ghi, mn = 4 * K;
  const double G = gen_cost >= 1.f ? gen_cost : 1.0;
  const long n_segs = std::max(1L, (long)((double)blocks / (n_int + G * n_gen)));
  const long n_segs_g = std::max(1L, (long)(G * n_segs));
  a.seg_rows_g = std::max((int)((a.nx + n_segs_g - 1) / n_segs_g), mn);
  a.n_segs_g = (a.nx + a.seg_rows_g - 1) / a.seg_rows_g;
  const int T = (int)((G - 1.0) * (P + K + 1));
  int L = a.nx, f = a.nx, ns = 1;
  if (n_segs > 1) {
    L = std::max((int)((a.nx + 2L * T + n_segs - 1) / n_segs), mn);
    f = std::min(std::max(L - T, mn), a.nx);
    ns = a.nx <= f ? 1 : 1 + (a.nx - f + L - 1) / L;
  }
  a.seg_rows = L;
  a.seg_first = f;
  a.n_segs = ns;
  a.n_gen_lo = glo;
  a.n_gen_hi = ghi;
  return (long)n_int * ns + (long)n_gen * a.n_segs_g;
}

// one pass of k steps, 4 or 8, over arrays of `pitch` columns a row (fd2d_chain.cu)
int launch_chain(const fdtd2d_params& p, int pitch, const float* naz, const float* nbz, const FieldSet& in,
                 const FieldSet& out, float* ez, int t0, int k, int* status, float gen_cost, cudaStream_t st);
// the same with the plane wave and the running DFT of `ext` (fd2d_chain_ext.cu); ez_rec: room for
// the ez of k steps, rec_slot floats each (nf > 0)
int launch_chain_ext(const fdtd2d_params& p, int pitch, const float* naz, const float* nbz, const FieldSet& in,
                     const FieldSet& out, float* ez, int t0, int k, int* status, float gen_cost, const MarchExt& ext,
                     float* ez_rec, size_t rec_slot, cudaStream_t st);

namespace {

__device__ __forceinline__ void chain_cp16(float* dst, const float* base, unsigned off, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(base + off), "r"(ok ? 16u : 0u) : "memory");
}
__device__ __forceinline__ F4 chain_lds(const float* p) { return f4(*reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void chain_sts(float* p, const F4& v) { *reinterpret_cast<float4*>(p) = to4(v); }
__device__ __forceinline__ bool chain_finite(const F4& v) {
  return isfinite(v.a.x) && isfinite(v.a.y) && isfinite(v.b.x) && isfinite(v.b.y);
}

struct ChainRow {
  F4 dz, iz, hx, hy, ihx, ihy, ez;
};

// EXT: the TF/SF box's corrections and the record of ez
template <int LV, int NC, bool LOSSY, bool PML, bool EXT>
__global__ void __launch_bounds__(32 * NC) k_chain(const __grid_constant__ ChainArgs a) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int W = kChainCols, RF = chain_rf(LV), K = LV * NC, HB = chain_halo(LV, NC);
  constexpr int NF = chain_fields(LOSSY, PML), NM = LOSSY ? 2 : 1, MT = chain_mat(LV, NC);
  constexpr int F_IZ = 3, F_IHX = 3 + (LOSSY ? 1 : 0), F_IHY = F_IHX + 1;
  extern __shared__ float4 chain_sm[];
  int stripe, i_s, i_e;
  if (!chain_work(a, blockIdx.x, stripe, i_s, i_e)) return;  // the whole block

  const int lane = threadIdx.x & 31, cw = threadIdx.x >> 5;
  const int nx = a.nx, ny = a.ny, pitch = a.pitch;
  const int j0 = stripe * (W - 2 * HB) - HB + lane * 4;
  const bool vin = j0 >= 0 && j0 + 4 <= pitch;  // pitch % 4 == 0: a lane's vector is wholly in or out of the arrays
  const bool vout = vin && lane * 4 >= HB && lane * 4 < W - HB;
  float* const sm = reinterpret_cast<float*>(chain_sm) + lane * 4;
  float* const links = sm + RF * NF * W;                      // [NC-1][RF][NF][W]
  float* const mring = links + (NC - 1) * RF * NF * W;              // [MT][NM][W], row r in slot r mod MT
  float* const cc = mring + MT * NM * W;                            // [5][W] gy2/2, gy3, fy1, fy2, fy3
  const float* const from = cw == 0 ? sm : links + (cw - 1) * RF * NF * W;  // rows into this warp
  float* const to = links + cw * RF * NF * W;                               // rows out of it (not the last warp's)

  // ---- columns
  bool col_ok = j0 >= 1 && j0 + 3 <= ny - 2;
  if (PML) {
    float v[5][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = j0 + c;
      const bool in = j >= 0 && j < ny;
      v[0][c] = 0.5f * (in ? __ldg(a.pml.gy2 + j) : 1.f);  // exact
      v[1][c] = in ? __ldg(a.pml.gy3 + j) : 1.f;
      v[2][c] = in ? __ldg(a.pml.fy1 + j) : 0.f;
      v[3][c] = in ? __ldg(a.pml.fy2 + j) : 1.f;
      v[4][c] = in ? __ldg(a.pml.fy3 + j) : 1.f;
      col_ok &= v[0][c] == 0.5f && v[1][c] == 1.f && v[2][c] == 0.f && v[3][c] == 1.f && v[4][c] == 1.f;
    }
    if (cw == 0)
#pragma unroll
      for (int k = 0; k < 5; ++k) chain_sts(cc + k * W, f4(make_float4(v[k][0], v[k][1], v[k][2], v[k][3])));
  }
  // TF/SF: the box's edge columns (D at np-1 and ny-np, hx at np-2 and ny-np)
  // make a stripe general; its edge rows np-2 and nx-np (hy) are general in
  // every stripe
  const int np = EXT ? a.np : 0;
  bool edge = false;  // any of the warp's columns is an edge column
  if (EXT && np > 0) {
#pragma unroll
    for (int c = 0; c < 4; ++c) edge |= j0 + c == np - 2 || j0 + c == np - 1 || j0 + c == ny - np;
    col_ok &= !edge;
    edge = __any_sync(kAll, edge);
  }
  const bool cint = __all_sync(kAll, col_ok);
  const bool src_here = a.src_kind != FDTD_SRC_NONE && a.src_j >= j0 - lane * 4 && a.src_j < j0 - lane * 4 + W;
  const bool col0 = j0 == 0;
  const int h_cols = ny - 1 - j0;  // of this lane's columns that H updates

  // bit l: row b+l may be touched by an interior iteration
  auto rows_ok = [&](int b) -> unsigned {
    const int row = b + lane;
    bool g = row >= 1 && row <= nx - 2;
    if (PML && g)
      g = __ldg(a.pml.gx2 + row) == 1.f && __ldg(a.pml.gx3 + row) == 1.f && __ldg(a.pml.fx1 + row) == 0.f &&
          __ldg(a.pml.fx2 + row) == 1.f && __ldg(a.pml.fx3 + row) == 1.f;
    if (src_here && row == a.src_i) g = false;
    if (EXT && np > 0 && (row == np - 2 || row == nx - np)) g = false;
    return __ballot_sync(kAll, g);
  };

  // ---- rows on their way in (first warp): fields into input ring slot `slot`,
  // materials into theirs; zeros outside the grid.  32-bit offsets (the launch
  // checks the grid's size): half the address arithmetic
  auto fetch = [&](int row, int slot, int mslot) {
    const bool ok = vin && row >= 0 && row < nx;
    const unsigned off = ok ? (unsigned)row * (unsigned)pitch + (unsigned)j0 : 0u;
    float* const f = sm + slot * NF * W;
    chain_cp16(f + 0 * W, a.in.dz, off, ok);
    chain_cp16(f + 1 * W, a.in.hx, off, ok);
    chain_cp16(f + 2 * W, a.in.hy, off, ok);
    if (LOSSY) chain_cp16(f + F_IZ * W, a.in.iz, off, ok);
    if (PML) {
      chain_cp16(f + F_IHX * W, a.in.ihx, off, ok);
      chain_cp16(f + F_IHY * W, a.in.ihy, off, ok);
    }
    float* const m = mring + mslot * NM * W;
    chain_cp16(m, a.naz, off, ok);
    if (LOSSY) chain_cp16(m + W, a.nbz, off, ok);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  const F4 zero = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  ChainRow R[RF];
#pragma unroll
  for (int k = 0; k < RF; ++k) R[k].dz = R[k].iz = R[k].hx = R[k].hy = R[k].ihx = R[k].ihy = R[k].ez = zero;
  // rows before the first that is read: no output depends on them
  for (int k = cw; k < (NC - 1) * RF * NF + MT * NM; k += NC) chain_sts(links + k * W, zero);
  __syncthreads();
  const int first = i_s - K;
  const int b0 = (first >= 0 ? first / RF : -((RF - 1 - first) / RF)) * RF;  // first row, of a block of RF
  int rb = b0 - chain_lag(LV) * cw;                     // this warp's first level's row
  int ms = ((rb - (LV - 1)) % MT + MT) % MT + LV - 1;  // material slot of row rb, in LV-1 .. MT+LV-2
  if (cw == 0) {
#pragma unroll
    for (int k = 0; k < RF - 1; ++k) fetch(rb + k, k, (ms + k) % MT);
  }
  bool fin = true;

  // ---- iteration I of the block of RF rows that starts at row rb: this warp's
  // level 0 takes row rb+I
  auto iterate = [&](auto itag, auto inttag) {
    constexpr int I = decltype(itag)::value;
    constexpr bool INT = decltype(inttag)::value;
    const int r = rb + I;
    const float* f = from + I * NF * W;
    if (cw == 0) {  // row r+RF-1 starts its way in, into row r-1's slot; row r's copies complete
      const int mf = ms + I + RF - 1;
      fetch(r + RF - 1, (I + RF - 1) % RF, mf >= MT ? mf - MT : mf);
      asm volatile("cp.async.wait_group %0;\n" ::"n"(RF - 1) : "memory");
    }
    {
      ChainRow& q = R[I];
      q.dz = chain_lds(f + 0 * W);
      q.hx = chain_lds(f + 1 * W);
      q.hy = chain_lds(f + 2 * W);
      if (LOSSY) q.iz = chain_lds(f + F_IZ * W);
      if (PML) {
        q.ihx = chain_lds(f + F_IHX * W);
        q.ihy = chain_lds(f + F_IHY * W);
      }
    }
    // every warp has taken its row: the warp before may refill the slot below
    if (NC > 1) __syncthreads();
#pragma unroll
    for (int s = 0; s < LV; ++s) {
      const int qi = (I - s + RF) % RF, pi = (I - s - 1 + RF) % RF;
      ChainRow &q = R[qi], &p = R[pi];
      const int row = r - s;
      const int t = a.t0 + LV * cw + s;  // table row of this level's time step
      // D and E on row r-s
      const float hl = __shfl_up_sync(kAll, q.hx.b.y, 1);
      const F4 d = sub4(sub4(q.hy, p.hy), q.hx);
      const F4 curl = {make_float2(__fadd_rn(d.a.x, hl), __fadd_rn(d.a.y, q.hx.a.x)),
                       make_float2(__fadd_rn(d.b.x, q.hx.a.y), __fadd_rn(d.b.y, q.hx.b.x))};
      if (INT) {
        q.dz = sub4(q.dz, mul4(-0.5f, curl));
      } else {
        F4 nd;
        const bool in = row >= 1 && row < nx;
        if (PML) {
          const float gx2 = in ? __ldg(a.pml.gx2 + row) : 1.f, gx3 = in ? __ldg(a.pml.gx3 + row) : 1.f;
          // gx2*(gy2/2) is (gx2*gy2)/2 exactly
          nd = fma4(mul4(gx3, chain_lds(cc + 1 * W)), q.dz, mul4(mul4(gx2, chain_lds(cc + 0 * W)), curl));
        } else {
          nd = sub4(q.dz, mul4(-0.5f, curl));
        }
        q.dz.a.x = in && !col0 ? nd.a.x : q.dz.a.x;
        q.dz.a.y = in ? nd.a.y : q.dz.a.y;
        q.dz.b.x = in ? nd.b.x : q.dz.b.x;
        q.dz.b.y = in ? nd.b.y : q.dz.b.y;
        if (src_here && row == a.src_i) {
          const float v = __ldg(a.src_table + t);
          auto put = [&](float& x, int j) {
            if (j == a.src_j) x = a.src_kind == FDTD_SRC_HARD ? v : __fadd_rn(x, v);
          };
          put(q.dz.a.x, j0);
          put(q.dz.a.y, j0 + 1);
          put(q.dz.b.x, j0 + 2);
          put(q.dz.b.y, j0 + 3);
        }
      }
      if constexpr (EXT && !INT) {
        if (edge && row >= np - 1 && row <= nx - np) {
          const float lo = __ldg(a.inc_h + 2 * (LV * cw + s)), hi = __ldg(a.inc_h + 2 * (LV * cw + s) + 1);
          auto put = [&](float& x, int j) {
            if (j == np - 1) x = __fmaf_rn(0.5f, lo, x);
            if (j == ny - np) x = __fmaf_rn(-0.5f, hi, x);
          };
          put(q.dz.a.x, j0);
          put(q.dz.a.y, j0 + 1);
          put(q.dz.b.x, j0 + 2);
          put(q.dz.b.y, j0 + 3);
        }
      }
      const int mi = ms + I - s;
      const float* const m = mring + (mi >= MT ? mi - MT : mi) * NM * W;
      const F4 na = chain_lds(m);
      if (LOSSY) {
        q.ez = mul4(na, sub4(q.dz, q.iz));
        q.iz = fma4(chain_lds(m + W), q.ez, q.iz);
      } else {
        q.ez = mul4(na, q.dz);
      }
      if constexpr (EXT) {
        if (a.ez_rec && vout && row >= i_s && row < i_e)
          __stcs(reinterpret_cast<float4*>(a.ez_rec + (LV * cw + s) * a.rec_slot + ((unsigned)row * (unsigned)pitch +
                                                                                   (unsigned)j0)),
                 to4(q.ez));
      }
      // H on row r-s-1
      const float er = __shfl_down_sync(kAll, p.ez.a.x, 1);
      const F4 cx = {make_float2(__fsub_rn(p.ez.a.x, p.ez.a.y), __fsub_rn(p.ez.a.y, p.ez.b.x)),
                     make_float2(__fsub_rn(p.ez.b.x, p.ez.b.y), __fsub_rn(p.ez.b.y, er))};
      const F4 cy = sub4(p.ez, q.ez);
      if (INT) {
        if (PML) {
          p.ihx = add4(p.ihx, cx);
          p.ihy = add4(p.ihy, cy);
          p.hx = sub4(p.hx, mul4(-0.5f, cx));
          p.hy = sub4(p.hy, mul4(0.5f, cy));
        } else {
          p.hx = fma4(0.5f, cx, p.hx);
          p.hy = fma4(-0.5f, cy, p.hy);
        }
      } else {
        const int pr = row - 1;
        const bool in = pr >= 0 && pr <= nx - 2;
        F4 nhx, nhy, nix, niy;
        if (PML) {
          const float fx1 = in ? __ldg(a.pml.fx1 + pr) : 0.f, fx2 = in ? __ldg(a.pml.fx2 + pr) : 1.f,
                      fx3 = in ? __ldg(a.pml.fx3 + pr) : 1.f;
          nix = add4(p.ihx, cx);
          niy = add4(p.ihy, cy);
          nhx = fma4(chain_lds(cc + 4 * W), p.hx, mul4(chain_lds(cc + 3 * W), fma4(fx1, nix, mul4(0.5f, cx))));
          // (-fx2)*z is -(fx2*z) exactly
          nhy = fma4(fx3, p.hy, mul4(-fx2, fma4(chain_lds(cc + 2 * W), niy, mul4(0.5f, cy))));
        } else {
          nhx = fma4(0.5f, cx, p.hx);
          nhy = fma4(-0.5f, cy, p.hy);
        }
        if constexpr (EXT) {
          if (np > 0) {
            const float* er0 = a.inc_e + (size_t)(LV * cw + s) * ny;
            if (edge && pr >= np - 1 && pr <= nx - np) {
              const float lo = __ldg(er0 + np - 1), hi = __ldg(er0 + ny - np);
              auto put = [&](float& x, int j) {
                if (j == np - 2) x = __fmaf_rn(0.5f, lo, x);
                if (j == ny - np) x = __fmaf_rn(-0.5f, hi, x);
              };
              put(nhx.a.x, j0);
              put(nhx.a.y, j0 + 1);
              put(nhx.b.x, j0 + 2);
              put(nhx.b.y, j0 + 3);
            }
            if ((pr == np - 2 || pr == nx - np) && vin) {
              const float wy = pr == np - 2 ? -0.5f : 0.5f;
              auto put = [&](float& x, int j) {
                if (j >= np - 1 && j <= ny - np) x = __fmaf_rn(wy, __ldg(er0 + j), x);
              };
              put(nhy.a.x, j0);
              put(nhy.a.y, j0 + 1);
              put(nhy.b.x, j0 + 2);
              put(nhy.b.y, j0 + 3);
            }
          }
        }
        // row nx-1 and column ny-1 are not updated
        const int n = in ? h_cols : 0;
        auto take = [&](F4& x, const F4& nw) {
          x.a.x = n > 0 ? nw.a.x : x.a.x;
          x.a.y = n > 1 ? nw.a.y : x.a.y;
          x.b.x = n > 2 ? nw.b.x : x.b.x;
          x.b.y = n > 3 ? nw.b.y : x.b.y;
        };
        take(p.hx, nhx);
        take(p.hy, nhy);
        if (PML) {
          take(p.ihx, nix);
          take(p.ihy, niy);
        }
      }
    }
    // ---- row r-LV is complete: to the next warp's ring, or out
    ChainRow& c = R[(I + 1) % RF];
    if (NC > 1 && cw < NC - 1) {
      float* const f = to + I * NF * W;
      chain_sts(f + 0 * W, c.dz);
      chain_sts(f + 1 * W, c.hx);
      chain_sts(f + 2 * W, c.hy);
      if (LOSSY) chain_sts(f + F_IZ * W, c.iz);
      if (PML) {
        chain_sts(f + F_IHX * W, c.ihx);
        chain_sts(f + F_IHY * W, c.ihy);
      }
    } else {
      const int row = r - LV;
      if (vout && row >= i_s && row < i_e) {
        const unsigned off = (unsigned)row * (unsigned)pitch + (unsigned)j0;
        auto st = [&](float* p, const F4& v) { __stcs(reinterpret_cast<float4*>(p + off), to4(v)); };
        st(a.out.dz, c.dz);
        st(a.out.hx, c.hx);
        st(a.out.hy, c.hy);
        if (LOSSY) st(a.out.iz, c.iz);
        if (PML) {
          st(a.out.ihx, c.ihx);
          st(a.out.ihy, c.ihy);
        }
        if (a.ez) st(a.ez, c.ez);
        if (a.status) {
          fin &= chain_finite(c.dz) && chain_finite(c.hx) && chain_finite(c.hy) && chain_finite(c.ez);
          if (LOSSY) fin &= chain_finite(c.iz);
          if (PML) fin &= chain_finite(c.ihx) && chain_finite(c.ihy);
        }
      }
    }
  };
  static_assert(RF <= 5, "block() names the iterations of a block");
  auto block = [&](auto inttag) {
    iterate(std::integral_constant<int, 0>{}, inttag);
    iterate(std::integral_constant<int, 1>{}, inttag);
    iterate(std::integral_constant<int, 2>{}, inttag);
    if constexpr (RF > 3) iterate(std::integral_constant<int, 3 % RF>{}, inttag);
    if constexpr (RF > 4) iterate(std::integral_constant<int, 4 % RF>{}, inttag);
  };

  // ---- down the segment: the last warp's last level has to complete row i_e-1
  const int n_blk = (i_e - 1 + LV - (RF - 1) + chain_lag(LV) * (NC - 1) - b0 + RF - 1) / RF + 1;
  int gb = rb - LV;  // rows gb .. gb+63 are in gm
  unsigned long long gm = cint ? rows_ok(gb) | (unsigned long long)rows_ok(gb + 32) << 32 : 0ull;
  constexpr unsigned long long kTouch = (1ull << (LV + RF)) - 1;  // rows rb-LV .. rb+RF-1 that a block touches
  for (int k = 0; k < n_blk; ++k) {
    bool interior = false;
    if (cint) {
      if (rb + RF - 1 - gb >= 64) {
        gb += 32;
        gm = gm >> 32 | (unsigned long long)rows_ok(gb + 32) << 32;
      }
      interior = ((gm >> (rb - LV - gb)) & kTouch) == kTouch;
    }
    if (interior) block(std::true_type{});
    else block(std::false_type{});
    rb += RF;
    ms = ms + RF >= MT + LV - 1 ? ms + RF - MT : ms + RF;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (a.status && __any_sync(kAll, !fin) && lane == 0) raise_status(a.status, ST_NONFINITE);
}

inline ChainArgs chain_args(const fdtd2d_params& p, int pitch, const float* naz, const float* nbz, const FieldSet& in,
                            const FieldSet& out, float* ez, int t0, int* status) {
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
  return a;
}

// waves: blocks launched over those resident.  One wave ends with its slowest
// block (SMs idle for 16% of a 2 x 4 pass at 6144^2); four short ones, the
// general stripes first, balance themselves, at the price of more recomputed
// rows: 8192^2 lossy with layer 580 -> 717 Gcell-updates/s, but 4096^2 521 -> 451.
template <int LV, int NC, bool LOSSY, bool PML, bool EXT>
int launch_t(ChainArgs a, int pml_cells, double waves, float gen_cost, cudaStream_t st) {
  auto kern = k_chain<LV, NC, LOSSY, PML, EXT>;
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

}  // namespace
}  // namespace fdtd
