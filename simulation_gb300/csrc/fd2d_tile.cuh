// 2D TM time loop with the whole grid held on the chip: grids of up to about
// 1.3 million cells.
//
// The streaming march (fd2d_march.cuh) moves every field through L2 once per
// pass; on a grid that fills the GPU with a few rows per warp its passes are
// chains of dependent rows (tm 1024^2: 10.5 us a step; 100^2: 6.2).  Here the
// grid is cut into tiles, one block each, all resident at once (a cooperative
// launch).  A block keeps its tile in registers and shared memory for the
// whole call and advances it T steps between exchanges, in which it refreshes
// a halo of T cells from its neighbours' tiles through global memory (L2).
//
// Tile: 128 columns (4 per lane) x 16*V rows (V per warp, 16 warps).  dz, hx,
// hy and (up to 4 rows a warp) ihx are in registers; the materials, iz, ihy,
// each read and written once per step by the lane that owns them, in shared
// memory.  Within
// a warp's strip the j-neighbours come by shuffle and the i-neighbours from
// the same lane's registers; a strip's first ez row and last hy row go to the
// neighbouring warps through shared memory: two block barriers per step.  The
// updates are packed two cells to an instruction (f32x2, the same rounding as
// the scalar operations).
//
// Wrong values from a tile's unrefreshed edge move in by one cell per step, so
// the halo absorbs T steps.  The exchange: every block writes the owned cells
// within T of its border, raises its flag to the exchange's number, waits for
// its neighbours' flags (bounded) and reads its halo.  Two sets of arrays
// alternate so that no block overwrites what a neighbour may still read.
//
// Same step order and per-cell formulas as the per-function kernels: results
// are bitwise equal to theirs.
//
// The adjoint's reverse sweep runs in the same frame (kTileRev): the adjoint
// fields take the fields' places, an undone step reaches one cell in each
// direction as a step does, and the two values that cross strips are the
// adjoint of cy downwards and that of the D update's curl upwards.  All it
// needs of the forward run is dz' - iz in the design box and ez at the probe,
// which a forward run in mode kTileRec leaves per step.  Mode kTileExt takes the
// TF/SF box's corrections from the incident line's table and leaves ez of every
// step for the running DFT (fd2d_dft_rec.cu).
#pragma once

#include <type_traits>

#include "fd2d_internal.cuh"
#include "fd2d_pack.cuh"
#include "fd2d_tile.h"

namespace fdtd {

struct TileArgs {
  int nx, ny;
  FieldSet in, out;   // read at the start; written at the end
  FieldSet x[2];      // exchange sets (exchange e uses x[(E - e) & 1], E the last); x[1] may be in/out
  float* ez;          // may be null (not wanted)
  const float* naz;
  const float* nbz;
  fdtd2d_pml pml;
  int src_kind, src_i, src_j;
  const float* src_table;
  int t0, nsteps;
  int* status;
  int check_finite;   // test the stored fields for Inf/NaN
  int probe_i, probe_j;
  float* probe_ez;
  unsigned* flags;    // one per block, 32 words apart, zero at the start
  TileAdj adj;        // modes kTileRec and kTileRev
  TileExt ext;        // mode kTileExt
  int T;              // steps between exchanges = halo rows
  int hc;             // halo columns on each side: T rounded up to whole lanes, or 0 with one tile per row
  int n_ti, n_tj;
  int own_r, own_c;   // owned rows and columns per tile
  int vec;            // ny % 4 == 0 and all arrays 16-byte aligned
};

// shared memory of a block, in float4: arrays of 16*V rows of 32 float4 (naz,
// [ihy], [nbz, iz]), the strips' edge rows, the column and row coefficients
// (at 5 rows a warp ihx moves there too: with it in registers the general
// steps spill)
__host__ __device__ constexpr bool tile_ihx_smem(int V, bool pml) { return pml && V >= 5; }
__host__ __device__ constexpr int tile_arrays(int V, bool lossy, bool pml, int mode) {
  return 1 + (pml ? 1 : 0) + (lossy ? 2 : 0) + (tile_ihx_smem(V, pml) ? 1 : 0) +
         (mode == kTileRev ? (lossy ? 2 : 1) : 0);  // the box's gradients
}
__host__ __device__ constexpr size_t tile_smem_bytes(int V, bool lossy, bool pml, int mode) {
  return sizeof(float4) * ((size_t)kTileWarps * V * 32 * tile_arrays(V, lossy, pml, mode) + 2 * kTileWarps * 32 + 5 * 32 +
                           3 * kTileWarps * V);
}

// defined in fd2d_tile_rec.cu
int launch_tile_rec(const TileArgs& a, int V, bool lossy, cudaStream_t st);
// defined in fd2d_tile_rev.cu
int launch_tile_rev(const TileArgs& a, int V, bool lossy, cudaStream_t st);
// defined in fd2d_tile_ext*.cu
int launch_tile_ext(const TileArgs& a, int V, bool lossy, bool pml, cudaStream_t st);
int launch_tile_ext_lossy(const TileArgs& a, int V, bool pml, cudaStream_t st);

// what a strip of a tile has to handle in its steps
constexpr int kTileInt = 0;    // unit coefficients
constexpr int kTileGen = 1;    // the absorbing layer's coefficients, column 0, column ny-1 as the last of its lane
constexpr int kTileEdge = 2;   // and row 0, row nx-1 or column ny-1 anywhere: the reference's loops leave them out
constexpr int kTilePoint = 3;  // and the source or the probe

namespace {

// one lane's four columns of row i from or to global memory, past L1 (other
// blocks write them); columns outside the grid read as 0
__device__ __forceinline__ float4 tile_ld(const float* p, size_t row, int j0, int ny, bool vec) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (vec) {
    if (j0 >= 0 && j0 + 4 <= ny) v = __ldcg(reinterpret_cast<const float4*>(p + row + j0));
  } else {
    if (j0 >= 0 && j0 < ny) v.x = __ldcg(p + row + j0);
    if (j0 + 1 >= 0 && j0 + 1 < ny) v.y = __ldcg(p + row + j0 + 1);
    if (j0 + 2 >= 0 && j0 + 2 < ny) v.z = __ldcg(p + row + j0 + 2);
    if (j0 + 3 >= 0 && j0 + 3 < ny) v.w = __ldcg(p + row + j0 + 3);
  }
  return v;
}
__device__ __forceinline__ void tile_st(float* p, size_t row, int j0, int ny, bool vec, float4 v) {
  if (vec) {
    if (j0 >= 0 && j0 + 4 <= ny) __stcg(reinterpret_cast<float4*>(p + row + j0), v);
  } else {
    if (j0 >= 0 && j0 < ny) __stcg(p + row + j0, v.x);
    if (j0 + 1 >= 0 && j0 + 1 < ny) __stcg(p + row + j0 + 1, v.y);
    if (j0 + 2 >= 0 && j0 + 2 < ny) __stcg(p + row + j0 + 2, v.z);
    if (j0 + 3 >= 0 && j0 + 3 < ny) __stcg(p + row + j0 + 3, v.w);
  }
}
// v = p[off .. off+3] where ok, past L1, else v as it is: predicated, so that
// many of them can be in flight, and in pairs, which is how the registers hold
// the cells (a 16-byte read into four others is waited for at once, to move
// them: 7 us an exchange of 1024^2 instead of 4)
__device__ __forceinline__ void tile_ld_if(const float* p, size_t off, bool ok, F4& v) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n @q ld.global.cg.v2.f32 {%0, %1}, [%4];\n"
      " @q ld.global.cg.v2.f32 {%2, %3}, [%4+8];\n}"
      : "+f"(v.a.x), "+f"(v.a.y), "+f"(v.b.x), "+f"(v.b.y)
      : "l"(p + off), "r"((int)ok)
      : "memory");
}
// the same into shared memory, without registers; waited for by tile_cp_wait
__device__ __forceinline__ void tile_cp_if(const float* p, size_t off, bool ok, float4* dst) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n @q cp.async.cg.shared.global [%0], [%1], 16;\n}" ::"r"(
          (unsigned)__cvta_generic_to_shared(dst)),
      "l"(p + off), "r"((int)ok)
      : "memory");
}
__device__ __forceinline__ void tile_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ bool tile_finite(const float4& v) {
  return isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w);
}

template <int V, bool LOSSY, bool PML, int MODE>
__global__ void __launch_bounds__(kTileWarps * 32, 1) k_tile(const TileArgs a) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int W = kTileWarps, R = W * V;
  constexpr bool IHXS = tile_ihx_smem(V, PML);
  constexpr int NARR = tile_arrays(V, LOSSY, PML, MODE);
  constexpr bool REC = MODE == kTileRec, REV = MODE == kTileRev, EXT = MODE == kTileExt;
  constexpr int A_NAZ = 0, A_IHY = 1, A_NBZ = PML ? 2 : 1, A_IZ = A_NBZ + 1, A_IHX = A_NBZ + (LOSSY ? 2 : 0),
                A_G = A_IHX + (IHXS ? 1 : 0), A_GB = A_G + 1;
  extern __shared__ float4 tsm[];
  __shared__ int s_dead;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float4* const xe = tsm + (size_t)NARR * R * 32;  // [W][32] first ez row of each strip
  float4* const xh = xe + W * 32;                  // [W][32] last hy row of each strip
  float4* const cc = xh + W * 32;                  // [5][32] gy2/2, gy3, fy1, fy2, fy3 of the columns
  float4* const rc = cc + 5 * 32;                  // [R][3] gx2, gx3 | fx1, -fx2 | fx3 of the rows, each twice (a pair)
  auto at = [&](int arr, int r) -> float4& { return tsm[((size_t)arr * R + w * V + r) * 32 + lane]; };

  const int nx = a.nx, ny = a.ny, T = a.T;
  const bool vec = a.vec != 0;
  const int ti = blockIdx.x / a.n_tj, tj = blockIdx.x % a.n_tj;
  const int i0 = ti * a.own_r - T + w * V;              // this strip's first row
  const int j0 = tj * a.own_c - a.hc + lane * 4;        // this lane's first column
  const int oi0 = ti * a.own_r, oi1 = min(oi0 + a.own_r, nx);  // owned rows
  const bool own_c = lane * 4 >= a.hc && lane * 4 < a.hc + a.own_c;  // owned columns (whole lanes)
  if (threadIdx.x == 0) s_dead = 0;

  // ---- load the tile
  F4 dz[V], hx[V], hy[V];
  [[maybe_unused]] F4 ihx_r[PML && !IHXS ? V : 1] = {};
  auto ihx_get = [&](int r) -> F4 {
    if constexpr (!PML) return F4{};
    else if constexpr (IHXS) return f4(at(A_IHX, r));
    else return ihx_r[r];
  };
  auto ihx_set = [&](int r, const F4& v) {
    if constexpr (PML && IHXS) at(A_IHX, r) = to4(v);
    else if constexpr (PML) ihx_r[r] = v;
  };
#pragma unroll
  for (int r = 0; r < V; ++r) {
    const int i = i0 + r;
    const bool in = i >= 0 && i < nx;
    const size_t row = in ? (size_t)i * ny : 0;
    auto ld = [&](const float* p) { return in ? tile_ld(p, row, j0, ny, vec) : make_float4(0.f, 0.f, 0.f, 0.f); };
    dz[r] = f4(ld(a.in.dz));
    hx[r] = f4(ld(a.in.hx));
    hy[r] = f4(ld(a.in.hy));
    at(A_NAZ, r) = ld(a.naz);
    if (PML) {
      ihx_set(r, f4(ld(a.in.ihx)));
      at(A_IHY, r) = ld(a.in.ihy);
    }
    if (LOSSY) {
      at(A_NBZ, r) = ld(a.nbz);
      at(A_IZ, r) = ld(a.in.iz);
    }
  }
  // ---- coefficients, and whether the strip's are all the unit ones
  bool col_ok = true, row_ok = true;
  if (PML) {
    float g2[4], g3[4], f1[4], f2[4], f3[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = j0 + c;
      const bool in = j >= 0 && j < ny;
      g2[c] = in ? __ldg(a.pml.gy2 + j) : 1.f;
      g3[c] = in ? __ldg(a.pml.gy3 + j) : 1.f;
      f1[c] = in ? __ldg(a.pml.fy1 + j) : 0.f;
      f2[c] = in ? __ldg(a.pml.fy2 + j) : 1.f;
      f3[c] = in ? __ldg(a.pml.fy3 + j) : 1.f;
      col_ok &= g2[c] == 1.f && g3[c] == 1.f && f1[c] == 0.f && f2[c] == 1.f && f3[c] == 1.f;
    }
    if (w == 0) {
      cc[0 * 32 + lane] = make_float4(0.5f * g2[0], 0.5f * g2[1], 0.5f * g2[2], 0.5f * g2[3]);  // exact
      cc[1 * 32 + lane] = make_float4(g3[0], g3[1], g3[2], g3[3]);
      cc[2 * 32 + lane] = make_float4(f1[0], f1[1], f1[2], f1[3]);
      cc[3 * 32 + lane] = make_float4(f2[0], f2[1], f2[2], f2[3]);
      cc[4 * 32 + lane] = make_float4(f3[0], f3[1], f3[2], f3[3]);
    }
  }
  if (lane < V) {
    const int i = i0 + lane;
    const bool in = i >= 0 && i < nx;
    if (PML) {
      const float4 k = in ? make_float4(__ldg(a.pml.gx2 + i), __ldg(a.pml.gx3 + i), __ldg(a.pml.fx1 + i),
                                        __ldg(a.pml.fx2 + i))
                          : make_float4(1.f, 1.f, 0.f, 1.f);
      const float k3 = in ? __ldg(a.pml.fx3 + i) : 1.f;
      rc[(w * V + lane) * 3] = make_float4(k.x, k.x, k.y, k.y);
      rc[(w * V + lane) * 3 + 1] = make_float4(k.z, k.z, -k.w, -k.w);
      rc[(w * V + lane) * 3 + 2] = make_float4(k3, k3, 0.f, 0.f);
      row_ok &= k.x == 1.f && k.y == 1.f && k.z == 0.f && k.w == 1.f && k3 == 1.f;
    }
  }
  auto in_strip = [&](int i, int j) { return i >= i0 && i < i0 + V && j >= j0 - 4 * lane && j < j0 - 4 * lane + kTileCols; };
  const bool src_here = a.src_kind != FDTD_SRC_NONE && in_strip(a.src_i, a.src_j);
  const bool probe_here = a.probe_ez != nullptr && in_strip(a.probe_i, a.probe_j);
  // what a strip's steps have to handle, the same in the whole warp (j0 is a multiple of 4)
  const bool last_col = j0 + 4 == ny;
  const bool masks = i0 <= 0 || i0 + V - 1 >= nx - 1 || __any_sync(kAll, j0 < ny && j0 + 4 > ny);
  // TF/SF box: strips with an edge column (D at np-1 and ny-np, hx at np-2 and
  // ny-np) or an edge row (hy at np-2 and nx-np)
  const int np = EXT ? a.ext.np : 0;
  bool edge_c = false;
  if (EXT && np > 0) {
#pragma unroll
    for (int c = 0; c < 4; ++c) edge_c |= j0 + c == np - 2 || j0 + c == np - 1 || j0 + c == ny - np;
    edge_c = __any_sync(kAll, edge_c);
  }
  const bool edge_r = np > 0 && ((np - 2 >= i0 && np - 2 < i0 + V) || (nx - np >= i0 && nx - np < i0 + V));
  const bool unit = __all_sync(kAll, col_ok && row_ok && j0 != 0 && !last_col) && !edge_c && !edge_r;
  const int kind = src_here || probe_here ? kTilePoint : masks ? kTileEdge : unit ? kTileInt : kTileGen;
  // owned cells of the design box, in whole lanes
  [[maybe_unused]] const int bc = j0 - a.adj.jb;
  [[maybe_unused]] const bool box_c = (REC || REV) && own_c && bc >= 0 && bc < a.adj.njp;
  [[maybe_unused]] auto box_row = [&](int i) {
    return i >= oi0 && i < oi1 && i >= a.adj.box.i0 && i < a.adj.box.i0 + a.adj.box.ni;
  };
  [[maybe_unused]] auto rec_at = [&](int s, int i) {  // dz' - iz of the lane's cells at the s-th step of the run
    return reinterpret_cast<float4*>(a.adj.rec + ((size_t)s * a.adj.box.ni + (i - a.adj.box.i0)) * a.adj.njp + bc);
  };
  if constexpr (REV) {
#pragma unroll
    for (int r = 0; r < V; ++r) {
      const int i = i0 + r;
      auto grad = [&](const float* g) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (g && box_c && box_row(i))
          for (int c = 0; c < 4; ++c) {
            const int bj = j0 + c - a.adj.box.j0;
            if (bj >= 0 && bj < a.adj.box.nj) v[c] = g[(size_t)(i - a.adj.box.i0) * a.adj.box.nj + bj];
          }
        return make_float4(v[0], v[1], v[2], v[3]);
      };
      at(A_G, r) = grad(a.adj.grad_naz);
      if (LOSSY) at(A_GB, r) = grad(a.adj.grad_nbz);
    }
    __syncthreads();  // the columns' and rows' coefficients
  }
  // how many of the lane's columns of row i have an H update (rows 0 .. nx-2, columns 0 .. ny-2)
  [[maybe_unused]] auto h_cols = [&](int i) { return i >= 0 && i <= nx - 2 ? ny - 1 - j0 : 0; };
  [[maybe_unused]] auto first = [&](const F4& v, const F4& o, int n) {  // the first n of v, then o's
    return F4{make_float2(n <= 0 ? o.a.x : v.a.x, n <= 1 ? o.a.y : v.a.y),
              make_float2(n <= 2 ? o.b.x : v.b.x, n <= 3 ? o.b.y : v.b.y)};
  };
  // REV: the adjoint of cy on strip row r, from the adjoints of hy and ihy
  [[maybe_unused]] auto lam_cy = [&](int r) {
    const float4 k = rc[(w * V + r) * 3 + 1];
    const float2 nfx2 = make_float2(k.z, k.w);
    const F4 t = fma4(mul4(nfx2, f4(cc[2 * 32 + lane])), hy[r], f4(at(A_IHY, r)));
    return first(fma4(make_float2(0.5f * k.z, 0.5f * k.w), hy[r], t), F4{}, h_cols(i0 + r));
  };
  // the row that the strip below needs: hy, or the adjoint of cy
  auto publish = [&] {
    if constexpr (REV) xh[w * 32 + lane] = to4(lam_cy(V - 1));
    else xh[w * 32 + lane] = to4(hy[V - 1]);
  };
  publish();
  __syncthreads();

  // ---- one step undone, step t0-s
  [[maybe_unused]] auto unstep = [&](auto kind_tag, const int s) {
    constexpr int KIND = decltype(kind_tag)::value;
    constexpr bool INT = KIND == kTileInt, MASK = KIND >= kTileEdge, POINT = KIND == kTilePoint;
    F4 gy2, gy3, fy1, fy2, fy3;
    if (!INT) {
      gy2 = f4(cc[0 * 32 + lane]);
      gy3 = f4(cc[1 * 32 + lane]);
      fy1 = f4(cc[2 * 32 + lane]);
      fy2 = f4(cc[3 * 32 + lane]);
      fy3 = f4(cc[4 * 32 + lane]);
    }
    F4 cup = f4(w > 0 ? xh[(w - 1) * 32 + lane] : make_float4(0.f, 0.f, 0.f, 0.f));
#pragma unroll
    for (int r = 0; r < V; ++r) {
      const int i = i0 + r;
      const bool boxed = box_c && box_row(i);
      float4 diff = make_float4(0.f, 0.f, 0.f, 0.f);
      if (boxed) diff = __ldg(rec_at(a.nsteps - 1 - s, i));
      // adjoints of cx and cy; the H update undone but for the D adjoint's terms
      F4 cx, cy;
      if (INT) {
        cx = fma4(0.5f, hx[r], ihx_get(r));
        cy = fma4(-0.5f, hy[r], f4(at(A_IHY, r)));
      } else {
        const float4 k = rc[(w * V + r) * 3 + 1];
        const float2 fx3 = *reinterpret_cast<const float2*>(&rc[(w * V + r) * 3 + 2]);
        const float2 fx1 = make_float2(k.x, k.y), nfx2 = make_float2(k.z, k.w);
        const F4 ix = ihx_get(r), iy = f4(at(A_IHY, r));
        F4 nix = fma4(mul4(fx1, fy2), hx[r], ix), niy = fma4(mul4(nfx2, fy1), hy[r], iy);
        cx = fma4(mul4(0.5f, fy2), hx[r], nix);
        cy = fma4(make_float2(0.5f * k.z, 0.5f * k.w), hy[r], niy);
        F4 nhx = mul4(fy3, hx[r]), nhy = mul4(fx3, hy[r]);
        if (MASK) {
          const int n = h_cols(i);
          cx = first(cx, F4{}, n);
          cy = first(cy, F4{}, n);
          nix = first(nix, ix, n);
          niy = first(niy, iy, n);
          nhx = first(nhx, hx[r], n);
          nhy = first(nhy, hy[r], n);
        } else {  // column ny-1, the last of its lane
          cx.b.y = last_col ? 0.f : cx.b.y;
          cy.b.y = last_col ? 0.f : cy.b.y;
          nix.b.y = last_col ? ix.b.y : nix.b.y;
          niy.b.y = last_col ? iy.b.y : niy.b.y;
          nhx.b.y = last_col ? hx[r].b.y : nhx.b.y;
          nhy.b.y = last_col ? hy[r].b.y : nhy.b.y;
        }
        ihx_set(r, nix);
        at(A_IHY, r) = to4(niy);
        hx[r] = nhx;
        hy[r] = nhy;
      }
      // adjoint of ez, then the E update undone
      float cl = __shfl_up_sync(kAll, cx.b.y, 1);
      cl = lane == 0 ? 0.f : cl;  // column 0, or a halo's edge
      F4 lez = {make_float2(__fsub_rn(cx.a.x, cl), __fsub_rn(cx.a.y, cx.a.x)),
                make_float2(__fsub_rn(cx.b.x, cx.a.y), __fsub_rn(cx.b.y, cx.b.x))};
      lez = sub4(add4(lez, cy), cup);
      cup = cy;
      if (POINT && probe_here && i == a.probe_i) {
        const float e = __ldg(a.probe_ez + a.t0 - 1 - s);
        auto seed = [&](float& x, int j) {
          if (j == a.probe_j) x = __fmaf_rn(a.adj.probe_w, e, x);
        };
        seed(lez.a.x, j0);
        seed(lez.a.y, j0 + 1);
        seed(lez.b.x, j0 + 2);
        seed(lez.b.y, j0 + 3);
      }
      const F4 na = f4(at(A_NAZ, r));
      if (LOSSY) {
        const F4 liz = f4(at(A_IZ, r));
        lez = fma4(f4(at(A_NBZ, r)), liz, lez);
        const F4 nna = {make_float2(-na.a.x, -na.a.y), make_float2(-na.b.x, -na.b.y)};
        at(A_IZ, r) = to4(fma4(nna, lez, liz));
        if (boxed) at(A_GB, r) = to4(fma4(liz, mul4(na, f4(diff)), f4(at(A_GB, r))));
      }
      if (boxed) at(A_G, r) = to4(fma4(lez, f4(diff), f4(at(A_G, r))));
      const F4 T = fma4(na, lez, dz[r]);
      // the D update undone; dg is the adjoint of its curl, ndg = -dg (the sums below as in sub4's comment)
      F4 dg, ndg;
      if (INT) {
        dz[r] = T;
        dg = mul4(0.5f, T);
        ndg = mul4(-0.5f, T);
      } else {
        const float4 k = rc[(w * V + r) * 3];
        F4 nd = mul4(mul4(make_float2(k.z, k.w), gy3), T);
        dg = mul4(mul4(make_float2(k.x, k.y), gy2), T);
        ndg = mul4(mul4(make_float2(-k.x, -k.y), gy2), T);
        if (j0 == 0) {  // column 0 has no D update
          nd.a.x = T.a.x;
          dg.a.x = ndg.a.x = 0.f;
        }
        if (MASK && i < 1) {  // nor has row 0
          nd = T;
          dg = ndg = F4{};
        }
        if (POINT && src_here && a.src_kind == FDTD_SRC_HARD && i == a.src_i) {
          auto cut = [&](float& x, float& y, float& z, int j) {
            if (j == a.src_j) x = y = z = 0.f;
          };
          cut(nd.a.x, dg.a.x, ndg.a.x, j0);
          cut(nd.a.y, dg.a.y, ndg.a.y, j0 + 1);
          cut(nd.b.x, dg.b.x, ndg.b.x, j0 + 2);
          cut(nd.b.y, dg.b.y, ndg.b.y, j0 + 3);
        }
        dz[r] = nd;
      }
      float nr = __shfl_down_sync(kAll, ndg.a.x, 1);
      nr = lane == 31 ? 0.f : nr;
      const F4 nj = {make_float2(ndg.a.y, ndg.b.x), make_float2(ndg.b.y, nr)};
      hx[r] = sub4(sub4(hx[r], dg), nj);
      hy[r] = sub4(hy[r], ndg);
      if (r == 0) xe[w * 32 + lane] = to4(dg);
      else hy[r - 1] = sub4(hy[r - 1], dg);
    }
    __syncthreads();
    hy[V - 1] = sub4(hy[V - 1], f4(w < W - 1 ? xe[(w + 1) * 32 + lane] : make_float4(0.f, 0.f, 0.f, 0.f)));
    if (INT) xh[w * 32 + lane] = to4(fma4(-0.5f, hy[V - 1], f4(at(A_IHY, V - 1))));
    else publish();
    __syncthreads();
  };

  // ---- one time step, t0+s+1; LAST stores ez
  [[maybe_unused]] auto step = [&](auto kind_tag, const int s, const bool last) {
    constexpr int KIND = decltype(kind_tag)::value;
    constexpr bool INT = KIND == kTileInt, MASK = KIND >= kTileEdge, POINT = KIND == kTilePoint;
    // the columns' coefficients for this step (read per row they bound it: shared memory)
    F4 gy2, gy3, fy1, fy2, fy3;
    if (PML && !INT) {
      gy2 = f4(cc[0 * 32 + lane]);
      gy3 = f4(cc[1 * 32 + lane]);
      fy1 = f4(cc[2 * 32 + lane]);
      fy2 = f4(cc[3 * 32 + lane]);
      fy3 = f4(cc[4 * 32 + lane]);
    }
    [[maybe_unused]] float hxi_lo = 0.f, hxi_hi = 0.f, ezi_lo = 0.f, ezi_hi = 0.f;
    if constexpr (EXT && !INT) {
      if (edge_c) {
        hxi_lo = __ldg(a.ext.inc_h + 2 * s);
        hxi_hi = __ldg(a.ext.inc_h + 2 * s + 1);
        ezi_lo = __ldg(a.ext.inc_e + (size_t)s * ny + np - 1);
        ezi_hi = __ldg(a.ext.inc_e + (size_t)s * ny + ny - np);
      }
    }
    // x of the lane's columns jl and jh: += lo/2, -= hi/2
    [[maybe_unused]] auto edges = [&](F4& x, int jl, float lo, int jh, float hi) {
      auto put = [&](float& y, int j) {
        if (j == jl) y = __fmaf_rn(0.5f, lo, y);
        if (j == jh) y = __fmaf_rn(-0.5f, hi, y);
      };
      put(x.a.x, j0);
      put(x.a.y, j0 + 1);
      put(x.b.x, j0 + 2);
      put(x.b.y, j0 + 3);
    };
    // H on strip row r, ez of rows r and r+1
    auto h_row = [&](int r, const F4& e, const F4& en) {
      const int i = i0 + r;
      const float er = __shfl_down_sync(kAll, e.a.x, 1);
      const F4 cx = {make_float2(__fsub_rn(e.a.x, e.a.y), __fsub_rn(e.a.y, e.b.x)),
                     make_float2(__fsub_rn(e.b.x, e.b.y), __fsub_rn(e.b.y, er))};
      const F4 cy = sub4(e, en);
      if (INT) {
        if (PML) {
          ihx_set(r, add4(ihx_get(r), cx));
          at(A_IHY, r) = to4(add4(f4(at(A_IHY, r)), cy));
          hx[r] = sub4(hx[r], mul4(-0.5f, cx));
          hy[r] = sub4(hy[r], mul4(0.5f, cy));
        } else {
          hx[r] = fma4(0.5f, cx, hx[r]);
          hy[r] = fma4(-0.5f, cy, hy[r]);
        }
      } else {
        F4 nhx, nhy, nix, niy, ix, iy;
        if (PML) {
          const float4 k = rc[(w * V + r) * 3 + 1];
          const float2 fx3 = *reinterpret_cast<const float2*>(&rc[(w * V + r) * 3 + 2]);
          const float2 fx1 = make_float2(k.x, k.y), nfx2 = make_float2(k.z, k.w);
          ix = ihx_get(r);
          iy = f4(at(A_IHY, r));
          nix = add4(ix, cx);
          niy = add4(iy, cy);
          nhx = fma4(fy3, hx[r], mul4(fy2, fma4(fx1, nix, mul4(0.5f, cx))));
          // (-fx2)*z is -(fx2*z) exactly
          nhy = fma4(fx3, hy[r], mul4(nfx2, fma4(fy1, niy, mul4(0.5f, cy))));
        } else {
          nhx = fma4(0.5f, cx, hx[r]);
          nhy = fma4(-0.5f, cy, hy[r]);
        }
        if constexpr (EXT) {
          if (edge_c && i >= np - 1 && i <= nx - np) edges(nhx, np - 2, ezi_lo, ny - np, ezi_hi);
          if (edge_r && (i == np - 2 || i == nx - np)) {
            const float wy = i == np - 2 ? -0.5f : 0.5f;
            auto put = [&](float& y, int j) {
              if (j >= np - 1 && j <= ny - np) y = __fmaf_rn(wy, __ldg(a.ext.inc_e + (size_t)s * ny + j), y);
            };
            put(nhy.a.x, j0);
            put(nhy.a.y, j0 + 1);
            put(nhy.b.x, j0 + 2);
            put(nhy.b.y, j0 + 3);
          }
        }
        if (!MASK) {  // column ny-1, the last of its lane (ny % 4 == 0), is not updated
          nhx.b.y = last_col ? hx[r].b.y : nhx.b.y;
          nhy.b.y = last_col ? hy[r].b.y : nhy.b.y;
          if (PML) {
            nix.b.y = last_col ? ix.b.y : nix.b.y;
            niy.b.y = last_col ? iy.b.y : niy.b.y;
          }
        }
        if (MASK) {  // row nx-1 and column ny-1 are not updated (selects: no branch between the rows' chains)
          const int n = i >= 0 && i <= nx - 2 ? ny - 1 - j0 : 0;
          auto keep = [&](F4& nw, const F4& old) {
            nw.a.x = n <= 0 ? old.a.x : nw.a.x;
            nw.a.y = n <= 1 ? old.a.y : nw.a.y;
            nw.b.x = n <= 2 ? old.b.x : nw.b.x;
            nw.b.y = n <= 3 ? old.b.y : nw.b.y;
          };
          keep(nhx, hx[r]);
          keep(nhy, hy[r]);
          if (PML) {
            keep(nix, ix);
            keep(niy, iy);
          }
        }
        hx[r] = nhx;
        hy[r] = nhy;
        if (PML) {
          ihx_set(r, nix);
          at(A_IHY, r) = to4(niy);
        }
      }
    };
    F4 hup = f4(w > 0 ? xh[(w - 1) * 32 + lane] : make_float4(0.f, 0.f, 0.f, 0.f));
    F4 ep;
#pragma unroll
    for (int r = 0; r < V; ++r) {
      const int i = i0 + r;
      const float hl = __shfl_up_sync(kAll, hx[r].b.y, 1);
      const F4 d = sub4(sub4(hy[r], hup), hx[r]);
      const F4 curl = {make_float2(__fadd_rn(d.a.x, hl), __fadd_rn(d.a.y, hx[r].a.x)),
                       make_float2(__fadd_rn(d.b.x, hx[r].a.y), __fadd_rn(d.b.y, hx[r].b.x))};
      hup = hy[r];
      if (INT) {
        dz[r] = sub4(dz[r], mul4(-0.5f, curl));
      } else {
        F4 nd;
        if (PML) {
          const float4 k = rc[(w * V + r) * 3];
          // gx2*(gy2/2) is (gx2*gy2)/2 exactly
          nd = fma4(mul4(make_float2(k.z, k.w), gy3), dz[r], mul4(mul4(make_float2(k.x, k.y), gy2), curl));
        } else {
          nd = sub4(dz[r], mul4(-0.5f, curl));
        }
        nd.a.x = j0 != 0 ? nd.a.x : dz[r].a.x;  // column 0 is not updated
        if (MASK) {                            // nor is row 0
          const bool row = i >= 1 && i < nx;
          nd.a.x = row ? nd.a.x : dz[r].a.x;
          nd.a.y = row ? nd.a.y : dz[r].a.y;
          nd.b.x = row ? nd.b.x : dz[r].b.x;
          nd.b.y = row ? nd.b.y : dz[r].b.y;
        }
        dz[r] = nd;
        if (POINT && src_here && i == a.src_i) {
          const float v = __ldg(a.src_table + a.t0 + s);
          auto put = [&](float& x, int j) {
            if (j == a.src_j) x = a.src_kind == FDTD_SRC_HARD ? v : __fadd_rn(x, v);
          };
          put(dz[r].a.x, j0);
          put(dz[r].a.y, j0 + 1);
          put(dz[r].b.x, j0 + 2);
          put(dz[r].b.y, j0 + 3);
        }
      }
      if constexpr (EXT && !INT) {
        if (edge_c && i >= np - 1 && i <= nx - np) edges(dz[r], np - 1, hxi_lo, ny - np, hxi_hi);
      }
      F4 e;
      const F4 na = f4(at(A_NAZ, r));
      if (LOSSY) {
        const F4 iz = f4(at(A_IZ, r));
        const F4 diff = sub4(dz[r], iz);
        if (REC && box_c && box_row(i)) __stcg(rec_at(s, i), to4(diff));
        e = mul4(na, diff);
        at(A_IZ, r) = to4(fma4(f4(at(A_NBZ, r)), e, iz));
      } else {
        if (REC && box_c && box_row(i)) __stcg(rec_at(s, i), to4(dz[r]));
        e = mul4(na, dz[r]);
      }
      if (POINT && probe_here && i == a.probe_i && own_c && i >= oi0 && i < oi1) {
        auto rec = [&](float x, int j) {
          if (j == a.probe_j) a.probe_ez[a.t0 + s] = x;
        };
        rec(e.a.x, j0);
        rec(e.a.y, j0 + 1);
        rec(e.b.x, j0 + 2);
        rec(e.b.y, j0 + 3);
      }
      if constexpr (EXT) {
        if (a.ext.ez_rec && own_c && i >= oi0 && i < oi1)
          tile_st(a.ext.ez_rec + s * a.ext.rec_slot, (size_t)i * ny, j0, ny, vec, to4(e));
      }
      if (last && a.ez && own_c && i >= oi0 && i < oi1) {
        const float4 v = to4(e);
        tile_st(a.ez, (size_t)i * ny, j0, ny, vec, v);
      }
      if (r == 0) xe[w * 32 + lane] = to4(e);
      else h_row(r - 1, ep, e);
      ep = e;
    }
    __syncthreads();
    h_row(V - 1, ep, f4(w < W - 1 ? xe[(w + 1) * 32 + lane] : make_float4(0.f, 0.f, 0.f, 0.f)));
    xh[w * 32 + lane] = to4(hy[V - 1]);
    __syncthreads();
  };

  // ---- exchange number e: owned border cells out, neighbours' flags, halo in
  auto raise_and_wait = [&](unsigned e) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(a.flags + (size_t)blockIdx.x * 32), "r"(e) : "memory");
    if (threadIdx.x < 9 && s_dead == 0) {
      const int ni = ti + (int)threadIdx.x / 3 - 1, nj = tj + (int)threadIdx.x % 3 - 1;
      if (ni >= 0 && ni < a.n_ti && nj >= 0 && nj < a.n_tj) {
        const unsigned* f = a.flags + (size_t)(ni * a.n_tj + nj) * 32;
        const long long c0 = clock64();
        for (;;) {
          unsigned v;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
          if (v >= e) break;
          if (clock64() - c0 > 4000000000LL) {  // about 2 s: report, and wait for nothing any more
            raise_status(a.status, ST_TIMEOUT);
            s_dead = 1;
            break;
          }
        }
      }
    }
    __syncthreads();
  };
  auto exchange = [&](const FieldSet& x, unsigned e) {
    const int oj0 = tj * a.own_c, oj1 = min(oj0 + a.own_c, ny);
#pragma unroll
    for (int r = 0; r < V; ++r) {
      const int i = i0 + r;
      if (i >= oi0 && i < oi1 && own_c) {
        const bool band = i < oi0 + T || i >= oi1 - T || j0 < oj0 + a.hc || j0 + 3 >= oj1 - a.hc;
        if (band) {
          const size_t row = (size_t)i * ny;
          tile_st(x.dz, row, j0, ny, vec, to4(dz[r]));
          tile_st(x.hx, row, j0, ny, vec, to4(hx[r]));
          tile_st(x.hy, row, j0, ny, vec, to4(hy[r]));
          if (PML) {
            tile_st(x.ihx, row, j0, ny, vec, to4(ihx_get(r)));
            tile_st(x.ihy, row, j0, ny, vec, at(A_IHY, r));
          }
          if (LOSSY) tile_st(x.iz, row, j0, ny, vec, at(A_IZ, r));
        }
      }
    }
    raise_and_wait(e);
    // every row's and field's read is on its way before the first is waited for
    auto halo = [&](int r) {
      const int i = i0 + r;
      return i >= 0 && i < nx && j0 >= 0 && j0 < ny && !(own_c && i >= oi0 && i < oi1);
    };
    if (vec) {
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const bool h = halo(r);
        const size_t off = h ? (size_t)(i0 + r) * ny + j0 : 0;
        if (PML) tile_cp_if(x.ihy, off, h, &at(A_IHY, r));
        if (LOSSY) tile_cp_if(x.iz, off, h, &at(A_IZ, r));
        tile_ld_if(x.dz, off, h, dz[r]);
        tile_ld_if(x.hx, off, h, hx[r]);
        tile_ld_if(x.hy, off, h, hy[r]);
        if (PML && IHXS) tile_cp_if(x.ihx, off, h, &at(A_IHX, r));
        if constexpr (PML && !IHXS) tile_ld_if(x.ihx, off, h, ihx_r[r]);
      }
      if (PML || LOSSY) tile_cp_wait();
    } else {
#pragma unroll
      for (int r = 0; r < V; ++r)
        if (halo(r)) {
          const size_t row = (size_t)(i0 + r) * ny;
          dz[r] = f4(tile_ld(x.dz, row, j0, ny, false));
          hx[r] = f4(tile_ld(x.hx, row, j0, ny, false));
          hy[r] = f4(tile_ld(x.hy, row, j0, ny, false));
          if (PML) {
            ihx_set(r, f4(tile_ld(x.ihx, row, j0, ny, false)));
            at(A_IHY, r) = tile_ld(x.ihy, row, j0, ny, false);
          }
          if (LOSSY) at(A_IZ, r) = tile_ld(x.iz, row, j0, ny, false);
        }
    }
    publish();
    __syncthreads();
  };

  // flag 1: this block has read the input arrays, so its neighbours may write
  // into them (they can be an exchange set and the output)
  const int n_ex = (a.nsteps + T - 1) / T - 1;
  if (a.n_ti * a.n_tj > 1) raise_and_wait(1);
  for (int s = 0, e = 0; s < a.nsteps;) {
    const int m = min(T, a.nsteps - s);
    auto run = [&](auto kind_tag) {
      for (int q = 0; q < m; ++q) {
        if constexpr (REV) unstep(kind_tag, s + q);
        else step(kind_tag, s + q, s + q + 1 == a.nsteps);
      }
    };
    if (kind == kTileInt) run(std::integral_constant<int, kTileInt>{});
    else if (kind == kTileGen) run(std::integral_constant<int, kTileGen>{});
    else if (kind == kTileEdge) run(std::integral_constant<int, kTileEdge>{});
    else run(std::integral_constant<int, kTilePoint>{});
    s += m;
    if (s < a.nsteps) {
      ++e;
      exchange((n_ex - e) & 1 ? a.x[1] : a.x[0], (unsigned)e + 1);
    }
  }

  // ---- results
  bool fin = true;
#pragma unroll
  for (int r = 0; r < V; ++r) {
    const int i = i0 + r;
    if (i >= oi0 && i < oi1 && own_c) {
      const size_t row = (size_t)i * ny;
      auto test = [&](const float4& v) {
        if (a.check_finite) {
          const bool f = (j0 + 3 < ny) ? tile_finite(v)
                                       : (j0 >= ny || isfinite(v.x)) && (j0 + 1 >= ny || isfinite(v.y)) &&
                                             (j0 + 2 >= ny || isfinite(v.z));
          fin &= f;
        }
      };
      auto st = [&](float* p, const float4& v) {
        tile_st(p, row, j0, ny, vec, v);
        test(v);
      };
      // ez = naz*dz; with loss an Inf or NaN of ez is in iz too.  (The adjoint's modes are
      // not tested; with this line in them 1500 steps at 1024^2 took 10.35 ms against 10.30)
      if (!LOSSY && !REC && !REV) test(to4(mul4(f4(at(A_NAZ, r)), dz[r])));
      st(a.out.dz, to4(dz[r]));
      st(a.out.hx, to4(hx[r]));
      st(a.out.hy, to4(hy[r]));
      if (PML) {
        st(a.out.ihx, to4(ihx_get(r)));
        st(a.out.ihy, at(A_IHY, r));
      }
      if (LOSSY) st(a.out.iz, at(A_IZ, r));
    }
    if constexpr (REV) {
      auto put = [&](float* g, const float4& v4) {
        const float v[4] = {v4.x, v4.y, v4.z, v4.w};
        if (g && box_c && box_row(i))
          for (int c = 0; c < 4; ++c) {
            const int bj = j0 + c - a.adj.box.j0;
            if (bj >= 0 && bj < a.adj.box.nj) g[(size_t)(i - a.adj.box.i0) * a.adj.box.nj + bj] = v[c];
          }
      };
      put(a.adj.grad_naz, at(A_G, r));
      if (LOSSY) put(a.adj.grad_nbz, at(A_GB, r));
    }
  }
  if (!fin) raise_status(a.status, ST_NONFINITE);
}

template <int V, bool LOSSY, bool PML, int MODE>
int launch_t(const TileArgs& a, cudaStream_t st) {
  auto kern = k_tile<V, LOSSY, PML, MODE>;
  const size_t smem = tile_smem_bytes(V, LOSSY, PML, MODE);
  cudaError_t e = cudaSuccess;
  if (smem > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.n_ti * a.n_tj, 1, 1);
    cfg.blockDim = dim3(kTileWarps * 32, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;  // all blocks resident: they wait on one another
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, a);
  }
  if (e != cudaSuccess) {
    fdtd_host::note_cuda_error(e);
    return FDTD_ERR_CUDA;
  }
  return fdtd_host::check_launch();
}

}  // namespace
}  // namespace fdtd
