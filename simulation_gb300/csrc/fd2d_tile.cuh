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
#pragma once

#include <type_traits>

#include "fd2d_internal.cuh"
#include "fd2d_pack.cuh"

namespace fdtd {

constexpr int kTileWarps = 16;
constexpr int kTileCols = 128;

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
  int probe_i, probe_j;
  float* probe_ez;
  unsigned* flags;    // one per block, 32 words apart, zero at the start
  int T;              // steps between exchanges = halo rows
  int hc;             // halo columns on each side: T rounded up to whole lanes, or 0 with one tile per row
  int n_ti, n_tj;
  int own_r, own_c;   // owned rows and columns per tile
  int vec;            // ny % 4 == 0 and all arrays 16-byte aligned
};

struct TilePlan {
  int V = 0, T = 0, hc = 0, n_ti = 0, n_tj = 0, own_r = 0, own_c = 0;
};
constexpr int kTileMaxBlocks = 152;                       // one per SM
constexpr size_t kTileFlagBytes = kTileMaxBlocks * 128;  // flags of the largest launch

// shared memory of a block, in float4: arrays of 16*V rows of 32 float4 (naz,
// [ihy], [nbz, iz]), the strips' edge rows, the column and row coefficients
// (at 5 rows a warp ihx moves there too: with it in registers the general
// steps spill)
__host__ __device__ constexpr bool tile_ihx_smem(int V, bool pml) { return pml && V >= 5; }
__host__ __device__ constexpr int tile_arrays(int V, bool lossy, bool pml) {
  return 1 + (pml ? 1 : 0) + (lossy ? 2 : 0) + (tile_ihx_smem(V, pml) ? 1 : 0);
}
__host__ __device__ constexpr size_t tile_smem_bytes(int V, bool lossy, bool pml) {
  return sizeof(float4) * ((size_t)kTileWarps * V * 32 * tile_arrays(V, lossy, pml) + 2 * kTileWarps * 32 + 5 * 32 +
                           3 * kTileWarps * V);
}

// defined in fd2d_tile.cu
bool tile_plan(int nx, int ny, bool lossy, bool pml, int max_blocks, TilePlan& best);
int launch_tile(const fdtd2d_params& p, const FieldSet& in, const FieldSet& out, const FieldSet& x0, const FieldSet& x1,
                float* ez, int t0, int nsteps, int* status, float* probe_ez, unsigned* flags, const TilePlan& pl,
                cudaStream_t st);

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

template <int V, bool LOSSY, bool PML>
__global__ void __launch_bounds__(kTileWarps * 32, 1) k_tile(const TileArgs a) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int W = kTileWarps, R = W * V;
  constexpr bool IHXS = tile_ihx_smem(V, PML);
  constexpr int NARR = tile_arrays(V, LOSSY, PML);
  constexpr int A_NAZ = 0, A_IHY = 1, A_NBZ = PML ? 2 : 1, A_IZ = A_NBZ + 1, A_IHX = NARR - 1;
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
  const bool unit = __all_sync(kAll, col_ok && row_ok && j0 != 0 && !last_col);
  const int kind = src_here || probe_here ? kTilePoint : masks ? kTileEdge : unit ? kTileInt : kTileGen;
  xh[w * 32 + lane] = to4(hy[V - 1]);
  __syncthreads();

  // ---- one time step, t0+s+1; LAST stores ez
  auto step = [&](auto kind_tag, const int s, const bool last) {
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
      F4 e;
      const F4 na = f4(at(A_NAZ, r));
      if (LOSSY) {
        const F4 iz = f4(at(A_IZ, r));
        e = mul4(na, sub4(dz[r], iz));
        at(A_IZ, r) = to4(fma4(f4(at(A_NBZ, r)), e, iz));
      } else {
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
    xh[w * 32 + lane] = to4(hy[V - 1]);
    __syncthreads();
  };

  // flag 1: this block has read the input arrays, so its neighbours may write
  // into them (they can be an exchange set and the output)
  const int n_ex = (a.nsteps + T - 1) / T - 1;
  if (a.n_ti * a.n_tj > 1) raise_and_wait(1);
  for (int s = 0, e = 0; s < a.nsteps;) {
    const int m = min(T, a.nsteps - s);
    auto run = [&](auto kind_tag) {
      for (int q = 0; q < m; ++q) step(kind_tag, s + q, s + q + 1 == a.nsteps);
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
      auto st = [&](float* p, const float4& v) {
        tile_st(p, row, j0, ny, vec, v);
        if (a.status) {
          const bool f = (j0 + 3 < ny) ? tile_finite(v)
                                       : (j0 >= ny || isfinite(v.x)) && (j0 + 1 >= ny || isfinite(v.y)) &&
                                             (j0 + 2 >= ny || isfinite(v.z));
          fin &= f;
        }
      };
      st(a.out.dz, to4(dz[r]));
      st(a.out.hx, to4(hx[r]));
      st(a.out.hy, to4(hy[r]));
      if (PML) {
        st(a.out.ihx, to4(ihx_get(r)));
        st(a.out.ihy, at(A_IHY, r));
      }
      if (LOSSY) st(a.out.iz, at(A_IZ, r));
    }
  }
  if (a.status && !fin) raise_status(a.status, ST_NONFINITE);
}

}  // namespace
}  // namespace fdtd
