// Fused 1D run of any line length: the line is cut into overlapping chunks,
// one warp each, and a warp exchanges cells with its neighbours only once in
// H steps instead of twice in every step.
//
// Layout.  Warp g of n holds the 32*CPT consecutive cells from g*S on in
// registers, CPT per lane, S = (32 - 2L)*CPT.  Its outer L lanes on either
// side are halo: copies of the neighbours' cells, advanced redundantly.  One
// step moves information by one cell, so after H = L*CPT steps the wrong
// values that creep in from the chunk's ends have just reached the owned
// cells, and the halo lanes are then rewritten with the neighbours' owned
// values.  Warp 0 and warp n-1 own their outer lanes too (the line ends
// there).  With n minimal, cell nx-1 lies in the last warp alone, so the
// high-side ABC state has one owner.
//
// What bounds a step is the dependent chain hy -> shuffle -> ex -> shuffle ->
// hy (about 70 cycles) when few warps share an SM, and the issue slots when
// many do; halo_plan weighs both against the cost of the exchange (a block or
// cluster barrier) and picks cells per lane, halo lanes and cluster size.
//
// The step order (E, source, DFT, ABC, H; fd1d/program/fd1d_2_2.py:138-142)
// and the per-cell formulas are those of the per-function kernels, so the
// results are bitwise equal to theirs.  Cells past the end of the line carry
// zero coefficients, so they stay 0; only the warps that hold the line's
// ends, the source or a probe leave the uniform cell loops, by warp-uniform
// branches.
//
// The running DFT of every cell is kept in registers (NFM frequencies per
// cell) for the whole run; only longer frequency lists accumulate in place.
#pragma once

#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "fdtd_common.cuh"

namespace fdtd {

struct Halo1DArgs {
  fdtd1d_params p;
  fdtd1d_state s;
  int t0, nsteps;
  int n;  // warps that hold cells
  int L;  // halo lanes on each side (0 when n = 1)
};

// NFM, what the run keeps of the every-cell DFT: 0 nothing (probes only);
// 1 accumulators in global memory; 4 or 8 in registers, up to NFM frequencies
__host__ __device__ constexpr int halo_fields(int form) {  // (ex|dx), hy, [ix], [sx]
  return form == FDTD1D_FORM_DEBYE ? 4 : form == FDTD1D_FORM_DFORM ? 3 : 2;
}
// threads per block each instantiation is compiled for: 512 leave 128
// registers a thread; Debye holds 9 values per cell, 144 at 16 cells
__host__ __device__ constexpr int halo_max_threads(int form, int cpt) {
  return form != FDTD1D_FORM_DEBYE ? 512 : cpt == 16 ? 256 : cpt == 8 ? 640 : 512;
}
constexpr int kHaloChunk = 32;  // steps per chunk of source values, DFT rows and probe samples
// dynamic shared memory in floats: two exchange buffers of both edges of each
// warp; per warp two chunks of (cos, -sin) rows (every-cell DFT in registers)
// and one chunk of samples of each probe
__host__ __device__ constexpr size_t halo_exch_floats(int form, int warps, int hc) {
  return (size_t)2 * warps * 2 * halo_fields(form) * hc;
}
__host__ __device__ constexpr size_t halo_tw_floats(int nfm, int nf) {
  return nfm >= 4 ? (size_t)2 * kHaloChunk * 2 * nf : 0;
}
__host__ __device__ constexpr size_t halo_smem_bytes(int form, int nfm, int warps, int hc, int nf, int nprobe) {
  return sizeof(float) * (halo_exch_floats(form, warps, hc) +
                          warps * (halo_tw_floats(nfm, nf) + (size_t)(nf > 0 ? nprobe : 0) * kHaloChunk));
}

namespace {

namespace cgx = cooperative_groups;

__device__ __forceinline__ void halo_cp4(float* dst, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}

// a if the mask is all ones, b if it is zero: one bitwise select, no predicate
__device__ __forceinline__ float halo_sel(unsigned m, float a, float b) {
  return __uint_as_float((__float_as_uint(a) & m) | (__float_as_uint(b) & ~m));
}

template <int FORM, int CPT, int NFM>
__global__ void __launch_bounds__(halo_max_threads(FORM, CPT)) k_fd1d_halo(const Halo1DArgs a) {
  constexpr bool DF = (FORM == FDTD1D_FORM_DFORM || FORM == FDTD1D_FORM_DEBYE);
  constexpr bool DB = (FORM == FDTD1D_FORM_DEBYE);
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int NFLD = halo_fields(FORM);
  constexpr bool REGD = NFM >= 4;
  constexpr int NFA = REGD ? NFM : 1;
  extern __shared__ float hsm[];
  const fdtd1d_params& p = a.p;
  const fdtd1d_state& s = a.s;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int rank = (int)cgx::this_cluster().block_rank(), C = (int)cgx::this_cluster().num_blocks();
  const int gw = rank * W + w;
  const int n = a.n, L = a.L, HC = L * CPT;
  const bool active = gw < n;
  const int nx = p.nx;
  const int g0 = (gw * (32 - 2 * L) + lane) * CPT;  // this lane's first cell, a multiple of CPT
  const bool owned = active && (gw == 0 || lane >= L) && (gw == n - 1 || lane < 32 - L);

  // ---- state and coefficients
  float ex[CPT], hy[CPT], dx[CPT], ixa[CPT], sxa[CPT];
  float k0[CPT], k1[CPT], k2[CPT], k3[CPT];
  float fr[NFA][CPT], fi[NFA][CPT];
  const int nf = p.nf;
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    const int g = g0 + c;
    const bool in = active && g < nx;
    ex[c] = in ? s.ex[g] : 0.f;
    hy[c] = in ? s.hy[g] : 0.f;
    dx[c] = (DF && in) ? s.dx[g] : 0.f;
    ixa[c] = (DF && in) ? s.ix[g] : 0.f;
    sxa[c] = (DB && in) ? s.sx[g] : 0.f;
    k0[c] = k1[c] = k2[c] = k3[c] = 0.f;
    if (in) {
      if (FORM == FDTD1D_FORM_CB) k0[c] = __ldg(p.cb + g);
      if (FORM == FDTD1D_FORM_CACB) {
        k0[c] = __ldg(p.ca + g);
        k1[c] = __ldg(p.cb + g);
      }
      if (DF) {
        k0[c] = __ldg(p.nax + g);
        k1[c] = __ldg(p.nbx + g);
      }
      if (DB) {
        k2[c] = __ldg(p.ncx + g);
        k3[c] = __ldg(p.ndx + g);
      }
    }
#pragma unroll
    for (int f = 0; f < NFA; ++f) {
      const bool have = REGD && in && f < nf;
      fr[f][c] = have ? s.r_pt[(size_t)f * nx + g] : 0.f;
      fi[f][c] = have ? s.i_pt[(size_t)f * nx + g] : 0.f;
    }
  }
  // ---- the cells that differ, as one-hot lane masks: the source cell, nx-1 and nx-2
  const int hi_c = (gw == n - 1 && (nx - 1) / CPT == g0 / CPT) ? (nx - 1) - g0 : -1;
  const bool own_lo = p.abc && gw == 0 && lane == 0, own_hi = p.abc && hi_c >= 0;
  const bool soft = p.src_kind == FDTD_SRC_SOFT, have_src = p.src_kind != FDTD_SRC_NONE;
  const int sp = (active && have_src && p.src_k / CPT == g0 / CPT) ? p.src_k - g0 : -1;
  const bool src_warp = __any_sync(kAll, sp >= 0);
  float bc0 = 0.f, bc1 = 0.f, bc2 = 0.f, bc3 = 0.f;
  if (own_lo) {
    bc0 = s.bc[0];
    bc1 = s.bc[1];
  }
  if (own_hi) {
    bc2 = s.bc[2];
    bc3 = s.bc[3];
  }
  const unsigned z0 = (gw == 0 && lane == 0) ? kAll : 0u;  // cell 0 is never E-updated
  const unsigned lo_m = own_lo ? kAll : 0u;
  // probes whose cell this warp owns: one byte of lane and one of cell index each
  int nq = 0;
  unsigned long long q_lane = 0, q_cell = 0, q_id = 0;
  if (nf > 0)
    for (int q = 0; q < p.nprobe; ++q) {
      const unsigned m = __ballot_sync(kAll, owned && p.probe_k[q] / CPT == g0 / CPT);
      if (m) {
        q_lane |= (unsigned long long)(__ffs(m) - 1) << (8 * nq);
        q_cell |= (unsigned long long)(p.probe_k[q] % CPT) << (8 * nq);
        q_id |= (unsigned long long)q << (8 * nq);
        ++nq;
      }
    }
  float* const xb = hsm;  // exchange buffers
  float* const tws = hsm + halo_exch_floats(FORM, W, HC) + (size_t)w * halo_tw_floats(NFM, nf);  // [2][32][nf][2]
  float* const prb = hsm + halo_exch_floats(FORM, W, HC) + (size_t)W * halo_tw_floats(NFM, nf) +
                     (size_t)w * p.nprobe * kHaloChunk;  // [nq][32] samples (nf > 0)
  const int t_end = a.t0 + a.nsteps;
  // rows tc .. tc+31 of the DFT tables on their way into chunk buffer b
  auto stage_tw = [&](int tc, int b) {
    if constexpr (REGD) {
      const int m = min(kHaloChunk, t_end - tc) * nf;
      float* const d = tws + b * 2 * kHaloChunk * nf;
      for (int x = lane; x < m; x += 32) {
        halo_cp4(d + 2 * x, p.dft_cos + (size_t)tc * nf + x);
        halo_cp4(d + 2 * x + 1, p.dft_sin + (size_t)tc * nf + x);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
  };

  // ---- m time steps t+1 .. t+m (rows j0 .. of the chunk); KIND bit 0: this
  // warp holds cell 0 or the source, bit 1: it holds nx-1, bit 2: a probe
  auto steps = [&](auto kind, const int t, const int j0, const int m, const float vc, const int b) {
    constexpr int KIND = decltype(kind)::value;
    constexpr bool LO = (KIND & 1) != 0, HI = (KIND & 2) != 0, PRB = (KIND & 4) != 0;
    constexpr int UN = CPT >= 16 ? 1 : CPT >= 8 ? 2 : 4;
    [[maybe_unused]] const float2* row = reinterpret_cast<const float2*>(tws + b * 2 * kHaloChunk * nf) + j0 * nf;
    // (masks are made here, so that the plain loop keeps no registers for them)
    unsigned sm[LO ? CPT : 1], hm[HI ? CPT : 1], nm[HI ? CPT : 1];
    float hc[HI ? CPT : 1];
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      if (LO) sm[c] = c == sp ? kAll : 0u;
      if (HI) {
        hm[c] = own_hi && c == hi_c ? kAll : 0u;
        nm[c] = own_hi && c + 1 == hi_c ? kAll : 0u;
        hc[c] = g0 + c <= nx - 2 ? 0.5f : 0.f;  // hy[nx-1] is never updated
      }
    }
    const unsigned sa = soft ? kAll : 0u;
    [[maybe_unused]] float2 cs[NFA];
    if constexpr (REGD) {
#pragma unroll
      for (int f = 0; f < NFA; ++f) cs[f] = f < nf ? row[f] : make_float2(0.f, 0.f);
    }
#pragma unroll UN
    for (int i = 0; i < m; ++i) {
      const float hy_left = __shfl_up_sync(kAll, hy[CPT - 1], 1);
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const float hym = (c == 0) ? hy_left : hy[c - 1];
        if (!DF) {
          const float e = FORM == FDTD1D_FORM_CB ? ex_update_cb(ex[c], hym, hy[c], k0[c])
                                                 : ex_update_cacb(ex[c], hym, hy[c], k0[c], k1[c]);
          ex[c] = LO && c == 0 ? halo_sel(z0, ex[0], e) : e;
        } else {
          const float d = dx_update(dx[c], hym, hy[c]);
          dx[c] = LO && c == 0 ? halo_sel(z0, dx[0], d) : d;
        }
      }
      if (LO) {
        const float v = __shfl_sync(kAll, vc, j0 + i);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          float& f = DF ? dx[c] : ex[c];
          // soft: f + v; hard: v, as 0 + v
          f = halo_sel(sm[c], __fadd_rn(__uint_as_float(__float_as_uint(f) & sa), v), f);
        }
      }
      if (DF) {
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          float ixn = ixa[c], sxn = sxa[c];
          const float e = !DB ? ex_from_dx(dx[c], ixn, k0[c], k1[c])
                              : ex_from_dx_debye(dx[c], ixn, sxn, k0[c], k1[c], k2[c], k3[c]);
          ex[c] = LO && c == 0 ? halo_sel(z0, ex[0], e) : e;
          ixa[c] = LO && c == 0 ? halo_sel(z0, ixa[0], ixn) : ixn;
          if (DB) sxa[c] = LO && c == 0 ? halo_sel(z0, sxa[0], sxn) : sxn;
        }
      }
      // running DFT, before the ABC; the row of the next step is read a step ahead
      if constexpr (REGD) {
        row += nf;
#pragma unroll
        for (int f = 0; f < NFA; ++f) {
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            fr[f][c] = __fmaf_rn(cs[f].x, ex[c], fr[f][c]);
            fi[f][c] = __fmaf_rn(-cs[f].y, ex[c], fi[f][c]);
          }
          if (f < nf && i + 1 < m) cs[f] = row[f];
        }
      }
      if constexpr (NFM == 1) {
        if (owned) {
          for (int f = 0; f < nf; ++f) {
            const size_t r = (size_t)(t + i) * nf + f;
            const float cf = __ldg(p.dft_cos + r), sf = __ldg(p.dft_sin + r);
#pragma unroll
            for (int c = 0; c < CPT; ++c)
              if (g0 + c < nx) {
                const size_t o = (size_t)f * nx + g0 + c;
                s.r_pt[o] = __fmaf_rn(cf, ex[c], s.r_pt[o]);
                s.i_pt[o] = __fmaf_rn(-sf, ex[c], s.i_pt[o]);
              }
          }
        }
      }
      if (PRB) {
        auto sample = [&](int q) {
          const int pc = (int)((q_cell >> (8 * q)) & 255);
          float e = ex[0];
#pragma unroll
          for (int c = 1; c < CPT; ++c) e = c == pc ? ex[c] : e;
          if (lane == (int)((q_lane >> (8 * q)) & 255)) prb[q * kHaloChunk + j0 + i] = e;
        };
        sample(0);
        if (nq > 1)
          for (int q = 1; q < nq; ++q) sample(q);
      }
      // two-step-back ABC (fd1d/program/fd1d_1_2.py:47-48); the state moves in
      // every lane, only the owners' values are kept
      if (LO) {
        const float e1 = ex[1];
        ex[0] = halo_sel(lo_m, bc0, ex[0]);
        bc0 = bc1;
        bc1 = e1;
      }
      if (HI) {
        float e2 = __shfl_up_sync(kAll, ex[CPT - 1], 1);  // nx-2 when nx-1 is its lane's first cell
        unsigned acc = 0u;
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          acc |= __float_as_uint(ex[c]) & nm[c];
          ex[c] = halo_sel(hm[c], bc3, ex[c]);
        }
        bc3 = bc2;
        bc2 = hi_c == 0 ? e2 : __uint_as_float(acc);
      }
      const float ex_right = __shfl_down_sync(kAll, ex[0], 1);
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const float er = (c == CPT - 1) ? ex_right : ex[c + 1];
        hy[c] = HI ? __fmaf_rn(hc[c], __fsub_rn(ex[c], er), hy[c]) : hy_update(hy[c], ex[c], er);
      }
    }
  };

  // ---- the probes' DFT over one chunk of samples, steps t+1 .. t+m: lane f
  // holds frequency f while it adds them in step order
  auto probe_chunk = [&](const int t, const int m, const int b) {
    __syncwarp();
    for (int q = 0; q < nq; ++q) {
      const size_t base = (size_t)((q_id >> (8 * q)) & 255) * nf;
      for (int f = lane; f < nf; f += 32) {
        float r = s.r_pr[base + f], im = s.i_pr[base + f];
        const float* const e = prb + q * kHaloChunk;
        auto add = [&](int i, float c, float sn) {
          r = __fmaf_rn(c, e[i], r);
          im = __fmaf_rn(-sn, e[i], im);
        };
        if constexpr (REGD) {
          const float2* const row = reinterpret_cast<const float2*>(tws + b * 2 * kHaloChunk * nf) + f;
#pragma unroll 8
          for (int i = 0; i < m; ++i) add(i, row[i * nf].x, row[i * nf].y);
        } else {
          const float* const c = p.dft_cos + (size_t)t * nf + f;
          const float* const sn = p.dft_sin + (size_t)t * nf + f;
          // 16 rows' loads are in flight at once: one row at a time waits for each
          int i = 0;
          for (; i + 16 <= m; i += 16) {
            float cv[16], sv[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              cv[k] = __ldg(c + (size_t)(i + k) * nf);
              sv[k] = __ldg(sn + (size_t)(i + k) * nf);
            }
#pragma unroll
            for (int k = 0; k < 16; ++k) add(i + k, cv[k], sv[k]);
          }
          for (; i < m; ++i) add(i, __ldg(c + (size_t)i * nf), __ldg(sn + (size_t)i * nf));
        }
        s.r_pr[base + f] = r;
        s.i_pr[base + f] = im;
      }
    }
    __syncwarp();
  };

  // ---- refresh of the halo lanes from the neighbours' owned cells
  // buffer [b][warp][side][field][c*L + i]: lane i of the edge's L lanes
  auto slot = [&](int b, int ww, int side) { return ((size_t)(b * W + ww) * 2 + side) * NFLD * HC; };
  auto exchange = [&](const int b) {
    auto put = [&](float* q, int i) {
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        q[c * L + i] = DF ? dx[c] : ex[c];
        q[HC + c * L + i] = hy[c];
        if (DF) q[2 * HC + c * L + i] = ixa[c];
        if (DB) q[3 * HC + c * L + i] = sxa[c];
      }
    };
    auto get = [&](const float* q, int i) {
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        (DF ? dx[c] : ex[c]) = q[c * L + i];
        hy[c] = q[HC + c * L + i];
        if (DF) ixa[c] = q[2 * HC + c * L + i];
        if (DB) sxa[c] = q[3 * HC + c * L + i];
      }
    };
    if (active) {
      if (gw > 0 && lane >= L && lane < 2 * L) put(xb + slot(b, w, 0), lane - L);
      if (gw < n - 1 && lane >= 32 - 2 * L && lane < 32 - L) put(xb + slot(b, w, 1), lane - (32 - 2 * L));
    }
    if (C > 1) cgx::this_cluster().sync();
    else __syncthreads();
    if (active) {
      if (gw > 0 && lane < L) {
        const float* q = w > 0 ? xb + slot(b, w - 1, 1)
                               : cgx::this_cluster().map_shared_rank(xb, rank - 1) + slot(b, W - 1, 1);
        get(q, lane);
      }
      if (gw < n - 1 && lane >= 32 - L) {
        const float* q = w < W - 1 ? xb + slot(b, w + 1, 0)
                                   : cgx::this_cluster().map_shared_rank(xb, rank + 1) + slot(b, 0, 0);
        get(q, lane - (32 - L));
      }
    }
  };

  // ---- time loop: runs of steps up to the next exchange or chunk end
  auto time_loop = [&](auto kind) {
    const int H = n > 1 ? HC : a.nsteps;
    float vc = (have_src && a.t0 + lane < t_end) ? __ldg(p.src_table + a.t0 + lane) : 0.f, vn = 0.f;
    stage_tw(a.t0, 0);
    int tb = 0, hb = 0;  // chunk and exchange buffers
    int since = 0;       // steps since the last exchange
    int j0 = 0;          // step within the chunk
    for (int t = a.t0; t < t_end;) {
      if (j0 == 0) {  // next chunk: its rows have been on their way for 32 steps
        if (t > a.t0) {
          vc = vn;
          tb ^= 1;
        }
        const int tn = t + kHaloChunk + lane;
        vn = (have_src && tn < t_end) ? __ldg(p.src_table + tn) : 0.f;
        if constexpr (REGD) {
          asm volatile("cp.async.wait_group 0;\n" ::: "memory");
          __syncwarp();  // every lane's copies have landed, and no lane still reads the other buffer
          if (t + kHaloChunk < t_end) stage_tw(t + kHaloChunk, tb ^ 1);
        }
      }
      const int m = min(min(H - since, kHaloChunk - j0), t_end - t);
      if (active) steps(kind, t, j0, m, vc, tb);
      t += m;
      since += m;
      j0 += m;
      if (nq > 0 && (j0 == kHaloChunk || t == t_end)) probe_chunk(t - j0, j0, tb);
      if (j0 == kHaloChunk) j0 = 0;
      if (since == H && t < t_end) {
        exchange(hb);
        hb ^= 1;
        since = 0;
      }
    }
  };
  const bool lo_kind = active && (gw == 0 || src_warp), hi_kind = gw == n - 1;
  if (nq > 0 && hi_kind) time_loop(std::integral_constant<int, 7>{});
  else if (nq > 0) time_loop(std::integral_constant<int, 5>{});
  else if (lo_kind && hi_kind) time_loop(std::integral_constant<int, 3>{});
  else if (lo_kind) time_loop(std::integral_constant<int, 1>{});
  else if (hi_kind) time_loop(std::integral_constant<int, 2>{});
  else time_loop(std::integral_constant<int, 0>{});
  // Results go where the fields came from, and a warp's halo lanes hold cells that
  // its neighbour stores.  A call of no more steps than H has no exchange, so this
  // barrier alone orders every warp's loads before any warp's stores; between blocks
  // it also keeps a block from leaving while a neighbour may read its buffers.
  if (C > 1) cgx::this_cluster().sync();
  else __syncthreads();

  // ---- results
  if (owned) {
    bool fin = true;
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const int g = g0 + c;
      if (g < nx) {
        s.ex[g] = ex[c];
        s.hy[g] = hy[c];
        fin &= isfinite(ex[c]) && isfinite(hy[c]);
        if (DF) {
          s.dx[g] = dx[c];
          s.ix[g] = ixa[c];
        }
        if (DB) s.sx[g] = sxa[c];
        if (REGD) {
#pragma unroll
          for (int f = 0; f < NFA; ++f)
            if (f < nf) {
              s.r_pt[(size_t)f * nx + g] = fr[f][c];
              s.i_pt[(size_t)f * nx + g] = fi[f][c];
            }
        }
      }
    }
    if (!fin) raise_status(s.status, ST_NONFINITE);
  }
  if (own_lo) {
    s.bc[0] = bc0;
    s.bc[1] = bc1;
  }
  if (own_hi) {
    s.bc[2] = bc2;
    s.bc[3] = bc3;
  }
}

}  // namespace

struct HaloPlan {
  int cpt = 0, L = 0, C = 0, W = 0, n = 0;  // cells per lane, halo lanes, blocks, warps per block, warps with cells
};

// Cells per lane, halo lanes and blocks for a line: the cheapest of all
// layouts that fit, by a model of the time of one step in ns, fitted to
// measured layouts of 200 to 65536 cells (cb form unless named):
//   * the dependent chain of a step, 50 + 3 per cell of a lane (longer for the
//     D forms and the DFT), which small lines cannot go below: 65 ns at 200
//     cells, 72 at 512;
//   * the issue slots of the warps that share a scheduler (q instructions per
//     cell, o per step): 38000 cells on 16 blocks take 128 ns with 8 cells per
//     lane and 3 warps per scheduler, 142 with 4 warps;
//   * one exchange (block barrier 220 ns, cluster barrier and distributed
//     shared memory 500-800) in H steps: 128 ns at H = 24, 142 at 16, 197 at 8.
//   * 16 cells per lane run 1.75x off the model (little interleaving of steps):
//     taken only where nothing smaller fits.
// False when no layout fits (the caller then steps per function).
inline bool halo_plan(int form, int nx, int nfm, int nf, int nprobe, int max_cluster, HaloPlan& best) {
  const double qs[4] = {4.6, 5.2, 7.5, 11.0};
  double best_cost = 1e30;
  for (int C = 1; C <= max_cluster; C *= 2)
    for (int cpt = 2; cpt <= 16; cpt *= 2) {
      if (nfm == 1 && cpt != 4 && cpt != (form == FDTD1D_FORM_DEBYE ? 8 : 16)) continue;  // the instantiations there are
      if ((nfm == 4 && cpt > 4) || (nfm == 8 && cpt > 2)) continue;
      for (int L = 1; L <= 8 && L * cpt <= kHaloChunk; ++L) {
        HaloPlan pl;
        pl.cpt = cpt;
        pl.C = C;
        if (nx <= 32 * cpt) {
          if (L > 1 || C > 1) continue;
          pl.n = 1;
        } else {
          const int S = (32 - 2 * L) * cpt;
          pl.L = L;
          pl.n = (nx - 2 * L * cpt + S - 1) / S;
        }
        pl.W = (pl.n + C - 1) / C;
        if (C > 1 && (pl.n + pl.W - 1) / pl.W <= C / 2) continue;  // half the blocks hold it
        if (pl.W * 32 > halo_max_threads(form, cpt)) continue;
        if (halo_smem_bytes(form, nfm, pl.W, pl.L * cpt, nf, nprobe) > 200 * 1024) continue;
        const double q = qs[form] + (nfm >= 4 ? 4.0 * nf : 0.0), o = nfm >= 4 ? 20.0 : 12.0;
        const double chain = 50.0 + 3.0 * cpt + (form >= FDTD1D_FORM_DFORM ? 25.0 : 0.0) + (nfm >= 4 ? 8.0 * cpt : 0.0);
        const double issue = ((pl.W + 3) / 4) * (cpt * q + o) * 0.6;
        const double exch = pl.n == 1 ? 0.0 : (C == 1 ? 220.0 : C <= 8 ? 500.0 : 800.0) / (pl.L * cpt);
        const double cost = std::max(chain, issue) * (cpt == 16 ? 1.75 : 1.0) + exch;
        if (cost < best_cost) {
          best_cost = cost;
          best = pl;
        }
      }
    }
  return best_cost < 1e30;
}

// launch of one form's instantiations (one translation unit per form)
int launch_fd1d_halo_cb(const Halo1DArgs& a, const HaloPlan& pl, int nfm, cudaStream_t st);
int launch_fd1d_halo_cacb(const Halo1DArgs& a, const HaloPlan& pl, int nfm, cudaStream_t st);
int launch_fd1d_halo_dform(const Halo1DArgs& a, const HaloPlan& pl, int nfm, cudaStream_t st);
int launch_fd1d_halo_debye(const Halo1DArgs& a, const HaloPlan& pl, int nfm, cudaStream_t st);

template <int FORM, int CPT, int NFM>
int launch_fd1d_halo_t(const Halo1DArgs& a, const HaloPlan& pl, cudaStream_t st) {
  auto kern = k_fd1d_halo<FORM, CPT, NFM>;
  if (pl.W * 32 > halo_max_threads(FORM, CPT)) return FDTD_ERR_ARG;
  const size_t smem = halo_smem_bytes(FORM, NFM, pl.W, pl.L * CPT, a.p.nf, a.p.nprobe);
  cudaError_t e = cudaSuccess;
  if (smem > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess && pl.C > 8) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) {
    fdtd_host::note_cuda_error(e);
    return FDTD_ERR_CUDA;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl.C, 1, 1);
  cfg.blockDim = dim3(pl.W * 32, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = pl.C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pl.C > 1 ? 1 : 0;
  if (pl.C > 8) {  // larger than every device must take: ask before launching
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
    if (e != cudaSuccess || clusters < 1) {
      (void)cudaGetLastError();
      return FDTD_ERR_UNSUPPORTED;
    }
  }
  e = cudaLaunchKernelEx(&cfg, kern, a);
  if (e != cudaSuccess) {
    fdtd_host::note_cuda_error(e);
    return FDTD_ERR_CUDA;
  }
  return fdtd_host::check_launch();
}

template <int FORM>
int launch_fd1d_halo_form(const Halo1DArgs& a, const HaloPlan& pl, int nfm, cudaStream_t st) {
#define FDTD_HALO_CASE(CC, NN) \
  if (pl.cpt == CC && nfm == NN) return launch_fd1d_halo_t<FORM, CC, NN>(a, pl, st);
  FDTD_HALO_CASE(2, 0) FDTD_HALO_CASE(4, 0) FDTD_HALO_CASE(8, 0) FDTD_HALO_CASE(16, 0)
  FDTD_HALO_CASE(4, 1) FDTD_HALO_CASE((FORM == FDTD1D_FORM_DEBYE ? 8 : 16), 1)
  FDTD_HALO_CASE(2, 4) FDTD_HALO_CASE(4, 4) FDTD_HALO_CASE(2, 8)
#undef FDTD_HALO_CASE
  return FDTD_ERR_ARG;
}

}  // namespace fdtd
