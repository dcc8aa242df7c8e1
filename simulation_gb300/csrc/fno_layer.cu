// One spectral layer of the surrogate, from its input activation to the next
// layer's DFT coefficients, in one kernel:
//
//   z  = x W^T + Psi G^T + b          (pointwise + inverse DFT, one accumulator)
//   x' = GELU(z)                      BF16 [B][N][128]
//   F  = x'^T Phi^T                   -> BF16 coefficients of the next mode mixing
//   or h = mean over positions of x'  (last layer)
//
// What bounds it: HBM.  A sample's activation is 0.5 MB at N = 2048, and as
// separate products a layer reads it twice (DFT, pointwise) and writes it
// once, with FP32 coefficients permuted by two more kernels between.  Here x is
// read once and x' written once; the DFT takes x' from shared memory while it
// is still there, and the last layer's x' is never stored.  The coefficients
// leave TMEM in the mode-major layout of the mixing product, and its BF16
// output is loaded as an MN-major operand, so nothing is permuted.
//
// A CTA takes whole samples (the DFT sums over a sample's positions in one
// accumulator, in the order of the separate product: results are bitwise the
// same), 128 positions a tile, one persistent CTA per SM:
//   warps 0-15  epilogue, two groups of eight on alternate tiles: 32 rows x 64
//               channels a warp from TMEM, bias, GELU, BF16 into the swizzled
//               shared tile that is at once the TMA store's source and the
//               DFT's A operand; once a sample, F to global;
//   warp 16     TMA: x (two stages), Psi (three), G once a sample;
//   warp 17     MMA: tile i's product, then tile i-1's DFT;
//   warp 18     TMA store of x'; in the last layer warps 18-25 add the rows.
// The DFT's B operand is the Psi tile that the inverse used (rows of cos and sin
// times 2/N, a power of two, undone exactly at the end), so Phi is not loaded.
// Shared memory: W 32 KB (resident), G 16, x 2 x 32, Psi 3 x 16, output 2 x 32.
// Every wait on an mbarrier is bounded (about 2 s): on expiry the kernel
// records FDTD_STATUS_TIMEOUT, waits for no further phase and finishes.
//
// 4096 samples of 2048 positions: 690 us a middle layer, 4.3 GB at 6.2 TB/s
// (with MMAs, GELU and stores to shared memory cut out one by one it stays
// above 650); 608 the first (packed inputs; 630 from rows padded to 64), 510 the
// last.  As separate
// kernels (DFT, permutes, pointwise, mean pool) the network took 6.1 ms, now
// 2.85; one sample alone 142 us instead of 171, so there is no size below
// which the separate form is kept for this shape.  With one group of eight
// warps 3.5 ms, sixteen on one tile 3.4, issuing the MMAs from a converged warp
// 3.3, Psi for Phi and alternating groups 3.0.
#include <algorithm>

#include "tc_common.cuh"

namespace fdtd {
namespace {

constexpr int LC = 128;             // channels
constexpr int LM2 = 64;             // retained coefficients per channel (32 cos + 32 sin)
constexpr int LT = 128;             // positions per tile
constexpr int LEPI = 16;            // epilogue warps: two groups of eight
constexpr int W_TMA = LEPI, W_MMA = LEPI + 1, W_OUT = LEPI + 2;  // W_OUT ..: one store warp or eight pool warps
constexpr int layer_threads(bool last) { return 32 * (LEPI + 2 + (last ? 8 : 1)); }
constexpr uint32_t OFF_G = 32768, OFF_X = OFF_G + 16384, X_STAGE = 32768, OFF_PSI = OFF_X + 2 * X_STAGE,
                   PSI_STAGE = 16384, OFF_OUT = OFF_PSI + 3 * PSI_STAGE, OUT_BYTES = 32768,
                   OFF_BIAS = OFF_OUT + 2 * OUT_BYTES, OFF_BAR = OFF_BIAS + 4 * LC, N_BAR = 26,
                   LAYER_SMEM = 1024 + OFF_BAR + 8 * N_BAR + 16;

struct LayerArgs {
  int B, N;
  const float* bias;
  __nv_bfloat16* fm;   // [32][B][256] (not of the last layer)
  __nv_bfloat16* h;    // [B][128] (last layer)
  __nv_bfloat16* pre;  // z in BF16 [B][N][128], optional
  int* status;
};

__device__ __forceinline__ void tma_store_3d(const CUtensorMap* tm, uint32_t src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tm)),
               "r"(src), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t a) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}

// two GELUs: the operations of gelu(), in pairs
__device__ __forceinline__ float2 gelu2(float2 z) {
  const float2 c = make_float2(0.044715f, 0.044715f), d = make_float2(0.7978845608028654f, 0.7978845608028654f);
  const float2 u = __fmul2_rn(d, __ffma2_rn(__fmul2_rn(c, z), __fmul2_rn(z, z), z));
  const float2 t = make_float2(tanh_hw(u.x), tanh_hw(u.y));
  return __fmul2_rn(__fmul2_rn(make_float2(0.5f, 0.5f), z), __fadd2_rn(make_float2(1.f, 1.f), t));
}

__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// K1: input channels, 128, or 16 for packed inputs
template <int K1, bool LAST, bool PRE>
__global__ void __launch_bounds__(layer_threads(LAST), 1)
    k_layer(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
            const __grid_constant__ CUtensorMap tmPsi, const __grid_constant__ CUtensorMap tmG,
            const __grid_constant__ CUtensorMap tmOut, const LayerArgs a) {
  // 64 channels (128 bytes) of 128 rows a block of x and of W, or all 16 (32 bytes)
  constexpr int XB = K1 == 16 ? 1 : K1 / 64, X_BLOCK = K1 == 16 ? 4096 : 16384;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sm = smem_u32(base);
  float* sbias = reinterpret_cast<float*>(base + OFF_BIAS);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base + OFF_BAR + 8 * N_BAR);
  auto bar = [&](int k) { return sm + OFF_BAR + 8u * (uint32_t)k; };
  // barrier numbers; those of two are indexed by the parity of the tile or the sample, Psi's by tile mod 3
  enum { XFULL = 0, XEMPTY = 2, TFULL = 4, TEMPTY = 6, OREADY = 8, OFREE = 10, FFULL = 12, FEMPTY = 14, PFULL = 16,
         PEMPTY = 19, GFULL = 22, GEMPTY = 23, WFULL = 24 };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tiles = a.N / LT;
  bool ok = true;
  auto wait = [&](int k, int n) {  // the n-th completion (0-based) of barrier k
    if (ok) ok = mbar_wait(bar(k), (uint32_t)(n & 1), a.status);
  };
  auto wait_warp = [&](int k, int n) {
    wait(k, n);
    ok = __all_sync(0xffffffffu, ok);
  };

  if (threadIdx.x < LC) sbias[threadIdx.x] = a.bias[threadIdx.x];
  if (threadIdx.x == 0) {
    for (int p = 0; p < 2; ++p) {
      mbar_init(bar(XFULL + p), 1);
      mbar_init(bar(XEMPTY + p), 1);
      mbar_init(bar(TFULL + p), 1);
      mbar_init(bar(TEMPTY + p), 8);
      mbar_init(bar(OREADY + p), 8);
      mbar_init(bar(OFREE + p), LAST ? 8 : 2);  // eight pool warps, or the DFT's commit and the store
      mbar_init(bar(FFULL + p), 1);
      mbar_init(bar(FEMPTY + p), 8);
    }
    for (int k = PFULL; k <= WFULL; ++k) mbar_init(bar(k), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;  // columns 0-255 tiles, 256-383 DFTs

  if (warp == W_TMA) {
    // ------------------------------------------------ x, Psi and G
    if (lane == 0) {
      mbar_expect_tx(bar(WFULL), XB * X_BLOCK);
      for (int k = 0; k < XB; ++k) tma_load_3d(sm + k * X_BLOCK, &tmW, 64 * k, 0, 0, bar(WFULL));
      int i = 0, np = 0, ng = 0;  // x tiles, Psi tiles and G loaded
      for (int b = blockIdx.x; b < a.B && ok; b += gridDim.x)
        for (int t = 0; t < tiles && ok; ++t) {
          const int p = i & 1, p3 = i % 3;
          if (i >= 2) wait(XEMPTY + p, (i >> 1) - 1);
          if (!ok) break;
          const uint32_t dst = sm + OFF_X + p * X_STAGE;
          mbar_expect_tx(bar(XFULL + p), XB * X_BLOCK);
          for (int k = 0; k < XB; ++k) tma_load_3d(dst + k * X_BLOCK, &tmX, 64 * k, t * LT, b, bar(XFULL + p));
          ++i;
          if (t == 0) {
            if (ng >= 1) wait(GEMPTY, ng - 1);
            if (!ok) break;
            mbar_expect_tx(bar(GFULL), 16384);
            for (int h = 0; h < 2; ++h)
              for (int part = 0; part < 2; ++part)
                tma_load_3d(sm + OFF_G + h * 8192 + part * 4096, &tmG, part * LC + 64 * h, b, 0, bar(GFULL));
            ++ng;
          }
          if (np >= 3) wait(PEMPTY + p3, np / 3 - 1);
          if (!ok) break;
          mbar_expect_tx(bar(PFULL + p3), 16384);
          tma_load_3d(sm + OFF_PSI + p3 * PSI_STAGE, &tmPsi, 0, t * LT, 0, bar(PFULL + p3));
          ++np;
        }
      if (!ok) {  // a wait ran out: let the copies in flight land before the CTA ends
        mbar_wait(bar(WFULL), 0, a.status);
        for (int j = i > 2 ? i - 2 : 0; j < i; ++j)
          mbar_wait(bar(XFULL + (j & 1)), (uint32_t)((j >> 1) & 1), a.status);
        for (int j = np > 3 ? np - 3 : 0; j < np; ++j)
          mbar_wait(bar(PFULL + j % 3), (uint32_t)((j / 3) & 1), a.status);
        if (ng >= 1) mbar_wait(bar(GFULL), (uint32_t)((ng - 1) & 1), a.status);
      }
    }
  } else if (warp == W_MMA) {
    // ------------------------------------------------ MMA issuer
    const uint32_t lead = elect_lane();
    constexpr uint32_t id_w = instr_desc(LT, LC, 0, 0), id_g = instr_desc(LT, LC, 0, 1),
                       id_f = instr_desc(LC, LM2, 1, 1);
    int i = 0, s = 0;
    // the DFT of the next tile: tile j of this CTA, tile t of its sj-th sample
    int j = 0, sj = 0, jt = 0;
    auto dft = [&]() {
      const int t = jt, p = j & 1, p3 = j % 3, q = sj & 1;
      if (t == 0 && sj >= 2) wait_warp(FEMPTY + q, (sj >> 1) - 1);
      wait_warp(OREADY + p, j >> 1);
      if (!ok) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t so = sm + OFF_OUT + p * OUT_BYTES, sp = sm + OFF_PSI + p3 * PSI_STAGE,
                     dacc = tmem + 256 + q * LM2;
#pragma unroll
      for (int kk = 0; kk < LT / 16; ++kk)
        mma_bf16(lead, dacc, smem_desc(so + kk * 2048, 16384, 1024), smem_desc(sp + kk * 2048, 8192, 1024), id_f,
                 (t > 0 || kk > 0) ? 1u : 0u);
      mma_commit(lead, bar(OFREE + p));
      mma_commit(lead, bar(PEMPTY + p3));
      if (t + 1 == tiles) mma_commit(lead, bar(FFULL + q));
      ++j;
      if (++jt == tiles) {
        jt = 0;
        ++sj;
      }
    };
    wait_warp(WFULL, 0);
    for (int b = blockIdx.x; b < a.B && ok; b += gridDim.x, ++s)
      for (int t = 0; t < tiles && ok; ++t, ++i) {
        const int p = i & 1, p3 = i % 3;
        if (i >= 2) wait_warp(TEMPTY + p, (i >> 1) - 1);
        wait_warp(XFULL + p, i >> 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sx = sm + OFF_X + p * X_STAGE, sp = sm + OFF_PSI + p3 * PSI_STAGE, dacc = tmem + p * LC;
        if constexpr (K1 == 16) {
          mma_bf16(lead, dacc, smem_desc32(sx), smem_desc32(sm), id_w, 0u);
        } else {
#pragma unroll
          for (int k = 0; k < XB; ++k)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              mma_bf16(lead, dacc, smem_desc(sx + k * 16384 + kk * 32, 16, 1024),
                     smem_desc(sm + k * 16384 + kk * 32, 16, 1024), id_w, (k > 0 || kk > 0) ? 1u : 0u);
        }
        mma_commit(lead, bar(XEMPTY + p));
        if (t == 0) wait_warp(GFULL, s);
        wait_warp(PFULL + p3, i / 3);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          mma_bf16(lead, dacc, smem_desc(sp + kk * 32, 16, 1024), smem_desc(sm + OFF_G + kk * 2048, 8192, 1024), id_g,
                   1u);
        if (LAST) mma_commit(lead, bar(PEMPTY + p3));
        if (t + 1 == tiles) mma_commit(lead, bar(GEMPTY));
        mma_commit(lead, bar(TFULL + p));
        if constexpr (!LAST) {
          if (i >= 1) dft();
        }
      }
    if constexpr (!LAST) {
      while (ok && j < i) dft();
    }
  } else if (warp >= W_OUT) {
    if constexpr (!LAST) {
      // ---------------------------------------------- store of x'
      if (lane == 0) {
        int i = 0;
        for (int b = blockIdx.x; b < a.B && ok; b += gridDim.x)
          for (int t = 0; t < tiles && ok; ++t, ++i) {
            const int p = i & 1;
            wait(OREADY + p, i >> 1);
            if (!ok) break;
            const uint32_t src = sm + OFF_OUT + p * OUT_BYTES;
            tma_store_3d(&tmOut, src, 0, t * LT, b);
            tma_store_3d(&tmOut, src + 16384, 64, t * LT, b);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            mbar_arrive(bar(OFREE + p));
          }
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
      }
    } else {
      // ---------------------------------------------- mean pool
      // sums in the order of the separate kernel: rows py, py + 16, .. of a sample
      // in one register per channel, then the 16 of them
      const int tid = threadIdx.x - 32 * W_OUT, pg = tid & 15, py = tid >> 4;
      int i = 0;
      for (int b = blockIdx.x; b < a.B; b += gridDim.x) {
        float2 pool[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) pool[k] = make_float2(0.f, 0.f);
        for (int t = 0; t < tiles; ++t, ++i) {
          const int p = i & 1;
          wait_warp(OREADY + p, i >> 1);
          const unsigned char* col =
              base + OFF_OUT + p * OUT_BYTES + (pg >> 3) * 16384 + py * 128 + (((pg & 7) ^ (py & 7)) << 4);
#pragma unroll
          for (int m = 0; m < LT / 16; ++m) {
            const uint4 u = *reinterpret_cast<const uint4*>(col + m * 2048);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 h2 = *reinterpret_cast<const __nv_bfloat162*>(&w[e]);
              pool[e] = __fadd2_rn(pool[e], make_float2(__low2float(h2), __high2float(h2)));
            }
          }
          if (t + 1 == tiles) {  // the tile just read makes room for the 16 x 128 sums
            float* part = reinterpret_cast<float*>(base + OFF_OUT + p * OUT_BYTES);
            asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
            for (int k = 0; k < 4; ++k) *reinterpret_cast<float2*>(part + py * LC + pg * 8 + 2 * k) = pool[k];
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (tid < LC) {
              float v = 0.f;
              for (int yy = 0; yy < 16; ++yy) v += part[yy * LC + tid];
              a.h[(size_t)b * LC + tid] = __float2bfloat16_rn(v / a.N);
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(OFREE + p));
        }
      }
    }
  } else {
    // ------------------------------------------------ epilogue: group grp takes tiles of its parity
    const int grp = warp >> 3, lg = warp & 3, hh = (warp >> 2) & 1;  // 32 TMEM lanes = rows, half of the channels
    const int row = lg * 32 + lane;
    const uint32_t lanes = (uint32_t)(lg * 32) << 16;
    // F of the sj-th sample (batch index b): lane = channel, half hh = real or imaginary part.  The DFT
    // was taken with Psi's rows, cos and sin scaled by 2/N (mode 0: 1/N), a power of two: undone exactly
    auto coefficients = [&](int sj, int b) {
      const int q = sj & 1;
      wait_warp(FFULL + q, sj >> 1);
      if (!ok) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t r[32];
      tmem_ld32(tmem + lanes + 256 + q * LM2 + hh * 32, r);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(FEMPTY + q));
      __nv_bfloat16* dst = a.fm + (size_t)b * 2 * LC + hh * LC + row;
      const float half = 0.5f * (float)a.N;
#pragma unroll
      for (int k = 0; k < 32; ++k)
        dst[(size_t)k * a.B * 2 * LC] = __float2bfloat16_rn(__uint_as_float(r[k]) * (k ? half : 2.f * half));
    };
    int i = 0, s = 0;
    for (int b = blockIdx.x; b < a.B; b += gridDim.x, ++s) {
      for (int t = 0; t < tiles; ++t, ++i) {
        const int p = i & 1;
        if (p == grp) {
          wait_warp(TFULL + p, i >> 1);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          unsigned char* out = base + OFF_OUT + p * OUT_BYTES + hh * 16384 + row * 128;
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            uint32_t r[32];
            tmem_ld32(tmem + lanes + p * LC + hh * 64 + g * 32, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (g == 1) {
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
              __syncwarp();
              if (lane == 0) mbar_arrive(bar(TEMPTY + p));
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // 8 channels = one 16-byte chunk of the swizzled row
              const int c0 = hh * 64 + g * 32 + 8 * j;
              const float4 b0 = *reinterpret_cast<const float4*>(sbias + c0);
              const float4 b1 = *reinterpret_cast<const float4*>(sbias + c0 + 4);
              const float2 bb[4] = {{b0.x, b0.y}, {b0.z, b0.w}, {b1.x, b1.y}, {b1.z, b1.w}};
              uint32_t w[4], wp[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int c = 8 * j + 2 * e;
                const float2 z =
                    __fadd2_rn(make_float2(__uint_as_float(r[c]), __uint_as_float(r[c + 1])), bb[e]);
                if constexpr (PRE) wp[e] = bf16x2(z.x, z.y);
                const float2 y = gelu2(z);
                w[e] = bf16x2(y.x, y.y);
              }
              if constexpr (PRE) {
                __nv_bfloat16* pre = a.pre + ((size_t)b * a.N + t * LT + row) * LC + c0;
                *reinterpret_cast<uint4*>(pre) = make_uint4(wp[0], wp[1], wp[2], wp[3]);
              }
              if (g == 0 && j == 0 && i >= 2) wait_warp(OFREE + p, (i >> 1) - 1);
              *reinterpret_cast<uint4*>(out + (((4 * g + j) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
          if constexpr (!LAST) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(OREADY + p));
        }
        if constexpr (!LAST) {
          if (t == min(1, tiles - 1) && s > 0 && ((s - 1) & 1) == grp) coefficients(s - 1, b - (int)gridDim.x);
        }
      }
    }
    if constexpr (!LAST) {
      if (s > 0 && ((s - 1) & 1) == grp) coefficients(s - 1, (int)blockIdx.x + (s - 1) * (int)gridDim.x);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

template <int K1, bool LAST, bool PRE>
int launch_layer(const CUtensorMap (&tm)[5], const LayerArgs& a, cudaStream_t st) {
  auto kern = k_layer<K1, LAST, PRE>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LAYER_SMEM);
  if (e != cudaSuccess) {
    fdtd_host::note_cuda_error(e);
    return FDTD_ERR_CUDA;
  }
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  kern<<<(unsigned)std::min(a.B, nsm), layer_threads(LAST), LAYER_SMEM, st>>>(tm[0], tm[1], tm[2], tm[3], tm[4], a);
  return fdtd_host::check_launch();
}

}  // namespace
}  // namespace fdtd

extern "C" int fno_layer_fwd(int B, int N, int C, int M, int K1, const void* x, const void* W, const float* bias,
                             const void* psi, const void* Gm, void* x_out, void* Fm_out, void* h_out,
                             void* pre, int* status, fdtd_stream_t stream) {
  using namespace fdtd;
  if (!x || !W || !bias || !psi || !Gm) return FDTD_ERR_NULL;
  if (!x_out != !Fm_out || !x_out == !h_out) return FDTD_ERR_ARG;  // (x_out, Fm_out) or h_out
  if (B < 1 || B > 65535 || N < LT || (N & (N - 1)) || C != LC || 2 * M != LM2 || (K1 != 16 && K1 != 128))
    return FDTD_ERR_SIZE;
  if (pre && K1 != 128) return FDTD_ERR_ARG;
  for (const void* p : {x, W, psi, Gm, (const void*)x_out, (const void*)pre})
    if ((uintptr_t)p & 15u) return FDTD_ERR_ALIGN;
  CUtensorMap tm[5];
  const int box = K1 == 16 ? 16 : 64;
  int rc = make_map(&tm[0], x, K1, N, B, K1, (uint64_t)N * K1, box, LT);
  if (!rc) rc = make_map(&tm[1], W, K1, LC, 1, K1, (uint64_t)LC * K1, box, LC);
  if (!rc) rc = make_map(&tm[2], psi, LM2, N, 1, LM2, (uint64_t)N * LM2, 64, LT);
  if (!rc) rc = make_map(&tm[3], Gm, 2 * LC, B, M, 2 * LC, (uint64_t)B * 2 * LC, 64, 1, 32);
  if (!rc && x_out) rc = make_map(&tm[4], x_out, LC, N, B, LC, (uint64_t)N * LC, 64, LT);
  if (rc) return rc;
  if (!x_out) tm[4] = tm[0];  // not used by the last layer
  const LayerArgs a{B, N, bias, (__nv_bfloat16*)Fm_out, (__nv_bfloat16*)h_out, (__nv_bfloat16*)pre, status};
  cudaStream_t st = (cudaStream_t)stream;
  if (K1 == 16) return h_out ? launch_layer<16, true, false>(tm, a, st) : launch_layer<16, false, false>(tm, a, st);
  if (pre) return h_out ? launch_layer<128, true, true>(tm, a, st) : launch_layer<128, false, true>(tm, a, st);
  return h_out ? launch_layer<128, true, false>(tm, a, st) : launch_layer<128, false, false>(tm, a, st);
}
