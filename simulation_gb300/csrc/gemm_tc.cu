// BF16 tensor-core GEMM for sm_103a (tcgen05 + TMA + TMEM), FP32 accumulation,
// with a fused epilogue (scale, bias, residual, GELU, accumulate, BF16/FP32
// output).  Written for the neural-operator surrogate's contractions
// (truncated DFT, inverse DFT, channel mixing, pointwise layers and their
// gradients).
//
// 128 x BN output tiles, persistent CTAs of 10 warps:
//   * warp 8, one lane: TMA producer.  Each pipeline stage holds a 128 x 64
//     A tile and a BN x 64 B tile in 128-byte-swizzled shared memory, loaded
//     by cp.async.bulk.tensor with mbarrier completion;
//   * warp 9, one lane: issues tcgen05.mma (kind::f16, BF16 inputs, FP32
//     accumulator in TMEM), four 16-deep MMAs per stage, and tcgen05.commit
//     to release the stage and, per tile, to signal the epilogue;
//   * warps 0-7: read the accumulator with tcgen05.ld (warp w owns TMEM lanes
//     32(w%4)..32(w%4)+31 = output rows, and half w/4 of the columns), return
//     the TMEM buffer, apply the epilogue and store; two accumulator buffers
//     overlap a tile's epilogue with the next tile's MMAs.  Eight epilogue
//     warps (two per SM sub-partition) rather than four: with four, the
//     pointwise layer's GEMM (K = 192) spent most of its time in the
//     epilogue and moved 3.6 TB/s; with eight it moves about 4.7 TB/s, and
//     sixteen (one 32-column chunk each) measured no faster.
// Operands may be K-major or MN-major (the transposed products of the
// backward pass need MN-major), selected per call.  Every wait on an mbarrier
// is bounded (about 2 s): on expiry the kernel records FDTD_STATUS_TIMEOUT in
// the status word and finishes without further waits.
#include <algorithm>

#include "tc_common.cuh"

namespace fdtd {
namespace {

constexpr int BM = 128;
constexpr int BK = 64;      // one 128-byte swizzle atom of BF16 along K
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 32 * (EPI_WARPS + 2);

struct GemmArgs {
  int M, N, K, batch;
  int a_mn, b_mn;
  float* c32;
  __nv_bfloat16* c16;
  long long ldc, stride_c;
  const float* bias;
  const __nv_bfloat16* res16;
  long long ldr, stride_r;
  float alpha;
  int act;
  int accumulate;
  __nv_bfloat16* pre16;  // optional pre-activation output (same layout as C)
  unsigned lbo_mn, sbo_mn;
  int a_shared, b_shared;  // operand shared by every batch entry (batch stride 0)
  int vec_ok;              // epilogue pointers/strides allow 16-byte vector access
  // optional second operand pair accumulated into the same tile: D += A2.B2'
  const __nv_bfloat16* z16;  // GB: pre-activations, laid out as C
  float* dsum;               // GB: column sums, added to
  int K2;
  int a2_mn, b2_mn, a2_shared, b2_shared;
  int* status;
};

// Persistent, warp-specialised kernel: warps 0-7 drain accumulators
// (epilogue), warp 8 is the TMA producer, warp 9 issues the MMAs.  Two TMEM
// accumulator buffers let the epilogue of one tile overlap the MMAs of the
// next; tiles are taken round-robin (tile = blockIdx.x + i * gridDim.x, M tiles
// fastest so neighbouring CTAs share B tiles in L2).
// GB: the output is the gradient through a GELU, BF16(acc * gelu'(z)), and its column
// sums are added to dsum: the backward pass of a layer needs its input's gradient
// only as that (N = BN, M % BM = 0).  Bound by HBM like the plain product, without
// the FP32 gradient's write and read: a training step of 256 took 2.47 ms with a
// separate pass, 2.25 so
template <int BN, int STAGES, bool GB>
__global__ void __launch_bounds__(THREADS, 1)
    k_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
           const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2, const GemmArgs a) {
  constexpr uint32_t A_BYTES = BM * BK * 2;
  constexpr uint32_t B_BYTES = BN * BK * 2;
  constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + STAGES * STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint64_t* tempty = bars + 2 * STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  // the bias of a one-column-tile GEMM (N <= BN: the same BN columns for every
  // tile) is staged once, so the epilogue reads it from shared memory
  float* sbias = reinterpret_cast<float*>(bars + 2 * STAGES + 6);  // 16-byte aligned for float4 reads

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int kb1 = (a.K + BK - 1) / BK;                       // k-blocks of the first pair
  const int kblocks = kb1 + (a.K2 > 0 ? (a.K2 + BK - 1) / BK : 0);
  const int mt = (a.M + BM - 1) / BM;
  const int nt = (a.N + BN - 1) / BN;
  const long long total = (long long)mt * nt * a.batch;
  const bool bias_smem = a.bias != nullptr && nt == 1;
  if (bias_smem)
    for (int c = threadIdx.x; c < BN; c += blockDim.x) sbias[c] = c < a.N ? a.bias[c] : 0.f;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&tfull[b]), 1);
      mbar_init(smem_u32(&tempty[b]), EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == EPI_WARPS) {
    // ------------------------------------------------ producer
    if (lane == 0) {
      long long g = 0;
      bool ok = true;
      for (long long t = blockIdx.x; t < total && ok; t += gridDim.x) {
        const int bz = (int)(t / ((long long)mt * nt));
        const int rem = (int)(t % ((long long)mt * nt));
        const int m0 = (rem % mt) * BM, n0 = (rem / mt) * BN;
        const int za = a.a_shared ? 0 : bz, zb = a.b_shared ? 0 : bz;
        for (int kb = 0; kb < kblocks; ++kb, ++g) {
          const int s = (int)(g % STAGES);
          if (g >= STAGES && !(ok = mbar_wait(smem_u32(&empty[s]), (uint32_t)(((g / STAGES) - 1) & 1), a.status)))
            break;
          const uint32_t fb = smem_u32(&full[s]);
          mbar_expect_tx(fb, STAGE_BYTES);
          const uint32_t sa = smem_u32(tiles + s * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
          const bool second = kb >= kb1;
          const CUtensorMap* ma = second ? &tmA2 : &tmA;
          const CUtensorMap* mb = second ? &tmB2 : &tmB;
          const int k0 = (second ? kb - kb1 : kb) * BK;
          const int amn = second ? a.a2_mn : a.a_mn, bmn = second ? a.b2_mn : a.b_mn;
          const int za2 = second ? (a.a2_shared ? 0 : bz) : za, zb2 = second ? (a.b2_shared ? 0 : bz) : zb;
          if (!amn) {
            tma_load_3d(sa, ma, k0, m0, za2, fb);
          } else {
            tma_load_3d(sa, ma, m0, k0, za2, fb);
            tma_load_3d(sa + A_BYTES / 2, ma, m0 + 64, k0, za2, fb);
          }
          if (!bmn) {
            tma_load_3d(sb, mb, k0, n0, zb2, fb);
          } else {
#pragma unroll
            for (int h = 0; h < BN / 64; ++h) tma_load_3d(sb + h * (BK * 128), mb, n0 + 64 * h, k0, zb2, fb);
          }
        }
      }
    }
  } else if (warp == EPI_WARPS + 1) {
    // ------------------------------------------------ MMA issuer
    {
      const uint32_t lead = elect_lane();
      const uint32_t idesc1 = instr_desc(BM, BN, a.a_mn, a.b_mn);
      const uint32_t idesc2 = instr_desc(BM, BN, a.a2_mn, a.b2_mn);
      long long g = 0;
      int i = 0;
      bool ok = true;
      for (long long t = blockIdx.x; t < total && ok; t += gridDim.x, ++i) {
        const int b = i & 1;
        if (i >= 2 && !(ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&tempty[b]), (uint32_t)(((i >> 1) - 1) & 1), a.status)))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t dacc = tmem + (uint32_t)(b * BN);
        for (int kb = 0; kb < kblocks; ++kb, ++g) {
          const int s = (int)(g % STAGES);
          if (!(ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&full[s]), (uint32_t)((g / STAGES) & 1), a.status)))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = smem_u32(tiles + s * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
          const bool second = kb >= kb1;
          const int amn = second ? a.a2_mn : a.a_mn, bmn = second ? a.b2_mn : a.b_mn;
          const uint32_t idesc = second ? idesc2 : idesc1;
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            // K-major: 32 bytes inside the swizzle atom; MN-major: 16 K rows of 128 bytes
            const uint64_t ad =
                amn ? smem_desc(sa + kk * 2048, a.lbo_mn, a.sbo_mn) : smem_desc(sa + kk * 32, 16, 1024);
            const uint64_t bd =
                bmn ? smem_desc(sb + kk * 2048, a.lbo_mn, a.sbo_mn) : smem_desc(sb + kk * 32, 16, 1024);
            const uint32_t acc = (kb > 0 || kk > 0) ? 1u : 0u;
            mma_bf16(lead, dacc, ad, bd, idesc, acc);
          }
          mma_commit(lead, smem_u32(&empty[s]));
        }
        if (ok)
          mma_commit(lead, smem_u32(&tfull[b]));
      }
    }
  } else {
    // ------------------------------------------------ epilogue warps 0-7
    const int lg = warp & 3;                       // TMEM lane group = 32 output rows
    const int c_begin = (warp >> 2) * (BN / 2), c_end = c_begin + BN / 2;
    int i = 0;
    float sum[GB ? BN / 2 : 1] = {};  // this thread's rows of its columns
    for (long long t = blockIdx.x; t < total; t += gridDim.x, ++i) {
      const int bz = (int)(t / ((long long)mt * nt));
      const int rem = (int)(t % ((long long)mt * nt));
      const int m0 = (rem % mt) * BM, n0 = (rem / mt) * BN;
      const int b = i & 1;
      const bool have =
          __all_sync(0xffffffffu, mbar_wait(smem_u32(&tfull[b]), (uint32_t)((i >> 1) & 1), a.status));
      if (!have) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int row = m0 + lg * 32 + lane;
      const size_t cbase = (size_t)bz * a.stride_c + (size_t)row * a.ldc;
      const size_t rbase = (size_t)bz * a.stride_r + (size_t)row * a.ldr;
      if constexpr (GB) {
#pragma unroll
        for (int g = 0; g < BN / 64; ++g) {
          const int c0 = c_begin + 32 * g;
          uint4 zv[4];
#pragma unroll
          for (int v = 0; v < 4; ++v) zv[v] = *reinterpret_cast<const uint4*>(a.z16 + cbase + c0 + 8 * v);
          uint32_t r[32];
          tmem_ld32(tmem + ((uint32_t)(lg * 32) << 16) + (uint32_t)(b * BN + c0), r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (g + 1 == BN / 64) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty[b])) : "memory");
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            float z[8];
            unpack8(zv[v], z);
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int q = 8 * v + 2 * e;
              const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[q]) * gelu_grad(z[2 * e]),
                                                             __uint_as_float(r[q + 1]) * gelu_grad(z[2 * e + 1]));
              w[e] = *reinterpret_cast<const uint32_t*>(&h);
              sum[GB ? 32 * g + q : 0] += __low2float(h);
              sum[GB ? 32 * g + q + 1 : 0] += __high2float(h);
            }
            *reinterpret_cast<uint4*>(a.c16 + cbase + c0 + 8 * v) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        continue;
      }
#pragma unroll 1
      for (int c0 = c_begin; c0 < c_end; c0 += 32) {
        uint32_t r[32];
        const uint32_t taddr = tmem + ((uint32_t)(lg * 32) << 16) + (uint32_t)(b * BN + c0);
        tmem_ld32(taddr, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 32 >= c_end) {
          // this warp's part of the accumulator has been read: release it
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty[b])) : "memory");
        }
      if (row < a.M && a.vec_ok && n0 + c0 + 32 <= a.N) {
        // 32 consecutive columns of this thread's row: 16-byte vector loads/stores
        const int col0 = n0 + c0;
        float z[32];
  #pragma unroll
        for (int q = 0; q < 32; ++q) z[q] = __uint_as_float(r[q]);
        if (a.alpha != 1.0f) {  // alpha = 1 (every surrogate product): no multiply, the same values
  #pragma unroll
          for (int q = 0; q < 32; ++q) z[q] = __fmul_rn(a.alpha, z[q]);
        }
        if (a.bias) {
          const float* bsrc = bias_smem ? sbias + c0 : a.bias + col0;
  #pragma unroll
          for (int v = 0; v < 8; ++v) {
            const float4 b = *reinterpret_cast<const float4*>(bsrc + 4 * v);
            z[4 * v] = __fadd_rn(z[4 * v], b.x);
            z[4 * v + 1] = __fadd_rn(z[4 * v + 1], b.y);
            z[4 * v + 2] = __fadd_rn(z[4 * v + 2], b.z);
            z[4 * v + 3] = __fadd_rn(z[4 * v + 3], b.w);
          }
        }
        if (a.res16) {
  #pragma unroll
          for (int v = 0; v < 4; ++v) {
            const uint4 u = *reinterpret_cast<const uint4*>(a.res16 + rbase + col0 + 8 * v);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  #pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 h2 = *reinterpret_cast<const __nv_bfloat162*>(&w[e]);
              z[8 * v + 2 * e] = __fadd_rn(z[8 * v + 2 * e], __low2float(h2));
              z[8 * v + 2 * e + 1] = __fadd_rn(z[8 * v + 2 * e + 1], __high2float(h2));
            }
          }
        }
        auto store_bf16 = [&](__nv_bfloat16* dst, const float* v32) {
  #pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint32_t w[4];
  #pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 h2 = __floats2bfloat162_rn(v32[8 * v + 2 * e], v32[8 * v + 2 * e + 1]);
              w[e] = *reinterpret_cast<const uint32_t*>(&h2);
            }
            *reinterpret_cast<uint4*>(dst + 8 * v) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        };
        if (a.pre16) store_bf16(a.pre16 + cbase + col0, z);
        if (a.act == 1) {
  #pragma unroll
          for (int q = 0; q < 32; ++q) z[q] = gelu(z[q]);
        }
        if (a.c32) {
          float* dst = a.c32 + cbase + col0;
  #pragma unroll
          for (int v = 0; v < 8; ++v) {
            float4 o = make_float4(z[4 * v], z[4 * v + 1], z[4 * v + 2], z[4 * v + 3]);
            if (a.accumulate) {
              const float4 c = *reinterpret_cast<const float4*>(dst + 4 * v);
              o.x = __fadd_rn(o.x, c.x);
              o.y = __fadd_rn(o.y, c.y);
              o.z = __fadd_rn(o.z, c.z);
              o.w = __fadd_rn(o.w, c.w);
            }
            *reinterpret_cast<float4*>(dst + 4 * v) = o;
          }
        } else {
          __nv_bfloat16* dst = a.c16 + cbase + col0;
          if (a.accumulate) {
  #pragma unroll
            for (int q = 0; q < 32; ++q) z[q] = __fadd_rn(z[q], __bfloat162float(dst[q]));
          }
          store_bf16(dst, z);
        }
      } else if (row < a.M) {
  #pragma unroll
        for (int q = 0; q < 32; ++q) {
          const int col = n0 + c0 + q;
          if (col < a.N) {
            float z = __fmul_rn(a.alpha, __uint_as_float(r[q]));
            if (a.bias) z = __fadd_rn(z, a.bias[col]);
            if (a.res16) z = __fadd_rn(z, __bfloat162float(a.res16[rbase + col]));
            if (a.pre16) a.pre16[cbase + col] = __float2bfloat16_rn(z);
            float y = a.act == 1 ? gelu(z) : z;
            if (a.c32) {
              if (a.accumulate) y = __fadd_rn(y, a.c32[cbase + col]);
              a.c32[cbase + col] = y;
            } else {
              if (a.accumulate) y = __fadd_rn(y, __bfloat162float(a.c16[cbase + col]));
              a.c16[cbase + col] = __float2bfloat16_rn(y);
            }
          }
        }
      }
      }
    }
    if constexpr (GB) {
#pragma unroll
      for (int q = 0; q < BN / 2; ++q) {
        float v = sum[GB ? q : 0];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == (q & 31)) atomicAdd(a.dsum + c_begin + q, v);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
  }
}

// ----------------------------------------------------------------- host
template <int BN, int STAGES>
size_t smem_bytes() {
  return 1024 + (size_t)STAGES * (BM * BK * 2 + BN * BK * 2) + 8 * (2 * STAGES + 6) + sizeof(float) * BN;
}

template <int BN, int STAGES, bool GB = false>
int launch_gemm_t(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& ta2, const CUtensorMap& tb2,
                  const GemmArgs& g, cudaStream_t st) {
  auto kern = k_gemm<BN, STAGES, GB>;
  const size_t smem = smem_bytes<BN, STAGES>();
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) {
    fdtd_host::note_cuda_error(e);
    return FDTD_ERR_CUDA;
  }
  int dev = 0, nsm = 0, occ = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, THREADS, smem);
  if (occ < 1) occ = 1;
  const long long tiles = (long long)((g.M + BM - 1) / BM) * ((g.N + BN - 1) / BN) * g.batch;
  const long long grid = std::min<long long>(tiles, (long long)nsm * occ);
  kern<<<(unsigned)grid, THREADS, smem, st>>>(ta, tb, ta2, tb2, g);
  return fdtd_host::check_launch();
}

int run_gemm(const fdtd_gemm_desc* d, const void* z16, float* dsum, int* status, fdtd_stream_t stream) {
  if (!d || !d->A || !d->B) return FDTD_ERR_NULL;
  if (!d->C32 == !d->C16) return FDTD_ERR_ARG;  // exactly one output
  if (d->M < 1 || d->N < 1 || d->K < 1 || d->batch < 1) return FDTD_ERR_SIZE;
  if (d->N > 65535 * 64 || d->batch > 65535) return FDTD_ERR_SIZE;
  auto al16 = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
  if (!al16(d->A) || !al16(d->B)) return FDTD_ERR_ALIGN;
  if (d->lda % 8 || d->ldb % 8 || (d->batch > 1 && (d->stride_a % 8 || d->stride_b % 8))) return FDTD_ERR_ALIGN;
  if (d->act < 0 || d->act > 1) return FDTD_ERR_ARG;
  if ((d->a_mn_major ? d->lda < d->M : d->lda < d->K) || (d->b_mn_major ? d->ldb < d->N : d->ldb < d->K))
    return FDTD_ERR_SIZE;
  int rc = FDTD_OK;
  const int BN = (d->N <= 64) ? 64 : 128;
  CUtensorMap ta, tb;
  // an operand with batch stride 0 is shared: one batch slice in its map
  const bool a_sh = d->batch == 1 || d->stride_a == 0;
  const bool b_sh = d->batch == 1 || d->stride_b == 0;
  const uint64_t sa = a_sh ? (uint64_t)d->lda * (d->a_mn_major ? d->K : d->M) : (uint64_t)d->stride_a;
  const uint64_t sb = b_sh ? (uint64_t)d->ldb * (d->b_mn_major ? d->K : d->N) : (uint64_t)d->stride_b;
  const uint64_t ba = a_sh ? 1 : (uint64_t)d->batch, bb = b_sh ? 1 : (uint64_t)d->batch;
  if (!d->a_mn_major) rc = make_map(&ta, d->A, d->K, d->M, ba, d->lda, sa, BK, BM);
  else rc = make_map(&ta, d->A, d->M, d->K, ba, d->lda, sa, 64, BK);
  if (rc) return rc;
  if (!d->b_mn_major) rc = make_map(&tb, d->B, d->K, d->N, bb, d->ldb, sb, BK, BN);
  else rc = make_map(&tb, d->B, d->N, d->K, bb, d->ldb, sb, 64, BK);
  if (rc) return rc;
  CUtensorMap ta2 = ta, tb2 = tb;
  int a2_sh = 0, b2_sh = 0;
  if (d->K2 > 0) {
    if (!d->A2 || !d->B2) return FDTD_ERR_NULL;
    if (!al16(d->A2) || !al16(d->B2)) return FDTD_ERR_ALIGN;
    if (d->lda2 % 8 || d->ldb2 % 8 || (d->batch > 1 && (d->stride_a2 % 8 || d->stride_b2 % 8))) return FDTD_ERR_ALIGN;
    if ((d->a2_mn_major ? d->lda2 < d->M : d->lda2 < d->K2) || (d->b2_mn_major ? d->ldb2 < d->N : d->ldb2 < d->K2))
      return FDTD_ERR_SIZE;
    a2_sh = (d->batch == 1 || d->stride_a2 == 0);
    b2_sh = (d->batch == 1 || d->stride_b2 == 0);
    const uint64_t sa2 = a2_sh ? (uint64_t)d->lda2 * (d->a2_mn_major ? d->K2 : d->M) : (uint64_t)d->stride_a2;
    const uint64_t sb2 = b2_sh ? (uint64_t)d->ldb2 * (d->b2_mn_major ? d->K2 : d->N) : (uint64_t)d->stride_b2;
    const uint64_t ba2 = a2_sh ? 1 : (uint64_t)d->batch, bb2 = b2_sh ? 1 : (uint64_t)d->batch;
    if (!d->a2_mn_major) rc = make_map(&ta2, d->A2, d->K2, d->M, ba2, d->lda2, sa2, BK, BM);
    else rc = make_map(&ta2, d->A2, d->M, d->K2, ba2, d->lda2, sa2, 64, BK);
    if (rc) return rc;
    if (!d->b2_mn_major) rc = make_map(&tb2, d->B2, d->K2, d->N, bb2, d->ldb2, sb2, BK, BN);
    else rc = make_map(&tb2, d->B2, d->N, d->K2, bb2, d->ldb2, sb2, 64, BK);
    if (rc) return rc;
  }
  GemmArgs g{};
  g.K2 = d->K2 > 0 ? d->K2 : 0;
  g.a2_mn = d->a2_mn_major;
  g.b2_mn = d->b2_mn_major;
  g.a2_shared = a2_sh;
  g.b2_shared = b2_sh;
  g.M = d->M;
  g.N = d->N;
  g.K = d->K;
  g.batch = d->batch;
  g.a_mn = d->a_mn_major;
  g.b_mn = d->b_mn_major;
  g.c32 = d->C32;
  g.c16 = reinterpret_cast<__nv_bfloat16*>(d->C16);
  g.ldc = d->ldc;
  g.stride_c = d->stride_c;
  g.bias = d->bias;
  g.res16 = reinterpret_cast<const __nv_bfloat16*>(d->res16);
  g.ldr = d->ldr;
  g.stride_r = d->stride_r;
  g.alpha = d->alpha;
  g.act = d->act;
  g.accumulate = d->accumulate;
  g.pre16 = reinterpret_cast<__nv_bfloat16*>(d->pre16);
  g.lbo_mn = d->mn_lbo ? (unsigned)d->mn_lbo : (unsigned)(BK * 128);
  g.sbo_mn = d->mn_sbo ? (unsigned)d->mn_sbo : 1024u;
  {
    const void* cptr = d->C32 ? (const void*)d->C32 : d->C16;
    bool v = al16(cptr) && d->ldc % 8 == 0 && d->stride_c % 8 == 0;
    if (d->bias) v = v && al16(d->bias);
    if (d->res16) v = v && al16(d->res16) && d->ldr % 8 == 0 && d->stride_r % 8 == 0;
    if (d->pre16) v = v && al16(d->pre16);
    g.vec_ok = v ? 1 : 0;
  }
  g.z16 = reinterpret_cast<const __nv_bfloat16*>(z16);
  g.dsum = dsum;
  g.a_shared = a_sh ? 1 : 0;
  g.b_shared = b_sh ? 1 : 0;
  g.status = status;
  // 4 pipeline stages throughout: with 2, a product of only one or two
  // k-blocks per tile (K = 16 + 64 in the folded first layer) cannot load the
  // next tile while the current one computes (1.6 ms instead of 0.9 at 4096)
  cudaStream_t st = (cudaStream_t)stream;
  if (z16) return launch_gemm_t<128, 4, true>(ta, tb, ta2, tb2, g, st);
  if (BN == 64) return launch_gemm_t<64, 4>(ta, tb, ta2, tb2, g, st);
  return launch_gemm_t<128, 4>(ta, tb, ta2, tb2, g, st);
}

}  // namespace
}  // namespace fdtd

extern "C" int fdtd_gemm_bf16(const fdtd_gemm_desc* d, int* status, fdtd_stream_t stream) {
  return fdtd::run_gemm(d, nullptr, nullptr, status, stream);
}

extern "C" int fdtd_gemm_bf16_gelu_bwd(const fdtd_gemm_desc* d, const void* z, float* dsum, int* status,
                                       fdtd_stream_t stream) {
  if (!d || !z || !dsum || !d->C16) return FDTD_ERR_NULL;
  if (d->M % fdtd::BM || d->N != 128) return FDTD_ERR_SIZE;
  if (d->bias || d->res16 || d->pre16 || d->act || d->accumulate || d->alpha != 1.0f) return FDTD_ERR_ARG;
  if (((uintptr_t)d->C16 | (uintptr_t)z) & 15u || d->ldc % 8 || d->stride_c % 8) return FDTD_ERR_ALIGN;
  return fdtd::run_gemm(d, z, dsum, status, stream);
}
