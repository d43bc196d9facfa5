// Blockwise FP8 (e4m3) support for sm_100a:
//   * weight quantiser: one fp32 scale per 128x128 tile (amax/448), stored as its reciprocal
//     ("dequant scale"), a pure function of the tile so that quantising a rank's rows locally
//     equals quantising after a bf16 gather bit for bit;
//   * activation quantiser: one scale per (row, 128-column group), written k-block major;
//   * block-scaled GEMM: tcgen05.mma kind::f8f6f4 accumulates one 128-deep K block at a time in
//     TMEM; the epilogue warps fold each block into fp32 registers with its (row, k-block) x
//     (n-block, k-block) scale while the tensor core already works on the next block.
//
//   D[M,N] (bf16) = sum_kb sa[kb][m] * sb(n/128, kb) * (Aq[m, kb] . Bq[n, kb]^T)
//
// A is K-major e4m3 [M, K]. B is e4m3, either K-major [N, K] (forward: B = W) or MN-major
// [K, N] (dgrad: B = W read as its transpose), with the weight's 128x128 scales indexed through
// two strides.
#include "common.cuh"
#include <cuda_fp8.h>

namespace {
using namespace fsb;

struct alignas(16) bf16x8 { __nv_bfloat162 v[4]; };

// ------------------------------------------------------------------ weight quantiser (128x128 tiles)
// grid = (ceil(cols/128), ceil(rows/128)); 256 threads; each thread owns 8 columns x 8 rows.
__global__ void __launch_bounds__(256)
quant_weight_128x128_kernel(const __nv_bfloat16* __restrict__ w, uint8_t* __restrict__ q,
                            float* __restrict__ inv_scale, int rows, int cols, long long ldw,
                            long long ldq, int scale_cols) {
  __shared__ float red[8];
  const int tr = blockIdx.y * 128, tc = blockIdx.x * 128;
  const int cg = threadIdx.x & 15;   // 16 column groups of 8
  const int rg = threadIdx.x >> 4;   // 16 row groups of 8
  const int c0 = tc + cg * 8;
  float vals[8][8];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = tr + rg * 8 + i;
    if (r < rows && c0 + 8 <= cols) {
      const bf16x8 t = *reinterpret_cast<const bf16x8*>(w + r * ldw + c0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(t.v[j]);
        vals[i][2 * j] = f.x;
        vals[i][2 * j + 1] = f.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        vals[i][j] = (r < rows && c0 + j < cols) ? __bfloat162float(w[r * ldw + c0 + j]) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(vals[i][j]));
  }
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
  amax = fmaxf(amax, 1e-12f);
  const float scale = 448.f / amax;
  if (threadIdx.x == 0) inv_scale[blockIdx.y * scale_cols + blockIdx.x] = 1.f / scale;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = tr + rg * 8 + i;
    if (r >= rows) continue;
    alignas(8) uint8_t o[8];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const float2 f = make_float2(fminf(fmaxf(vals[i][j] * scale, -448.f), 448.f),
                                   fminf(fmaxf(vals[i][j + 1] * scale, -448.f), 448.f));
      *reinterpret_cast<uint16_t*>(o + j) = __nv_cvt_float2_to_fp8x2(f, __NV_SATFINITE, __NV_E4M3);
    }
    if (c0 + 8 <= cols) {
      *reinterpret_cast<uint2*>(q + r * ldq + c0) = *reinterpret_cast<const uint2*>(o);
    } else {
      for (int j = 0; j < 8 && c0 + j < cols; ++j) q[r * ldq + c0 + j] = o[j];
    }
  }
}

// ------------------------------------------------------------------ activation quantiser (1x128 groups)
// Eight threads per (row, 128-column group), 16 columns each: a 32-byte read and a 16-byte write per thread, which keeps
// enough bytes in flight to be bound by memory (3 bytes an element; a warp per group, 8 bytes a thread, ran at 2.2 TB/s).
// inv_scale is written [K/128, T] (k-block major).
__global__ void __launch_bounds__(256)
quant_act_1x128_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ inv_scale,
                       long long T, int K, long long ldx, long long ldq, int vec) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const int units = K / 16;                       // threads of a row: a multiple of 8, as is the block size
  const long long row = i / units;
  const int u = static_cast<int>(i - row * units);
  if (row >= T) return;                           // all eight threads of a group leave together
  const __nv_bfloat16* p = x + row * ldx + u * 16;
  alignas(16) __nv_bfloat162 raw[8];
  if (vec) {
    reinterpret_cast<uint4*>(raw)[0] = reinterpret_cast<const uint4*>(p)[0];
    reinterpret_cast<uint4*>(raw)[1] = reinterpret_cast<const uint4*>(p)[1];
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) reinterpret_cast<uint2*>(raw)[j] = reinterpret_cast<const uint2*>(p)[j];
  }
  float2 f[8];
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    f[j] = __bfloat1622float2(raw[j]);
    amax = fmaxf(amax, fmaxf(fabsf(f[j].x), fabsf(f[j].y)));
  }
  const unsigned group = 0xffu << (threadIdx.x & 24);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(group, amax, o));
  amax = fmaxf(amax, 1e-12f);
  const float scale = 448.f / amax;
  if ((u & 7) == 0) inv_scale[static_cast<long long>(u >> 3) * T + row] = 1.f / scale;
  alignas(16) uint16_t o[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = __nv_cvt_float2_to_fp8x2(make_float2(f[j].x * scale, f[j].y * scale), __NV_SATFINITE, __NV_E4M3);
  uint8_t* d = q + row * ldq + u * 16;
  if (vec) {
    *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(o);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) reinterpret_cast<uint32_t*>(d)[j] = reinterpret_cast<const uint32_t*>(o)[j];
  }
}

// ------------------------------------------------------------------ block-scaled GEMM
constexpr int BM = 128, BN = 128, BK = 128;  // BK bytes == elements (fp8)
constexpr int STAGES = 6;
constexpr int BUFS = 4;                      // block products in TMEM: 4 x 128 columns
constexpr int A_STAGE = BM * BK, B_STAGE = BN * BK, STAGE_BYTES = A_STAGE + B_STAGE;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int NUM_THREADS = 320;  // warp 0 TMA, warp 1 MMA, warps 2..9 scale-accumulate (two per lane quarter)

// Every 128-deep block is a product of its own, whose 128 x 128 fp32 values leave TMEM and are folded into registers with
// the block's scales: bound by that chain (wait, TMEM read, FMA) per block and warp, not by a unit (ncu, when it read and
// folded in turn from two buffers: tensor pipe 31 %, L2 37 %, issue slots 35 %). So the read of the next 32 columns, or
// of the next block, is in flight while 32 columns are folded with two-element FMAs, and four buffers keep the tensor core
// ahead.
struct Fp8Args {
  int M, N, K;
  int b_mn;
  const float* sa;            // [K/128][M]
  const float* sb;            // weight scales, addressed sb[nb * sb_stride_n + kb * sb_stride_k]
  long long sb_stride_n, sb_stride_k;
  __nv_bfloat16* d;
  long long ldd;
  int* status;
};

// acc (two fp32) = v * s + acc, one instruction for both
__device__ __forceinline__ void fma2(unsigned long long& acc, uint32_t v0, uint32_t v1, unsigned long long s2) {
  asm("{\n\t.reg .b64 v;\n\tmov.b64 v, {%1, %2};\n\tfma.rn.f32x2 %0, v, %3, %0;\n\t}" : "+l"(acc) : "r"(v0), "r"(v1), "l"(s2));
}

__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const Fp8Args args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tmem_full = bars + 2 * STAGES;          // [BUFS]
  uint64_t* tmem_empty = bars + 2 * STAGES + BUFS;  // [BUFS]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 2 * BUFS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (args.M + BM - 1) / BM, tiles_n = (args.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int num_kb = args.K / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < BUFS; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 8);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BUFS * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&map_a);
      tma_prefetch_desc(&map_b);
      uint32_t it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        int tm, tn;
        grouped_tile_coords(tile, tiles_m, tiles_n, tm, tn);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&empty_bar[s], ph ^ 1, abort_flag)) {
            atomicExch(args.status, FSB_ERR_WAIT_TIMEOUT_EMPTY);
            *abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t* sa = smem + s * STAGE_BYTES;
          uint8_t* sb = sa + A_STAGE;
          mbar_expect_tx(&full_bar[s], STAGE_BYTES);
          tma_load_2d(sa, &map_a, &full_bar[s], kb * BK, tm * BM);
          if (!args.b_mn) tma_load_2d(sb, &map_b, &full_bar[s], kb * BK, tn * BN);
          else tma_load_2d(sb, &map_b, &full_bar[s], tn * BN, kb * BK);  // [K rows][128 N bytes]
        }
      }
    }
  } else if (warp == 1) {
    // The whole warp walks the loop (waits and descriptor arithmetic stay warp-uniform); one elected
    // lane issues the tcgen05 instructions.
    {
      // e4m3 x e4m3 -> fp32; B MN-major for the transposed-weight product
      const uint32_t idesc = make_idesc(BM, BN, 0, 0, 0, args.b_mn ? 1u : 0u);
      // K-major: 32 elements (bytes) per MMA inside the 128-byte row. MN-major B: one 128-wide
      // N group, 8-deep K groups 1 KB apart, 32 K = 4 groups = 4 KB per MMA.
      const uint32_t b_kstep = (args.b_mn ? 4096u : 32u) >> 4;
      uint32_t it = 0, blk = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        for (int kb = 0; kb < num_kb; ++kb, ++it, ++blk) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          const uint32_t buf = blk % BUFS, bph = (blk / BUFS) & 1;
          if (!mbar_wait(&full_bar[s], ph, abort_flag) || !mbar_wait(&tmem_empty[buf], bph ^ 1, abort_flag)) {
            if (lane == 0) {
              atomicExch(args.status, FSB_ERR_WAIT_TIMEOUT_FULL);
              *abort_flag = 1;
            }
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * STAGE_BYTES);
          const uint64_t da = make_smem_desc_sw128(sa, 16, 1024);
          const uint64_t db = make_smem_desc_sw128(sa + A_STAGE, 16, 1024);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / 32; ++k)
              umma_f8(tmem_base + buf * BN, da + k * 2, db + k * b_kstep, idesc, k != 0);
            umma_commit(&empty_bar[s]);
            umma_commit(&tmem_full[buf]);
          }
          __syncwarp();
        }
      }
    }
  } else {
    // Two warps per TMEM lane quarter, each folding 64 of the tile's 128 columns.
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    constexpr int HC = BN / 2;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * HC;
    uint32_t blk = 0;
    bool ok = true;
    auto wait_full = [&](uint32_t b) {
      if (mbar_wait_warp(&tmem_full[b % BUFS], (b / BUFS) & 1, abort_flag)) {
        tc_fence_after();
        return true;
      }
      if (lane == 0) {
        atomicExch(args.status, FSB_ERR_WAIT_TIMEOUT_TMEM_FULL);
        *abort_flag = 1;
      }
      return false;
    };
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      int tm, tn;
      grouped_tile_coords(tile, tiles_m, tiles_n, tm, tn);
      const int row = tm * BM + quarter * 32 + lane;
      const bool row_ok = row < args.M;
      unsigned long long acc2[HC / 2];
#pragma unroll
      for (int i = 0; i < HC / 2; ++i) acc2[i] = 0ull;
      // the scales of a block are loaded one block ahead: their latency is longer than a block
      const float* pa = args.sa + (row_ok ? row : 0);
      const float* pb = args.sb + tn * args.sb_stride_n;
      float next_a = row_ok ? *pa : 0.f, next_b = *pb;
      uint32_t v0[32], v1[32];
      ok = wait_full(blk);
      if (ok) tmem_ld_32x32(t_row + (blk % BUFS) * BN, v0);
      for (int kb = 0; kb < num_kb && ok; ++kb, ++blk) {
        const uint32_t buf = blk % BUFS;
        const float s = next_a * next_b;
        if (kb + 1 < num_kb) {
          pa += args.M;
          pb += args.sb_stride_k;
          next_a = row_ok ? *pa : 0.f;
          next_b = *pb;
        }
        unsigned long long s2;
        asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
        tmem_ld_wait_for(v0);
        tmem_ld_32x32(t_row + buf * BN + 32, v1);
#pragma unroll
        for (int i = 0; i < 16; ++i) fma2(acc2[i], v0[2 * i], v0[2 * i + 1], s2);
        tmem_ld_wait_for(v1);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[buf]);  // the block is in registers
        if (kb + 1 < num_kb) {
          ok = wait_full(blk + 1);
          if (ok) tmem_ld_32x32(t_row + ((blk + 1) % BUFS) * BN, v0);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) fma2(acc2[16 + i], v1[2 * i], v1[2 * i + 1], s2);
      }
      if (!ok) tmem_ld_wait();   // nothing may be in flight when TMEM is given back
      float acc[HC];
#pragma unroll
      for (int i = 0; i < HC / 2; ++i) asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[2 * i]), "=f"(acc[2 * i + 1]) : "l"(acc2[i]));
      if (ok && row_ok) {
        const int cbase = tn * BN + half * HC;
        __nv_bfloat16* dp = args.d + static_cast<long long>(row) * args.ldd + cbase;
        const int ncols = min(HC, args.N - cbase);
        if (ncols == HC && (args.ldd % 8) == 0) {
#pragma unroll
          for (int i = 0; i < HC; i += 8) {
            uint4 o;
            o.x = pack_bf16x2(acc[i], acc[i + 1]);
            o.y = pack_bf16x2(acc[i + 2], acc[i + 3]);
            o.z = pack_bf16x2(acc[i + 4], acc[i + 5]);
            o.w = pack_bf16x2(acc[i + 6], acc[i + 7]);
            *reinterpret_cast<uint4*>(dp + i) = o;
          }
        } else {
#pragma unroll
          for (int i = 0; i < HC; ++i)
            if (i < ncols) dp[i] = __float2bfloat16(acc[i]);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*abort_flag) {
      const unsigned long long t0 = clock64();
      while (clock64() - t0 < 2000000ull) {
      }
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, BUFS * BN);
  }
}

int g_sms[64] = {0};
}  // namespace

// w: bf16 [rows, cols] (row stride ldw); q: e4m3 bytes [rows, cols] (row stride ldq);
// inv_scale: fp32 [ceil(rows/128), ceil(cols/128)].
FSB_API int fsb_fp8_quant_weight(const void* w, void* q, float* inv_scale, int rows, int cols, long long ldw,
                                 long long ldq, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return FSB_OK;
  dim3 grid((cols + 127) / 128, (rows + 127) / 128);
  quant_weight_128x128_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(w),
                                                        static_cast<uint8_t*>(q), inv_scale, rows, cols, ldw,
                                                        ldq, (cols + 127) / 128);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}

// x: bf16 [T, K] with K % 128 == 0; q: e4m3 [T, K]; inv_scale: fp32 [K/128, T].
FSB_API int fsb_fp8_quant_act(const void* x, void* q, float* inv_scale, long long T, int K, long long ldx,
                              long long ldq, cudaStream_t stream) {
  if (K % 128 != 0 || ldx % 4 != 0 || ldq % 4 != 0) return FSB_ERR_BAD_ARG;
  if (T <= 0) return FSB_OK;
  const long long blocks = (T * (K / 16) + 255) / 256;
  const int vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(q)) & 15) == 0 && ldx % 8 == 0 && ldq % 16 == 0;
  quant_act_1x128_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q), inv_scale, T, K, ldx, ldq, vec);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}

// D[M,N] bf16 = block-scaled Aq . Bq^T. K % 128 == 0. b_mn: B stored [K, N] (N contiguous).
FSB_API int fsb_gemm_fp8(const void* aq, const float* sa, const void* bq, const float* sb,
                         long long sb_stride_n, long long sb_stride_k, void* d, int M, int N, int K,
                         long long lda, long long ldb, long long ldd, int b_mn, int* status,
                         cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || K % BK != 0) return FSB_ERR_BAD_ARG;
  if (b_mn && N % 16 != 0) return FSB_ERR_BAD_ARG;
  CUtensorMap map_a, map_b;
  int rc = fsb_make_tmap_2d(&map_a, aq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, M, K, lda, BM, BK);
  if (rc != FSB_OK) return rc;
  if (!b_mn) rc = fsb_make_tmap_2d(&map_b, bq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K, ldb, BN, BK);
  else rc = fsb_make_tmap_2d(&map_b, bq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K, N, ldb, BK, BN);
  if (rc != FSB_OK) return rc;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return FSB_ERR_BAD_ARG;
  if (g_sms[dev] == 0) {
    if (cudaFuncSetAttribute(gemm_fp8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) !=
        cudaSuccess)
      return FSB_ERR_LAUNCH;
    cudaDeviceGetAttribute(&g_sms[dev], cudaDevAttrMultiProcessorCount, dev);
  }
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  const int grid = tiles < g_sms[dev] ? tiles : g_sms[dev];
  Fp8Args a;
  a.M = M; a.N = N; a.K = K; a.b_mn = b_mn;
  a.sa = sa; a.sb = sb; a.sb_stride_n = sb_stride_n; a.sb_stride_k = sb_stride_k;
  a.d = static_cast<__nv_bfloat16*>(d); a.ldd = ldd; a.status = status;
  gemm_fp8_kernel<<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(map_a, map_b, a);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}
