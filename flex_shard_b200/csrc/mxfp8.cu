// MXFP8 (e4m3 data, one power-of-two e8m0 scale per 32 elements) for sm_100a:
//   * weight quantiser: one scale per 32x32 tile, so the same data serves a product that contracts
//     over the columns (forward) and one that contracts over the rows (input gradient); the tile
//     exponents are expanded into one scale tensor per orientation;
//   * activation quantiser: one scale per (row, 32-column group);
//   * block-scaled GEMM: tcgen05.mma kind::mxf8f6f4.block_scale. The tensor core applies the
//     scales itself: they sit in TMEM next to the accumulators, copied there from shared memory
//     with tcgen05.cp by the MMA-issuing thread right before the four 32-deep MMAs of a stage.
//
// Scale exponent ("round up" rule): the smallest power of two s with amax / s <= 448, stored as
// the biased byte e = log2(s) + 127 (0 when the group is all zeros); q = round_to_e4m3(x / s).
//
// Scale tensors use the tensor core's block layout: rows in blocks of 128, 32-element groups in
// blocks of 4; block (rb, gb) is 512 contiguous bytes at ((rb * n_gb + gb) * 512) with the byte of
// (row r, group g) at (r % 32) * 16 + (r / 32) * 4 + g. One block is exactly what one 128-row
// operand tile needs for one 128-deep stage, so a stage's scales arrive with one 512-byte bulk copy.
#include "common.cuh"
#include <cuda_fp8.h>

namespace {
using namespace fsb;

struct alignas(16) bf16x8 { __nv_bfloat162 v[4]; };

// biased exponent of the smallest power of two >= amax / 448
__device__ __forceinline__ uint32_t e8m0_round_up(float amax) {
  const float v = amax * (1.f / 448.f);
  const uint32_t bits = __float_as_uint(v);
  uint32_t e = (bits >> 23) & 0xffu;
  if ((bits & 0x7fffffu) != 0 && e < 254u) e += 1;
  return amax > 0.f ? (e > 254u ? 254u : e) : 0u;
}
__device__ __forceinline__ float e8m0_inv(uint32_t e) {   // 2^(127 - e), finite for every e in [0, 254]
  return __uint_as_float(e == 254u ? 0x00400000u : ((254u - e) << 23));
}
__device__ __forceinline__ long long blocked_offset(long long r, int g, int n_gb) {
  return ((r >> 7) * n_gb + (g >> 2)) * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4 + (g & 3);
}

// Four bf16 pairs, scaled by a power of two, as eight e4m3 bytes.
__device__ __forceinline__ uint2 quant8(const uint4& raw, float inv) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
  uint2 o;
  uint16_t* w = reinterpret_cast<uint16_t*>(&o);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __bfloat1622float2(h[j]);
    w[j] = __nv_cvt_float2_to_fp8x2(make_float2(f.x * inv, f.y * inv), __NV_SATFINITE, __NV_E4M3);
  }
  return o;
}
__device__ __forceinline__ float amax8(const uint4& raw, float m) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __bfloat1622float2(h[j]);
    m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
  }
  return m;
}

// ------------------------------------------------------------------ weight quantiser (32x32 tiles)
// A warp per tile: lane l holds 8 columns of rows l/4, l/4 + 8, l/4 + 16, l/4 + 24, four 16-byte reads in flight. The four
// warps of a block take neighbouring tiles. vec == 0 (a row stride or pointer off the 16-byte grid): element by element.
// Bound by memory, 3 bytes an element; with element-wise accesses everywhere 218 M weights took 0.63 ms (1.0 TB/s).
__global__ void __launch_bounds__(128)
mx_quant_weight_kernel(const __nv_bfloat16* __restrict__ w, uint8_t* __restrict__ q, uint8_t* __restrict__ tile_exp,
                       int rows, int cols, long long ldw, long long ldq, int exp_cols, int vec) {
  const int tile = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (tile >= exp_cols) return;
  const int r0 = blockIdx.y * 32 + (lane >> 2), c0 = tile * 32 + (lane & 3) * 8;
  const bool wide = vec && c0 + 8 <= cols;
  uint4 v[4];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + 8 * i;
    v[i] = make_uint4(0, 0, 0, 0);
    if (r < rows) {
      const __nv_bfloat16* p = w + r * ldw + c0;
      if (wide) {
        v[i] = *reinterpret_cast<const uint4*>(p);
      } else {
        uint32_t h[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (c0 + j < cols) h[j >> 1] |= static_cast<uint32_t>(__bfloat16_as_ushort(p[j])) << (16 * (j & 1));
        v[i] = make_uint4(h[0], h[1], h[2], h[3]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) amax = amax8(v[i], amax);
  amax = warp_max(amax);
  const uint32_t e = e8m0_round_up(amax);
  if (lane == 0) tile_exp[blockIdx.y * exp_cols + tile] = static_cast<uint8_t>(e);
  const float inv = e8m0_inv(e);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + 8 * i;
    if (r >= rows) continue;
    const uint2 o = quant8(v[i], inv);
    uint8_t* d = q + r * ldq + c0;
    if (wide) {
      *reinterpret_cast<uint2*>(d) = o;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c0 + j < cols) d[j] = static_cast<uint8_t>((j < 4 ? o.x : o.y) >> (8 * (j & 3)));
    }
  }
}

// Tile exponents [ceil(rows/32), ceil(cols/32)] -> blocked scales for the operand [rows, cols]
// (transpose == 0: groups run along the columns) or for its transpose [cols, rows] (groups run
// along the rows). Padding rows / groups get exponent 127 (scale 1).
__global__ void mx_expand_scales_kernel(const uint8_t* __restrict__ tile_exp, uint8_t* __restrict__ out, int op_rows,
                                        int op_groups, int pad_rows, int pad_groups, int exp_cols, int transpose) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const long long total = static_cast<long long>(pad_rows) * pad_groups;
  if (i >= total) return;
  const long long r = i / pad_groups;
  const int g = static_cast<int>(i % pad_groups);
  uint8_t e = 127;
  if (r < op_rows && g < op_groups)
    e = transpose ? tile_exp[static_cast<long long>(g) * exp_cols + (r >> 5)] : tile_exp[(r >> 5) * exp_cols + g];
  out[blocked_offset(r, g, pad_groups >> 2)] = e;
}

// ------------------------------------------------------------------ activation quantiser (1x32 groups)
// Four threads per (row, 32-column group), 8 columns each, two rows' worth of units per thread in flight: bound by memory.
__global__ void __launch_bounds__(256)
mx_quant_act_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, uint8_t* __restrict__ scales, long long T,
                    int K, long long ldx, long long ldq, int n_gb, int vec) {
  const int units = K / 8;                            // threads of a row, a multiple of 16
  const long long total = T * units;
  const long long half = (total / 4 + 1) / 2 * 4;     // a thread takes units i and i + half; half is a multiple of 4
  const long long i0 = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i0 >= half) return;                             // the four threads of a group leave together
  uint4 v[2];
  long long row[2];
  int u[2];
  bool live[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const long long i = i0 + j * half;
    live[j] = i < total;
    row[j] = live[j] ? i / units : 0;
    u[j] = live[j] ? static_cast<int>(i - row[j] * units) : 0;
    const __nv_bfloat16* p = x + row[j] * ldx + u[j] * 8;
    if (vec) v[j] = *reinterpret_cast<const uint4*>(p);
    else {
      const uint2 a = reinterpret_cast<const uint2*>(p)[0], b = reinterpret_cast<const uint2*>(p)[1];
      v[j] = make_uint4(a.x, a.y, b.x, b.y);
    }
  }
  const unsigned group = 0xfu << (threadIdx.x & 28);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    float amax = amax8(v[j], 0.f);
    amax = fmaxf(amax, __shfl_xor_sync(group, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(group, amax, 1));
    if (!live[j]) continue;
    const uint32_t e = e8m0_round_up(amax);
    if ((u[j] & 3) == 0) scales[blocked_offset(row[j], u[j] >> 2, n_gb)] = static_cast<uint8_t>(e);
    const uint2 o = quant8(v[j], e8m0_inv(e));
    uint8_t* d = q + row[j] * ldq + u[j] * 8;
    if (vec) *reinterpret_cast<uint2*>(d) = o;
    else {
      reinterpret_cast<uint32_t*>(d)[0] = o.x;
      reinterpret_cast<uint32_t*>(d)[1] = o.y;
    }
  }
}

// ------------------------------------------------------------------ transposed-use quantiser (32x1 groups)
// For products that contract over the rows of x (weight gradients): one scale per (32-row group, column). The data keeps
// its row-major layout; the scales are those of the operand x^T, i.e. blocked with "rows" = columns of x and groups =
// 32-row groups of x. A warp takes 128 columns of a row group, lane l columns 4 l to 4 l + 3: 256-byte rows in, 128-byte
// rows out, 32 rows in flight (a column per thread moved 64 bytes per warp and row and reached 1.9 TB/s).
__global__ void __launch_bounds__(128)
mx_quant_rows_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, uint8_t* __restrict__ scales, int K,
                     long long ldx, long long ldq, int n_gb, int vec) {
  const int span = blockIdx.x * 4 + (threadIdx.x >> 5);       // 128-column span
  if (span * 128 >= K) return;
  const int col = span * 128 + (threadIdx.x & 31) * 4;
  const long long r0 = static_cast<long long>(blockIdx.y) * 32;
  const __nv_bfloat16* p = x + r0 * ldx + col;
  uint2 v[32];
  if (vec) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = *reinterpret_cast<const uint2*>(p + i * ldx);
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const unsigned short* h = reinterpret_cast<const unsigned short*>(p + i * ldx);
      v[i] = make_uint2(h[0] | static_cast<uint32_t>(h[1]) << 16, h[2] | static_cast<uint32_t>(h[3]) << 16);
    }
  }
  float amax[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[i]);
    const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
    amax[0] = fmaxf(amax[0], fabsf(a.x));
    amax[1] = fmaxf(amax[1], fabsf(a.y));
    amax[2] = fmaxf(amax[2], fabsf(b.x));
    amax[3] = fmaxf(amax[3], fabsf(b.y));
  }
  float inv[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t e = e8m0_round_up(amax[j]);
    inv[j] = e8m0_inv(e);
    scales[blocked_offset(col + j, static_cast<int>(blockIdx.y), n_gb)] = static_cast<uint8_t>(e);
  }
  uint8_t* d = q + r0 * ldq + col;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[i]);
    const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a.x * inv[0], a.y * inv[1]), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(b.x * inv[2], b.y * inv[3]), __NV_SATFINITE, __NV_E4M3);
    const uint32_t o = lo | hi << 16;
    if (vec) *reinterpret_cast<uint32_t*>(d + i * ldq) = o;
    else {
#pragma unroll
      for (int j = 0; j < 4; ++j) d[i * ldq + j] = static_cast<uint8_t>(o >> (8 * j));
    }
  }
}

// ------------------------------------------------------------------ block-scaled GEMM
constexpr int BM = 128, BN = 128, BK = 128;  // BK bytes == elements (fp8)
constexpr int STAGES = 6;
constexpr int A_STAGE = BM * BK, B_STAGE = BN * BK, SF_BYTES = 512;
constexpr int STAGE_BYTES = A_STAGE + B_STAGE + 2 * SF_BYTES;   // 33 KB
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int NUM_THREADS = 192;   // warp 0 TMA, warp 1 MMA, warps 2..5 epilogue
constexpr int TMEM_COLS = 512;     // two 128-column accumulators + two sets of (4 + 4) scale columns
constexpr int SF_COL0 = 256;

struct MxArgs {
  int M, N, K;
  int a_mn, b_mn;
  const uint8_t* sfa;   // blocked scales of A: [ceil(M/128)][K/128][512]
  const uint8_t* sfb;   // blocked scales of B: [ceil(N/128)][K/128][512]
  void* d;
  long long ldd;
  int d_fp32;
  int* status;
};

__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// 32 rows x 16 bytes of shared memory -> 4 TMEM columns, repeated in all four lane quarters
__device__ __forceinline__ void tmem_cp_32x128b_x4(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
// Unswizzled K-major descriptor: 8-row groups of 16-byte rows are 128 bytes apart.
__device__ __forceinline__ uint64_t make_sf_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr >> 4) & 0x3FFF);
  d |= static_cast<uint64_t>(128 >> 4) << 32;   // SBO
  d |= 1ull << 46;
  return d;
}
__device__ __forceinline__ void umma_mxf8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                          uint32_t tsfa, uint32_t tsfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tsfa), "r"(tsfb)
      : "memory");
}
// e4m3 x e4m3, e8m0 scales; sf_id selects which of a scale word's four bytes (which 32-deep group
// of the stage) this MMA uses.
__device__ __forceinline__ uint32_t make_idesc_mx(uint32_t m, uint32_t n, uint32_t a_mn, uint32_t b_mn, uint32_t sf_id) {
  return (sf_id << 4) | (a_mn << 15) | (b_mn << 16) | ((n >> 3) << 17) | (1u << 23) | ((m >> 4) << 24) | (sf_id << 29);
}

__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_mxfp8_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const MxArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tmem_full = bars + 2 * STAGES;       // [2]
  uint64_t* tmem_empty = bars + 2 * STAGES + 2;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
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
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
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
        const int tm = tile % tiles_m, tn = tile / tiles_m;
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
          uint8_t* ssf = sb + B_STAGE;
          mbar_expect_tx(&full_bar[s], STAGE_BYTES);
          if (!args.a_mn) tma_load_2d(sa, &map_a, &full_bar[s], kb * BK, tm * BM);
          else tma_load_2d(sa, &map_a, &full_bar[s], tm * BM, kb * BK);  // [K rows][128 M bytes]
          if (!args.b_mn) tma_load_2d(sb, &map_b, &full_bar[s], kb * BK, tn * BN);
          else tma_load_2d(sb, &map_b, &full_bar[s], tn * BN, kb * BK);  // [K rows][128 N bytes]
          bulk_load_1d(ssf, args.sfa + (static_cast<long long>(tm) * num_kb + kb) * SF_BYTES, SF_BYTES, &full_bar[s]);
          bulk_load_1d(ssf + SF_BYTES, args.sfb + (static_cast<long long>(tn) * num_kb + kb) * SF_BYTES, SF_BYTES,
                       &full_bar[s]);
        }
      }
    }
  } else if (warp == 1) {
    // The whole warp walks the loop; one elected lane issues the tcgen05 instructions.
    // K-major: 32 elements (bytes) per MMA inside the 128-byte row. MN-major B: one 128-wide
    // N group, 8-deep K groups 1 KB apart, 32 K = 4 groups = 4 KB per MMA.
    const uint32_t a_kstep = (args.a_mn ? 4096u : 32u) >> 4, b_kstep = (args.b_mn ? 4096u : 32u) >> 4;
    const uint32_t a_mn = args.a_mn ? 1u : 0u, b_mn = args.b_mn ? 1u : 0u;
    uint32_t it = 0, local_tile = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      const uint32_t acc = local_tile & 1;
      const uint32_t acc_ph = (local_tile >> 1) & 1;
      ++local_tile;
      if (!mbar_wait(&tmem_empty[acc], acc_ph ^ 1, abort_flag)) {
        if (lane == 0) {
          atomicExch(args.status, FSB_ERR_WAIT_TIMEOUT_TMEM_EMPTY);
          *abort_flag = 1;
        }
        break;
      }
      tc_fence_after();
      for (int kb = 0; kb < num_kb; ++kb, ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!mbar_wait(&full_bar[s], ph, abort_flag)) {
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
        const uint32_t ssf = sa + A_STAGE + B_STAGE;
        const uint32_t tsfa = tmem_base + SF_COL0 + (it & 1) * 8, tsfb = tsfa + 4;
        if (elect_one()) {
          tmem_cp_32x128b_x4(tsfa, make_sf_desc(ssf));
          tmem_cp_32x128b_x4(tsfb, make_sf_desc(ssf + SF_BYTES));
#pragma unroll
          for (int k = 0; k < BK / 32; ++k)
            umma_mxf8(tmem_base + acc * BN, da + k * a_kstep, db + k * b_kstep, make_idesc_mx(BM, BN, a_mn, b_mn, k), tsfa, tsfb,
                      (kb | k) != 0);
          umma_commit(&empty_bar[s]);
        }
        __syncwarp();
      }
      if (ok) {
        if (elect_one()) umma_commit(&tmem_full[acc]);
        __syncwarp();
      }
    }
  } else {
    const int quarter = warp & 3;
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    uint32_t local_tile = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      const int tm = tile % tiles_m, tn = tile / tiles_m;
      const long long row = static_cast<long long>(tm) * BM + quarter * 32 + lane;
      const bool row_ok = row < args.M;
      const uint32_t acc = local_tile & 1;
      const uint32_t acc_ph = (local_tile >> 1) & 1;
      ++local_tile;
      if (!mbar_wait(&tmem_full[acc], acc_ph, abort_flag)) {
        if (lane == 0) {
          atomicExch(args.status, FSB_ERR_WAIT_TIMEOUT_TMEM_FULL);
          *abort_flag = 1;
        }
        break;
      }
      tc_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 32) {
        const int col = tn * BN + c0;
        if (col >= args.N) break;
        uint32_t v[32];
        tmem_ld_32x32(tmem_base + lane_off + acc * BN + c0, v);
        tmem_ld_wait();
        if (!row_ok) continue;
        const int ncols = min(32, args.N - col);
        if (args.d_fp32) {
          float* dp = static_cast<float*>(args.d) + row * args.ldd + col;
          for (int i = 0; i < ncols; ++i) dp[i] = __uint_as_float(v[i]);
        } else {
          __nv_bfloat16* dp = static_cast<__nv_bfloat16*>(args.d) + row * args.ldd + col;
          if (ncols == 32 && (args.ldd % 8) == 0) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(v[i]), __uint_as_float(v[i + 1]));
              o.y = pack_bf16x2(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
              o.z = pack_bf16x2(__uint_as_float(v[i + 4]), __uint_as_float(v[i + 5]));
              o.w = pack_bf16x2(__uint_as_float(v[i + 6]), __uint_as_float(v[i + 7]));
              *reinterpret_cast<uint4*>(dp + i) = o;
            }
          } else {
            for (int i = 0; i < ncols; ++i) dp[i] = __float2bfloat16(__uint_as_float(v[i]));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[acc]);
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
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------ block-scaled GEMM on SM pairs
// The same product on 256 x 256 tiles of a CTA pair. Per CTA and stage: 128 rows of A, 128 rows of B, the scales of its
// own A rows (one 512-byte block) and those of all 256 B rows (two blocks), which the tensor core of each SM wants in its
// own TMEM; tcgen05.cp on a pair copies them in both CTAs at once. An accumulator of 256 columns and the scales leave no
// room for a second accumulator, so eight warps move a finished tile from TMEM into registers and hand the accumulator
// back before they store it. Bound by the tensor cores; a 128 x 128 tile per SM is bound by operand traffic, 32 KB from
// L2 per 4.2 MFLOP against 34 KB per 8.4 MFLOP here. 5760 x 28672 x 4096: 879 -> 538 us (2.5 PFLOP/s), 2048 cubed: 21.1
// -> 17.0 us.
constexpr int P_STAGE_BYTES = A_STAGE + B_STAGE + 4 * SF_BYTES;   // the last 512 bytes keep every stage 1 KB aligned
constexpr int P_STAGE_TX = A_STAGE + B_STAGE + 3 * SF_BYTES;
constexpr int P_STAGES = 6;
constexpr int P_BN = 256;
constexpr int P_SMEM = P_STAGES * P_STAGE_BYTES + 1024 + 256;
constexpr int P_THREADS = 64 + 32 * 8;   // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue (two per lane quarter, 128 columns each)

__device__ __forceinline__ void tmem_cp_32x128b_x4_pair(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void umma_mxf8_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                               uint32_t tsfa, uint32_t tsfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tsfa), "r"(tsfb)
      : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1)
gemm_mxfp8_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                       const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb,
                       const MxArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + P_STAGES * P_STAGE_BYTES);
  uint64_t* full_bar = bars;                    // [P_STAGES]  used in CTA 0
  uint64_t* empty_bar = bars + P_STAGES;        // [P_STAGES]  one per CTA
  uint64_t* tmem_full = bars + 2 * P_STAGES;    // one per CTA
  uint64_t* tmem_empty = bars + 2 * P_STAGES + 1;   // used in CTA 0: the epilogue warps of both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * P_STAGES + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int tiles_m = (args.M + 2 * BM - 1) / (2 * BM), tiles_n = (args.N + P_BN - 1) / P_BN;
  const int num_tiles = tiles_m * tiles_n;
  const int num_kb = args.K / BK;
  const int tile0 = static_cast<int>(blockIdx.x >> 1), tile_step = static_cast<int>(gridDim.x >> 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < P_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tmem_full, 1);
    mbar_init(tmem_empty, 16);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer's barriers are initialised before anything is signalled across the pair
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&map_a);
      tma_prefetch_desc(&map_b);
      tma_prefetch_desc(&map_sfa);
      tma_prefetch_desc(&map_sfb);
      uint32_t it = 0;
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
        int tm, tn;
        grouped_tile_coords(tile, tiles_m, tiles_n, tm, tn);
        const int mb = tm * 2 + static_cast<int>(rank);   // 128-row block of A
        const int m0 = mb * BM, n0 = tn * P_BN + static_cast<int>(rank) * BN;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % P_STAGES;
          const uint32_t ph = (it / P_STAGES) & 1;
          if (!mbar_wait(&empty_bar[s], ph ^ 1, abort_flag)) {
            atomicExch(args.status, FSB_ERR_WAIT_TIMEOUT_EMPTY);
            *abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t* sa = smem + s * P_STAGE_BYTES;
          uint8_t* sb = sa + A_STAGE;
          uint8_t* ssf = sb + B_STAGE;
          const uint32_t full0 = map_to_cta(smem_u32(&full_bar[s]), 0);
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * P_STAGE_TX);   // the bytes of both CTAs
          if (!args.a_mn) tma_load_2d_pair(sa, &map_a, full0, kb * BK, m0);
          else tma_load_2d_pair(sa, &map_a, full0, m0, kb * BK);   // [K rows][128 M bytes]
          if (!args.b_mn) tma_load_2d_pair(sb, &map_b, full0, kb * BK, n0);
          else tma_load_2d_pair(sb, &map_b, full0, n0, kb * BK);   // [K rows][128 N bytes]
          // blocks past the last one read as zeros, like the rows they belong to
          tma_load_2d_pair(ssf, &map_sfa, full0, 0, mb * num_kb + kb);
          tma_load_2d_pair(ssf + SF_BYTES, &map_sfb, full0, 0, (tn * 2) * num_kb + kb);
          tma_load_2d_pair(ssf + 2 * SF_BYTES, &map_sfb, full0, 0, (tn * 2 + 1) * num_kb + kb);
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {   // one CTA issues for the pair; the whole warp walks the loop
      const uint32_t a_kstep = (args.a_mn ? 4096u : 32u) >> 4, b_kstep = (args.b_mn ? 4096u : 32u) >> 4;
      const uint32_t a_mn = args.a_mn ? 1u : 0u, b_mn = args.b_mn ? 1u : 0u;
      uint32_t it = 0, local_tile = 0;
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step, ++local_tile) {
        if (!mbar_wait(tmem_empty, (local_tile & 1) ^ 1, abort_flag)) {
          if (lane == 0) {
            atomicExch(args.status, FSB_ERR_WAIT_TIMEOUT_TMEM_EMPTY);
            *abort_flag = 1;
          }
          break;
        }
        tc_fence_after();
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % P_STAGES;
          const uint32_t ph = (it / P_STAGES) & 1;
          if (!mbar_wait(&full_bar[s], ph, abort_flag)) {
            if (lane == 0) {
              atomicExch(args.status, FSB_ERR_WAIT_TIMEOUT_FULL);
              *abort_flag = 1;
            }
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * P_STAGE_BYTES);
          const uint64_t da = make_smem_desc_sw128(sa, 16, 1024);
          const uint64_t db = make_smem_desc_sw128(sa + A_STAGE, 16, 1024);
          const uint32_t ssf = sa + A_STAGE + B_STAGE;
          const uint32_t tsfa = tmem_base + SF_COL0 + (it & 1) * 16, tsfb = tsfa + 8;   // 4 columns of A, 2 x 4 of B
          const uint32_t e_own = smem_u32(&empty_bar[s]);
          if (elect_one()) {
            tmem_cp_32x128b_x4_pair(tsfa, make_sf_desc(ssf));
            tmem_cp_32x128b_x4_pair(tsfb, make_sf_desc(ssf + SF_BYTES));
            tmem_cp_32x128b_x4_pair(tsfb + 4, make_sf_desc(ssf + 2 * SF_BYTES));
#pragma unroll
            for (int k = 0; k < BK / 32; ++k)
              umma_mxf8_pair(tmem_base, da + k * a_kstep, db + k * b_kstep, make_idesc_mx(2 * BM, P_BN, a_mn, b_mn, k), tsfa,
                             tsfb, (kb | k) != 0);
            umma_commit_pair(e_own);
            umma_commit_pair(map_to_cta(e_own, 1));
          }
          __syncwarp();
        }
        if (ok) {
          const uint32_t f_own = smem_u32(tmem_full);
          if (elect_one()) {
            umma_commit_pair(f_own);
            umma_commit_pair(map_to_cta(f_own, 1));
          }
          __syncwarp();
        }
      }
    }
  } else {
    const int quarter = warp & 3;
    const int part = (warp - 2) >> 2;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + part * 128;
    uint32_t local_tile = 0;
    for (int tile = tile0; tile < num_tiles; tile += tile_step, ++local_tile) {
      int tm, tn;
      grouped_tile_coords(tile, tiles_m, tiles_n, tm, tn);
      const int row = (tm * 2 + static_cast<int>(rank)) * BM + quarter * 32 + lane;
      if (!mbar_wait_warp(tmem_full, local_tile & 1, abort_flag)) {
        if (lane == 0) {
          atomicExch(args.status, FSB_ERR_WAIT_TIMEOUT_TMEM_FULL);
          *abort_flag = 1;
        }
        break;
      }
      tc_fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_row + 32 * c, v[c]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(tmem_empty), 0));   // the next tile may start
      if (row >= args.M) continue;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int col = tn * P_BN + part * 128 + c * 32;
        const int ncols = min(32, args.N - col);
        if (args.d_fp32) {
          float* dp = static_cast<float*>(args.d) + static_cast<long long>(row) * args.ldd + col;
          if (ncols == 32 && (reinterpret_cast<uintptr_t>(dp) & 15) == 0) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) *reinterpret_cast<uint4*>(dp + i) = make_uint4(v[c][i], v[c][i + 1], v[c][i + 2], v[c][i + 3]);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i < ncols) dp[i] = __uint_as_float(v[c][i]);
          }
        } else {
          __nv_bfloat16* dp = static_cast<__nv_bfloat16*>(args.d) + static_cast<long long>(row) * args.ldd + col;
          if (ncols == 32 && (reinterpret_cast<uintptr_t>(dp) & 15) == 0) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
              o.y = pack_bf16x2(__uint_as_float(v[c][i + 2]), __uint_as_float(v[c][i + 3]));
              o.z = pack_bf16x2(__uint_as_float(v[c][i + 4]), __uint_as_float(v[c][i + 5]));
              o.w = pack_bf16x2(__uint_as_float(v[c][i + 6]), __uint_as_float(v[c][i + 7]));
              *reinterpret_cast<uint4*>(dp + i) = o;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i < ncols) dp[i] = __float2bfloat16(__uint_as_float(v[c][i]));
          }
        }
      }
    }
  }

  // Every loop above is bounded, so all warps of both CTAs arrive here; neither CTA may leave before both are done.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    if (*abort_flag) {
      const unsigned long long t0 = clock64();
      while (clock64() - t0 < 2000000ull) {
      }
    }
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

int g_sms[64] = {0};
int g_pairs[64] = {0};   // co-resident clusters of the pair kernel, per device (-1: unusable)
}  // namespace

// w: bf16 [rows, cols]; q: e4m3 [rows, cols]; tile_exp: uint8 [ceil(rows/32), ceil(cols/32)].
FSB_API int fsb_mx_quant_weight(const void* w, void* q, void* tile_exp, int rows, int cols, long long ldw,
                                long long ldq, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return FSB_OK;
  const int exp_cols = (cols + 31) / 32;
  dim3 grid((exp_cols + 3) / 4, (rows + 31) / 32);
  const int vec = (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0 && ldw % 8 == 0 && ldq % 8 == 0;
  mx_quant_weight_kernel<<<grid, 128, 0, stream>>>(static_cast<const __nv_bfloat16*>(w), static_cast<uint8_t*>(q),
                                                   static_cast<uint8_t*>(tile_exp), rows, cols, ldw, ldq, exp_cols, vec);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}

// Blocked scales of the operand [rows, cols] (transpose == 0) or [cols, rows] (transpose == 1) from
// the tile exponents of a [rows, cols] weight. out: pad128(op rows) * pad4(ceil(op cols / 32)) bytes.
FSB_API int fsb_mx_expand_scales(const void* tile_exp, void* out, int rows, int cols, int transpose,
                                 cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return FSB_OK;
  const int op_rows = transpose ? cols : rows;
  const int op_groups = ((transpose ? rows : cols) + 31) / 32;
  const int pad_rows = (op_rows + 127) / 128 * 128, pad_groups = (op_groups + 3) / 4 * 4;
  const long long total = static_cast<long long>(pad_rows) * pad_groups;
  mx_expand_scales_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>(
      static_cast<const uint8_t*>(tile_exp), static_cast<uint8_t*>(out), op_rows, op_groups, pad_rows, pad_groups,
      (cols + 31) / 32, transpose);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}

// x: bf16 [T, K], K % 128 == 0; q: e4m3 [T, K]; scales: blocked, pad128(T) * (K/32) bytes (rows past T
// are not written: allocate zeroed or ignore them, they only feed output rows that are masked).
FSB_API int fsb_mx_quant_act(const void* x, void* q, void* scales, long long T, int K, long long ldx, long long ldq,
                             cudaStream_t stream) {
  if (K % 128 != 0 || ldx % 4 != 0 || ldq % 4 != 0) return FSB_ERR_BAD_ARG;
  if (T <= 0) return FSB_OK;
  const long long half = (T * (K / 32) + 1) / 2 * 4;   // as in the kernel: threads, two units each
  const int vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0 && ldx % 8 == 0 && ldq % 8 == 0;
  mx_quant_act_kernel<<<static_cast<unsigned>((half + 255) / 256), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q), static_cast<uint8_t*>(scales), T, K, ldx, ldq,
      K / 128, vec);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}

// x: bf16 [T, K] with T % 128 == 0 and K % 128 == 0; q: e4m3 [T, K] (same layout); scales: blocked scales of
// the operand x^T ([K rows, T/32 groups]): K * (T/32) bytes.
FSB_API int fsb_mx_quant_rows(const void* x, void* q, void* scales, long long T, int K, long long ldx, long long ldq,
                              cudaStream_t stream) {
  if (K % 128 != 0 || T % 128 != 0) return FSB_ERR_BAD_ARG;
  if (T <= 0) return FSB_OK;
  dim3 grid((K / 128 + 3) / 4, static_cast<unsigned>(T / 32));
  const int vec = (reinterpret_cast<uintptr_t>(x) & 7) == 0 && (reinterpret_cast<uintptr_t>(q) & 3) == 0 && ldx % 4 == 0 && ldq % 4 == 0;
  mx_quant_rows_kernel<<<grid, 128, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q),
                                                 static_cast<uint8_t*>(scales), K, ldx, ldq, static_cast<int>(T / 128), vec);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}

// D[M,N] = (Aq * 2^sfa) . (Bq * 2^sfb)^T with K % 128 == 0. A: e4m3 [M, K] (a_mn == 0) or [K, M]
// (a_mn == 1: M contiguous, M % 16 == 0). B: e4m3 [N, K] (b_mn == 0) or [K, N] (b_mn == 1: N contiguous,
// N % 16 == 0). sfa / sfb: blocked scales of the
// operands as the GEMM sees them ([M, K] and [N, K]).
FSB_API int fsb_gemm_mxfp8(const void* aq, const void* sfa, const void* bq, const void* sfb, void* d, int M, int N,
                           int K, long long lda, long long ldb, long long ldd, int a_mn, int b_mn, int d_fp32,
                           int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || K % BK != 0) return FSB_ERR_BAD_ARG;
  if ((b_mn && N % 16 != 0) || (a_mn && M % 16 != 0)) return FSB_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(sfa) | reinterpret_cast<uintptr_t>(sfb)) & 15) return FSB_ERR_BAD_ARG;
  CUtensorMap map_a, map_b;
  int rc;
  if (!a_mn) rc = fsb_make_tmap_2d(&map_a, aq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, M, K, lda, BM, BK);
  else rc = fsb_make_tmap_2d(&map_a, aq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K, M, lda, BK, BM);
  if (rc != FSB_OK) return rc;
  if (!b_mn) rc = fsb_make_tmap_2d(&map_b, bq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K, ldb, BN, BK);
  else rc = fsb_make_tmap_2d(&map_b, bq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K, N, ldb, BK, BN);
  if (rc != FSB_OK) return rc;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return FSB_ERR_BAD_ARG;
  if (g_sms[dev] == 0) {
    if (cudaFuncSetAttribute(gemm_mxfp8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) !=
        cudaSuccess)
      return FSB_ERR_LAUNCH;
    cudaDeviceGetAttribute(&g_sms[dev], cudaDevAttrMultiProcessorCount, dev);
  }
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  const int grid = tiles < g_sms[dev] ? tiles : g_sms[dev];
  MxArgs a;
  a.M = M; a.N = N; a.K = K; a.a_mn = a_mn; a.b_mn = b_mn;
  a.sfa = static_cast<const uint8_t*>(sfa); a.sfb = static_cast<const uint8_t*>(sfb);
  a.d = d; a.ldd = ldd; a.d_fp32 = d_fp32; a.status = status;
  if (g_pairs[dev] == 0) g_pairs[dev] = fsb_resident_pairs(gemm_mxfp8_pair_kernel, P_THREADS, P_SMEM);
  const int pairs = g_pairs[dev];
  if (pairs > 0) {
    const int tiles2 = ((M + 2 * BM - 1) / (2 * BM)) * ((N + P_BN - 1) / P_BN);
    const int waves1 = (tiles + g_sms[dev] - 1) / g_sms[dev], waves2 = (tiles2 + pairs - 1) / pairs;
    // A pair's tile takes about 1.2 times as long as the quarter of it that one SM takes otherwise (14.7 against 12.2 us at a
    // depth of 4096), so the pairs win where they need few enough waves; a single wave of either is the small tiles'.
    if (5 * waves2 <= 4 * waves1) {
      // one row of 128 words per 512-byte scale block
      CUtensorMap map_sfa, map_sfb;
      rc = fsb_make_tmap_2d_plain(&map_sfa, sfa, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4,
                                  static_cast<uint64_t>((M + BM - 1) / BM) * (K / BK), 128, 128, 1, 128);
      if (rc != FSB_OK) return rc;
      rc = fsb_make_tmap_2d_plain(&map_sfb, sfb, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4,
                                  static_cast<uint64_t>((N + BN - 1) / BN) * (K / BK), 128, 128, 1, 128);
      if (rc != FSB_OK) return rc;
      const int clusters = tiles2 < pairs ? tiles2 : pairs;
      gemm_mxfp8_pair_kernel<<<2 * clusters, P_THREADS, P_SMEM, stream>>>(map_a, map_b, map_sfa, map_sfb, a);
      return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
    }
  }
  gemm_mxfp8_kernel<<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(map_a, map_b, a);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}
