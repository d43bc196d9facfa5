// Gradient of a token embedding, written once, straight into its destination (the fp32 rows of a reduction bucket, or a
// bf16 gradient).
//
// Every row of the [V, D] result is written exactly once: zeros, or the sum of the output gradients of the tokens that
// read it, added in fp32 in token order (the same bits on every run). The tokens are grouped by value first: a histogram,
// a scan over the vocabulary, a list of token positions per value whose order the row's block then restores. Bound by
// writing the result: 2.1 GB for 128256 x 4096 in fp32. The sort of the library's backward, its zero fill in bf16 and the
// widening copy into the bucket that followed moved twice that in some twenty launches: 1.8 ms
// against 0.9.
#include "common.cuh"
#include <type_traits>

namespace {
using namespace fsb;

constexpr int THREADS = 256;
constexpr int SCAN_THREADS = 1024;
constexpr int LIST = 2048;   // positions a block orders at a time
constexpr int MAX_D = 4 * THREADS * 8;

__device__ __forceinline__ long long token(const void* t, int is64, long long i) {
  return is64 ? static_cast<const long long*>(t)[i] : static_cast<const int*>(t)[i];
}

__global__ void __launch_bounds__(THREADS)
count_kernel(const void* __restrict__ tokens, int is64, int T, int V, int* __restrict__ count) {
  const int i = blockIdx.x * THREADS + threadIdx.x;
  if (i >= T) return;
  const long long v = token(tokens, is64, i);
  if (v >= 0 && v < V) atomicAdd(count + v, 1);
}

// start[v] = number of tokens with a value below v, start[V] = all; one block, a contiguous range per thread.
__global__ void __launch_bounds__(SCAN_THREADS)
scan_kernel(const int* __restrict__ count, int V, int* __restrict__ start, int* __restrict__ cursor) {
  __shared__ int warp_sum_s[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int PER = 16;   // values per thread and round: 8 rounds for 128 K values
  int base = 0;
  for (int v0 = 0; v0 < V; v0 += PER * SCAN_THREADS) {
    int c[PER], own = 0;
    const int v = v0 + threadIdx.x * PER;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      c[j] = v + j < V ? count[v + j] : 0;
      own += c[j];
    }
    int sum = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, d);
      if (lane >= d) sum += up;
    }
    if (lane == 31) warp_sum_s[warp] = sum;
    __syncthreads();
    if (warp == 0) {
      int w = warp_sum_s[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w += up;
      }
      warp_sum_s[lane] = w;
    }
    __syncthreads();
    int at = base + sum - own + (warp > 0 ? warp_sum_s[warp - 1] : 0);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (v + j < V) {
        start[v + j] = at;
        cursor[v + j] = at;
      }
      at += c[j];
    }
    base += warp_sum_s[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) start[V] = base;
}

__global__ void __launch_bounds__(THREADS)
place_kernel(const void* __restrict__ tokens, int is64, int T, int V, int* __restrict__ cursor, int* __restrict__ list) {
  const int i = blockIdx.x * THREADS + threadIdx.x;
  if (i >= T) return;
  const long long v = token(tokens, is64, i);
  if (v >= 0 && v < V) list[atomicAdd(cursor + v, 1)] = i;
}

// A block per vocabulary row; a thread holds the sums of STEPS groups of 8 columns.
template <bool FP32, int STEPS>
__global__ void __launch_bounds__(THREADS)
rows_kernel(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ start, const int* __restrict__ list, int T, int D,
            int accumulate, void* __restrict__ out) {
  __shared__ int raw[LIST], order[LIST];
  __shared__ int found;
  const int v = blockIdx.x;
  const int lo = start[v], n = start[v + 1] - lo;
  if (n == 0 && accumulate) return;
  float s[STEPS][8] = {};
  const int passes = n <= LIST ? 1 : (T + LIST - 1) / LIST;   // long lists: the positions of a range at a time
  for (int p = 0; p < passes; ++p) {
    int m = n;
    if (passes == 1) {
      for (int i = threadIdx.x; i < n; i += THREADS) raw[i] = list[lo + i];
    } else {
      if (threadIdx.x == 0) found = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += THREADS) {
        const int t = list[lo + i];
        if (t / LIST == p) raw[atomicAdd(&found, 1)] = t;     // at most LIST distinct positions
      }
      __syncthreads();
      m = found;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += THREADS) {          // positions are distinct: the rank is the place
      int rank = 0;
      for (int j = 0; j < m; ++j) rank += raw[j] < raw[i];
      order[rank] = raw[i];
    }
    __syncthreads();
    for (int i = 0; i < m; ++i) {
      const __nv_bfloat16* row = dy + static_cast<long long>(order[i]) * D;
#pragma unroll
      for (int k = 0; k < STEPS; ++k) {
        const int c = (k * THREADS + threadIdx.x) * 8;
        if (c >= D) break;
        const uint4 x = *reinterpret_cast<const uint4*>(row + c);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __bfloat1622float2(h[j]);
          s[k][2 * j] += f.x;
          s[k][2 * j + 1] += f.y;
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {
    const int c = (k * THREADS + threadIdx.x) * 8;
    if (c >= D) break;
    const long long at = static_cast<long long>(v) * D + c;
    if (FP32) {
      float4* o = reinterpret_cast<float4*>(static_cast<float*>(out) + at);
      float4 a = make_float4(s[k][0], s[k][1], s[k][2], s[k][3]), b = make_float4(s[k][4], s[k][5], s[k][6], s[k][7]);
      if (accumulate) {
        const float4 c0 = o[0], c1 = o[1];
        a.x += c0.x; a.y += c0.y; a.z += c0.z; a.w += c0.w;
        b.x += c1.x; b.y += c1.y; b.z += c1.z; b.w += c1.w;
      }
      o[0] = a;
      o[1] = b;
    } else {
      uint4 x;
      x.x = pack_bf16x2(s[k][0], s[k][1]);
      x.y = pack_bf16x2(s[k][2], s[k][3]);
      x.z = pack_bf16x2(s[k][4], s[k][5]);
      x.w = pack_bf16x2(s[k][6], s[k][7]);
      *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(out) + at) = x;
    }
  }
}
}  // namespace

// out [V, D] (fp32 or bf16, dense) = (out +) sum over tokens t of dy[t] in row tokens[t]; dy bf16 [T, D], D % 8 == 0 and at
// most 8192, dy and out on 16-byte boundaries. Values outside [0, V) add nothing. scratch: 3 V + T + 1 ints. accumulate:
// fp32 only.
FSB_API int fsb_embedding_grad(const void* dy, const void* tokens, int tokens_i64, long long T, int V, int D, void* out,
                               int out_fp32, int accumulate, int* scratch, cudaStream_t stream) {
  if (T <= 0 || T >= (1ll << 31) || V <= 0 || D <= 0 || D % 8 != 0 || D > MAX_D || (accumulate && !out_fp32)) return FSB_ERR_BAD_ARG;
  if (((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(out)) & 15) != 0) return FSB_ERR_BAD_ARG;
  int* count = scratch;
  int* start = count + V;            // V + 1
  int* cursor = start + V + 1;
  int* list = cursor + V;            // T
  const int n = static_cast<int>(T);
  const unsigned blocks = static_cast<unsigned>((T + THREADS - 1) / THREADS);
  if (cudaMemsetAsync(count, 0, static_cast<size_t>(V) * sizeof(int), stream) != cudaSuccess) return FSB_ERR_LAUNCH;
  count_kernel<<<blocks, THREADS, 0, stream>>>(tokens, tokens_i64, n, V, count);
  scan_kernel<<<1, SCAN_THREADS, 0, stream>>>(count, V, start, cursor);
  place_kernel<<<blocks, THREADS, 0, stream>>>(tokens, tokens_i64, n, V, cursor, list);
  const __nv_bfloat16* g = static_cast<const __nv_bfloat16*>(dy);
  const int steps = (D + THREADS * 8 - 1) / (THREADS * 8);
  auto rows = [&](auto fp32, auto st) {
    rows_kernel<decltype(fp32)::value, decltype(st)::value><<<V, THREADS, 0, stream>>>(g, start, list, n, D, accumulate, out);
  };
  auto sized = [&](auto fp32) {
    if (steps == 1) rows(fp32, std::integral_constant<int, 1>{});
    else if (steps == 2) rows(fp32, std::integral_constant<int, 2>{});
    else rows(fp32, std::integral_constant<int, 4>{});
  };
  if (out_fp32) sized(std::true_type{});
  else sized(std::false_type{});
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}
