// Gradient of a token embedding, written once, straight into its destination (the fp32 rows of a reduction bucket, or a
// bf16 gradient).
//
// Every row of the [V, D] result is written exactly once: zeros, or the sum of the output gradients of the tokens that
// read it, added in fp32 in an order that only the tokens decide (the same bits on every run). The tokens are grouped by
// value first: a histogram, a scan over the vocabulary, a list of token positions per value. A value that up to SEG tokens
// read is the work of its row's block, which restores their order and adds them. The list of a more frequent one is put in
// order by a block, segments of SEG positions are added by a block each, and the row's block adds the segments' sums: a
// padding token or a long row of text would otherwise leave thousands of rows to one SM (8192 x 4096, half of the tokens
// equal: 3.6 ms with a block to a value, 0.70 ms in segments, 2.2 ms with the library's sort; 65536 tokens, all equal:
// 48.7, 1.5 and 3.8 ms).
// Spread over the vocabulary, tokens leave mostly the result to be written, 2.1 GB for 128256 x 4096 in fp32: 0.64 ms
// (3.3 TB/s; a block to a row is short of stores in flight), where the library's backward, its zero fill in bf16 and the
// widening copy into the bucket took 2.4 ms.
#include "common.cuh"
#include <type_traits>

namespace {
using namespace fsb;

constexpr int THREADS = 256;
constexpr int SCAN_THREADS = 1024;
constexpr int SEG = 64;             // rows that one block adds
constexpr int ORDER_THREADS = 512;
constexpr int LIST = 2048;          // positions that are ordered in shared memory; longer lists are found again in order
constexpr int MAX_D = 4 * THREADS * 8;

__device__ __forceinline__ long long token(const void* t, int is64, long long i) {
  return is64 ? static_cast<const long long*>(t)[i] : static_cast<const int*>(t)[i];
}

// Lanes with the same value `v`: the first of them changes its counter by their number, once. Returns the lane's rank
// among them; `old` is the counter before (where v >= 0; a negative value counts nothing).
__device__ __forceinline__ int count_equal(int* counters, int v, int sign, int& old) {
  const unsigned same = __match_any_sync(0xffffffffu, v);
  const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
  old = 0;
  if (v >= 0 && lane == leader) old = atomicAdd(counters + v, sign * __popc(same));
  old = __shfl_sync(0xffffffffu, old, leader);
  return __popc(same & ((1u << lane) - 1));
}
__device__ __forceinline__ int value_at(const void* tokens, int is64, int i, int T, int V) {
  if (i >= T) return -1;
  const long long v = token(tokens, is64, i);
  return v >= 0 && v < V ? static_cast<int>(v) : -1;
}

__global__ void __launch_bounds__(THREADS)
count_kernel(const void* __restrict__ tokens, int is64, int T, int V, int* __restrict__ count) {
  int old;
  count_equal(count, value_at(tokens, is64, blockIdx.x * THREADS + threadIdx.x, T, V), 1, old);
}

__device__ __forceinline__ int segments(int n) { return n > SEG ? (n + SEG - 1) / SEG : 0; }

// start[v] = number of tokens with a value below v, start[V] = all; owner[s] = value of segment s (the segments of all
// values with more than SEG tokens, in order of the values), *total their number. One block; count and start on 16-byte
// boundaries, with room for whole vectors.
__global__ void __launch_bounds__(SCAN_THREADS, 1)
scan_kernel(const int* __restrict__ count, int V, int* __restrict__ start, int* __restrict__ owner, int* __restrict__ total) {
  __shared__ unsigned long long warp_sum_s[32];   // segments in the upper half, tokens in the lower
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int PER = 16;   // values per thread and round: 8 rounds for 128 K values
  unsigned long long base = 0;
  for (int v0 = 0; v0 < V; v0 += PER * SCAN_THREADS) {
    alignas(16) int c[PER];
    unsigned long long own = 0;
    const int v = v0 + threadIdx.x * PER;
#pragma unroll
    for (int j = 0; j < PER; j += 4)
      *reinterpret_cast<int4*>(c + j) = v + j < V ? *reinterpret_cast<const int4*>(count + v + j) : make_int4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (v + j >= V) c[j] = 0;
      own += (static_cast<unsigned long long>(segments(c[j])) << 32) + c[j];
    }
    unsigned long long sum = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, sum, d);
      if (lane >= d) sum += up;
    }
    if (lane == 31) warp_sum_s[warp] = sum;
    __syncthreads();
    if (warp == 0) {
      unsigned long long w = warp_sum_s[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long up = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w += up;
      }
      warp_sum_s[lane] = w;
    }
    __syncthreads();
    const unsigned long long before = base + sum - own + (warp > 0 ? warp_sum_s[warp - 1] : 0);
    int seg = static_cast<int>(before >> 32);
    if (own >> 32) {
#pragma unroll 1
      for (int j = 0; j < PER; ++j) {
        const int k = v + j < V ? segments(count[v + j]) : 0;
        for (int i = 0; i < k; ++i) owner[seg + i] = v + j;
        seg += k;
      }
    }
    int at = static_cast<int>(before & 0xffffffffu);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int n = c[j];
      c[j] = at;
      at += n;
    }
#pragma unroll
    for (int j = 0; j < PER; j += 4)
      if (v + j < V) *reinterpret_cast<int4*>(start + v + j) = *reinterpret_cast<const int4*>(c + j);   // start[V] too, if it is there
    base += warp_sum_s[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    start[V] = static_cast<int>(base & 0xffffffffu);
    *total = static_cast<int>(base >> 32);
  }
}

// First segment of value v.
__device__ __forceinline__ int first_segment(const int* __restrict__ owner, int total, int v) {
  int lo = 0, hi = total;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (owner[mid] < v) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Fills the lists; counts down to 0.
__global__ void __launch_bounds__(THREADS)
place_kernel(const void* __restrict__ tokens, int is64, int T, int V, const int* __restrict__ start, int* __restrict__ count,
             int* __restrict__ list) {
  const int i = blockIdx.x * THREADS + threadIdx.x;
  const int v = value_at(tokens, is64, i, T, V);
  int left;
  const int rank = count_equal(count, v, -1, left);
  if (v >= 0) list[start[v] + left - 1 - rank] = i;
}

// Puts the list of every value with segments in order; the block of a value's first segment does it.
__global__ void __launch_bounds__(ORDER_THREADS)
order_kernel(const void* __restrict__ tokens, int is64, int T, const int* __restrict__ owner, const int* __restrict__ total,
             const int* __restrict__ start, int* __restrict__ list) {
  __shared__ int raw[LIST];
  __shared__ int warp_n[ORDER_THREADS / 32];
  const int s = blockIdx.x;
  if (s >= *total || (s > 0 && owner[s - 1] == owner[s])) return;
  const int v = owner[s], lo = start[v], n = start[v + 1] - lo;
  constexpr int PER = LIST / ORDER_THREADS;
  if (n <= LIST) {
    for (int i = threadIdx.x; i < n; i += ORDER_THREADS) raw[i] = list[lo + i];
    __syncthreads();
    int own[PER], rank[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = threadIdx.x + k * ORDER_THREADS;
      own[k] = i < n ? raw[i] : 0;
      rank[k] = 0;
    }
    for (int j = 0; j < n; ++j) {                    // positions are distinct: the rank is the place
      const int r = raw[j];
#pragma unroll
      for (int k = 0; k < PER; ++k) rank[k] += r < own[k];
    }
#pragma unroll
    for (int k = 0; k < PER; ++k)
      if (threadIdx.x + k * ORDER_THREADS < n) list[lo + rank[k]] = own[k];
    return;
  }
  int at = lo;                                       // the tokens again, in order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (long long t0 = 0; t0 < T; t0 += PER * ORDER_THREADS) {
    const long long i0 = t0 + threadIdx.x * PER;
    bool hit[PER];
    int own = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      hit[k] = i0 + k < T && token(tokens, is64, i0 + k) == v;
      own += hit[k];
    }
    int sum = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, d);
      if (lane >= d) sum += up;
    }
    if (lane == 31) warp_n[warp] = sum;
    __syncthreads();
    int put = at + sum - own;
    for (int w = 0; w < ORDER_THREADS / 32; ++w) {
      if (w < warp) put += warp_n[w];
      at += warp_n[w];
    }
#pragma unroll
    for (int k = 0; k < PER; ++k)
      if (hit[k]) list[put++] = static_cast<int>(i0) + k;
    __syncthreads();
  }
}

// s += the rows of dy at the m positions, in order; a thread holds the sums of STEPS groups of 8 columns.
template <int STEPS>
__device__ __forceinline__ void add_rows(float (&s)[STEPS][8], const __nv_bfloat16* __restrict__ dy,
                                         const int* __restrict__ positions, int m, int D) {
#pragma unroll 4
  for (int i = 0; i < m; ++i) {
    const __nv_bfloat16* row = dy + static_cast<long long>(positions[i]) * D;
#pragma unroll
    for (int k = 0; k < STEPS; ++k) {
      const int c = (k * THREADS + threadIdx.x) * 8;
      if (c < D) {
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
  }
}

// A block per segment: its rows' sum in fp32.
template <int STEPS>
__global__ void __launch_bounds__(THREADS)
segments_kernel(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ owner, const int* __restrict__ total,
                const int* __restrict__ start, const int* __restrict__ list, int D, float* __restrict__ partial) {
  const int seg = blockIdx.x;
  if (seg >= *total) return;
  const int v = owner[seg], lo = start[v] + (seg - first_segment(owner, seg, v)) * SEG;
  float s[STEPS][8] = {};
  add_rows<STEPS>(s, dy, list + lo, min(SEG, start[v + 1] - lo), D);
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {
    const int c = (k * THREADS + threadIdx.x) * 8;
    if (c >= D) break;
    float4* o = reinterpret_cast<float4*>(partial + static_cast<long long>(seg) * D + c);
    o[0] = make_float4(s[k][0], s[k][1], s[k][2], s[k][3]);
    o[1] = make_float4(s[k][4], s[k][5], s[k][6], s[k][7]);
  }
}

// A block per vocabulary row.
template <bool FP32, int STEPS>
__global__ void __launch_bounds__(THREADS)
rows_kernel(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ start, const int* __restrict__ list,
            const int* __restrict__ owner, const int* __restrict__ total, const float* __restrict__ partial, int D,
            int accumulate, void* __restrict__ out) {
  __shared__ int raw[SEG], order[SEG];
  const int v = blockIdx.x;
  const int lo = start[v], n = start[v + 1] - lo;
  if (n == 0 && accumulate) return;
  float s[STEPS][8] = {};
  if (n > SEG) {
    const float* p = partial + static_cast<long long>(first_segment(owner, *total, v)) * D;
    const int m = segments(n);
#pragma unroll 4
    for (int i = 0; i < m; ++i, p += D) {
#pragma unroll
      for (int k = 0; k < STEPS; ++k) {
        const int c = (k * THREADS + threadIdx.x) * 8;
        if (c < D) {
          const float4 a = *reinterpret_cast<const float4*>(p + c), b = *reinterpret_cast<const float4*>(p + c + 4);
          s[k][0] += a.x; s[k][1] += a.y; s[k][2] += a.z; s[k][3] += a.w;
          s[k][4] += b.x; s[k][5] += b.y; s[k][6] += b.z; s[k][7] += b.w;
        }
      }
    }
  } else if (n > 0) {
    if (threadIdx.x < n) raw[threadIdx.x] = list[lo + threadIdx.x];
    __syncthreads();
    if (threadIdx.x < n) {                            // positions are distinct: the rank is the place
      int rank = 0;
      for (int j = 0; j < n; ++j) rank += raw[j] < raw[threadIdx.x];
      order[rank] = raw[threadIdx.x];
    }
    __syncthreads();
    add_rows<STEPS>(s, dy, order, n, D);
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

struct Scratch {                // offsets in ints, multiples of 4
  long long start, list, owner, total, partial, size;
  long long most;               // segments: a value with n > SEG tokens has fewer than 2 n / SEG of them
  static long long up4(long long n) { return (n + 3) / 4 * 4; }
  Scratch(long long T, long long V, long long D) {
    most = T > SEG ? 2 * T / SEG : 0;
    start = up4(V);             // count [V] at 0
    list = start + up4(V + 1);
    owner = list + up4(T);
    total = owner + up4(most);
    partial = total + 4;
    size = partial + most * D;
  }
};
}  // namespace

// Ints of scratch that fsb_embedding_grad needs.
FSB_API long long fsb_embedding_scratch_ints(long long T, int V, int D) { return Scratch(T, V, D).size; }

// out [V, D] (fp32 or bf16, dense) = (out +) sum over tokens t of dy[t] in row tokens[t]; dy bf16 [T, D], D % 8 == 0 and at
// most 8192, dy, out and scratch on 16-byte boundaries. Values outside [0, V) add nothing. accumulate: fp32 only.
FSB_API int fsb_embedding_grad(const void* dy, const void* tokens, int tokens_i64, long long T, int V, int D, void* out,
                               int out_fp32, int accumulate, int* scratch, cudaStream_t stream) {
  if (T <= 0 || T >= (1ll << 31) || V <= 0 || D <= 0 || D % 8 != 0 || D > MAX_D || (accumulate && !out_fp32)) return FSB_ERR_BAD_ARG;
  if (((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(scratch)) & 15) != 0)
    return FSB_ERR_BAD_ARG;
  const Scratch at(T, V, D);
  int* count = scratch;
  int *start = scratch + at.start, *list = scratch + at.list, *owner = scratch + at.owner, *total = scratch + at.total;
  float* partial = reinterpret_cast<float*>(scratch + at.partial);
  const int n = static_cast<int>(T);
  const unsigned blocks = static_cast<unsigned>((T + THREADS - 1) / THREADS), most = static_cast<unsigned>(at.most);
  if (cudaMemsetAsync(count, 0, static_cast<size_t>(V) * sizeof(int), stream) != cudaSuccess) return FSB_ERR_LAUNCH;
  count_kernel<<<blocks, THREADS, 0, stream>>>(tokens, tokens_i64, n, V, count);
  scan_kernel<<<1, SCAN_THREADS, 0, stream>>>(count, V, start, owner, total);
  place_kernel<<<blocks, THREADS, 0, stream>>>(tokens, tokens_i64, n, V, start, count, list);
  if (most > 0) order_kernel<<<most, ORDER_THREADS, 0, stream>>>(tokens, tokens_i64, n, owner, total, start, list);
  const __nv_bfloat16* g = static_cast<const __nv_bfloat16*>(dy);
  const int steps = (D + THREADS * 8 - 1) / (THREADS * 8);
  auto sized = [&](auto st) {
    constexpr int STEPS = decltype(st)::value;
    if (most > 0) segments_kernel<STEPS><<<most, THREADS, 0, stream>>>(g, owner, total, start, list, D, partial);
    if (out_fp32) rows_kernel<true, STEPS><<<V, THREADS, 0, stream>>>(g, start, list, owner, total, partial, D, accumulate, out);
    else rows_kernel<false, STEPS><<<V, THREADS, 0, stream>>>(g, start, list, owner, total, partial, D, accumulate, out);
  };
  if (steps == 1) sized(std::integral_constant<int, 1>{});
  else if (steps == 2) sized(std::integral_constant<int, 2>{});
  else sized(std::integral_constant<int, 4>{});
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}
