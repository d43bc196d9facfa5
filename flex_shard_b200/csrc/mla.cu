// Operand layout of multi-head latent attention in one pass each way.
//
// forward:  q [T, H, nope + rope], kv [T, H, nope + value] and the rotary key shared by all heads, k_pe [T, rope]
//   ->      query [T, H, nope + rope] (rotary part rotated), key [T, H, nope + rope] (the head's own part, then the
//           rotated shared part), value [T, H, value]
// backward: the gradients of those three -> dq, dkv (both parts written in place, no zero-filled halves to add) and
//           dk_pe (summed over the heads in fp32, in head order, rotated back, rounded once).
//
// Bound by memory, so one block per token and 16 bytes per thread and access; rotating in fp32 costs nothing next to it.
// As slices, concatenations and element-wise rotations this was about 25 kernels a layer and pass, which moved each
// element five to eight times: a step of two blocks at 8192 tokens, 16 heads of 128 + 64, went from 31.8 to 29.6 ms.
#include "common.cuh"

namespace {
using namespace fsb;

constexpr int THREADS = 256;

// Rotates the four pairs of a 16-byte vector; cs points at the (cos, sin) of the first one.
template <bool INVERSE>
__device__ __forceinline__ uint4 rotate8(uint4 raw, const float2* __restrict__ cs) {
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 x = __bfloat1622float2(h[i]);
    const float c = cs[i].x, s = INVERSE ? -cs[i].y : cs[i].y;
    h[i] = __floats2bfloat162_rn(x.x * c - x.y * s, x.x * s + x.y * c);
  }
  return raw;
}

struct MlaArgs {
  int S, H, nope, rope, value;   // widths in elements, multiples of 8
  long long ld_pe;               // row stride of k_pe (forward)
};

__global__ void __launch_bounds__(THREADS)
mla_pack_kernel(const uint4* __restrict__ q, const uint4* __restrict__ kv, const __nv_bfloat16* __restrict__ k_pe,
                const float2* __restrict__ table, uint4* __restrict__ qo, uint4* __restrict__ ko, uint4* __restrict__ vo,
                const MlaArgs a) {
  const long long t = blockIdx.x;
  const float2* cs = table + static_cast<long long>(t % a.S) * (a.rope / 2);
  const int n8 = a.nope / 8, v8 = a.value / 8, w8 = n8 + a.rope / 8, kv8 = n8 + v8;
  const uint4* pe = reinterpret_cast<const uint4*>(k_pe + t * a.ld_pe);
  q += t * a.H * w8;
  qo += t * a.H * w8;
  ko += t * a.H * w8;
  kv += t * a.H * kv8;
  vo += t * a.H * v8;
  for (int u = threadIdx.x; u < a.H * w8; u += THREADS) {
    const int h = u / w8, c = u - h * w8;
    uint4 x = q[u];
    uint4 y = c < n8 ? kv[h * kv8 + c] : pe[c - n8];
    if (c >= n8) {
      x = rotate8<false>(x, cs + (c - n8) * 4);
      y = rotate8<false>(y, cs + (c - n8) * 4);
    }
    qo[u] = x;
    ko[u] = y;
  }
  for (int u = threadIdx.x; u < a.H * v8; u += THREADS) {
    const int h = u / v8, c = u - h * v8;
    vo[u] = kv[h * kv8 + n8 + c];
  }
}

__global__ void __launch_bounds__(THREADS)
mla_unpack_kernel(const uint4* __restrict__ dqo, const uint4* __restrict__ dko, const uint4* __restrict__ dvo,
                  const float2* __restrict__ table, uint4* __restrict__ dq, uint4* __restrict__ dkv,
                  __nv_bfloat16* __restrict__ dk_pe, const MlaArgs a) {
  const long long t = blockIdx.x;
  const float2* cs = table + static_cast<long long>(t % a.S) * (a.rope / 2);
  const int n8 = a.nope / 8, v8 = a.value / 8, w8 = n8 + a.rope / 8, kv8 = n8 + v8;
  const __nv_bfloat162* pe = reinterpret_cast<const __nv_bfloat162*>(dko + t * a.H * w8) + a.nope / 2;
  dqo += t * a.H * w8;
  dko += t * a.H * w8;
  dvo += t * a.H * v8;
  dq += t * a.H * w8;
  dkv += t * a.H * kv8;
  for (int p = threadIdx.x; p < a.rope / 2; p += THREADS) {   // a thread per pair of the shared key, over the heads
    float2 s = make_float2(0.f, 0.f);
    for (int h = 0; h < a.H; ++h) {
      const float2 x = __bfloat1622float2(pe[h * (w8 * 4) + p]);
      s.x += x.x;
      s.y += x.y;
    }
    const float c = cs[p].x, sn = -cs[p].y;
    reinterpret_cast<__nv_bfloat162*>(dk_pe + t * a.rope)[p] = __floats2bfloat162_rn(s.x * c - s.y * sn, s.x * sn + s.y * c);
  }
  for (int u = threadIdx.x; u < a.H * w8; u += THREADS) {
    const int h = u / w8, c = u - h * w8;
    const uint4 x = dqo[u];
    dq[u] = c < n8 ? x : rotate8<true>(x, cs + (c - n8) * 4);
    if (c < n8) dkv[h * kv8 + c] = dko[u];
  }
  for (int u = threadIdx.x; u < a.H * v8; u += THREADS) {
    const int h = u / v8, c = u - h * v8;
    dkv[h * kv8 + n8 + c] = dvo[u];
  }
}

bool bad(long long T, const MlaArgs& a, const void* const* ptrs, int n) {
  uintptr_t bits = 0;
  for (int i = 0; i < n; ++i) bits |= reinterpret_cast<uintptr_t>(ptrs[i]);
  return T <= 0 || T >= (1ll << 31) || a.S <= 0 || a.H <= 0 || a.nope <= 0 || a.rope <= 0 || a.value <= 0 || a.nope % 8 ||
         a.rope % 8 || a.value % 8 || a.ld_pe % 8 || (bits & 15);
}
}  // namespace

// q, kv, query, key, value: dense bf16 as in the header comment; k_pe: rows of `rope` elements ld_pe apart; table: fp32
// (cos, sin) [>= S, rope / 2]. Row t holds position t % S. All pointers on 16-byte boundaries.
FSB_API int fsb_mla_pack(const void* q, const void* kv, const void* k_pe, const float* table, void* query, void* key,
                         void* value, long long T, int S, int H, int nope, int rope, int vdim, long long ld_pe,
                         cudaStream_t stream) {
  const MlaArgs a{S, H, nope, rope, vdim, ld_pe};
  const void* ptrs[] = {q, kv, k_pe, table, query, key, value};
  if (bad(T, a, ptrs, 7)) return FSB_ERR_BAD_ARG;
  mla_pack_kernel<<<static_cast<unsigned>(T), THREADS, 0, stream>>>(
      static_cast<const uint4*>(q), static_cast<const uint4*>(kv), static_cast<const __nv_bfloat16*>(k_pe),
      reinterpret_cast<const float2*>(table), static_cast<uint4*>(query), static_cast<uint4*>(key),
      static_cast<uint4*>(value), a);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}

FSB_API int fsb_mla_unpack(const void* dquery, const void* dkey, const void* dvalue, const float* table, void* dq, void* dkv,
                           void* dk_pe, long long T, int S, int H, int nope, int rope, int vdim, cudaStream_t stream) {
  const MlaArgs a{S, H, nope, rope, vdim, rope};
  const void* ptrs[] = {dquery, dkey, dvalue, table, dq, dkv, dk_pe};
  if (bad(T, a, ptrs, 7)) return FSB_ERR_BAD_ARG;
  mla_unpack_kernel<<<static_cast<unsigned>(T), THREADS, 0, stream>>>(
      static_cast<const uint4*>(dquery), static_cast<const uint4*>(dkey), static_cast<const uint4*>(dvalue),
      reinterpret_cast<const float2*>(table), static_cast<uint4*>(dq), static_cast<uint4*>(dkv),
      static_cast<__nv_bfloat16*>(dk_pe), a);
  return cudaGetLastError() == cudaSuccess ? FSB_OK : FSB_ERR_LAUNCH;
}
