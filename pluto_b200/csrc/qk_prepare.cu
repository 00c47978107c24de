// Per-head RMSNorm(1 + w) -> optional bf16 rounding -> split-half partial RoPE for queries and
// keys, plus the K/V append into the cache.  Stands in for PrepareAttentionKernel
// (src/llm/layers/util/cached_attention_ops.cc:30-79) and its sequence form PrepareKernel
// (src/llm/layers/qwen_attention.cc:30-63): the rounding sequence
//     n = R(x * inv * (1 + w));  out = R(R(n * R(cos)) + R(+-n_partner * R(sin)))
// is reproduced step by step because the reference pins sequence and cached paths to bit equality.
//
// A CTA of eight warps owns one token and up to gridDim.y-th of its heads: the token's cos / sin
// table is computed once into shared memory and every warp then walks heads, a lane owning kPer
// channels of every 32 * kPer (4 consecutive ones where width, rotary half and strides allow).  A
// stream bound by HBM; a CTA per (token, head), each computing its own sines, took 60 us at 1000
// tokens of 24 + 4 heads of 256, this 23.  Token (b, t) has RoPE position positions[b] + t.
#include "common.cuh"
#include "engine.h"
#include "qk_rows.cuh"

namespace pluto {
namespace {

__device__ __forceinline__ float load_in(const void* p, size_t i, int is_bf16) {
  return is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i])
                 : static_cast<const float*>(p)[i];
}
__device__ __forceinline__ void store_out(void* p, size_t i, int is_bf16, float v) {
  if (is_bf16) static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else static_cast<float*>(p)[i] = v;
}
__device__ __forceinline__ float rnd(float v, int round) { return round ? bf16_round(v) : v; }

template <int kPer>
__device__ __forceinline__ void load_in_vec(const void* p, size_t i, int is_bf16, float* v) {
  if (kPer == 4 && is_bf16) {
    const uint2 raw = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p) + i);
    v[0] = bf16_lo(raw.x); v[1] = bf16_hi(raw.x); v[2] = bf16_lo(raw.y); v[3] = bf16_hi(raw.y);
  } else if (kPer == 4) {
    const float4 f = *reinterpret_cast<const float4*>(static_cast<const float*>(p) + i);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
    v[0] = load_in(p, i, is_bf16);
  }
}
template <int kPer>
__device__ __forceinline__ void store_out_vec(void* p, size_t i, int is_bf16, const float* v) {
  if (kPer == 4 && is_bf16)
    *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p) + i) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
  else if (kPer == 4)
    *reinterpret_cast<float4*>(static_cast<float*>(p) + i) = make_float4(v[0], v[1], v[2], v[3]);
  else
    store_out(p, i, is_bf16, v[0]);
}

template <int kPer>
__global__ void __launch_bounds__(256) qk_prepare_kernel(PrepareArgs a) {
  __shared__ float cosine[128], sine[128];
  const int heads = a.q_heads + a.kv_heads;
  const int token = blockIdx.x, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int b = token / a.tokens, t = token % a.tokens;
  const int D = a.head_dim, half = a.rotary / 2;
  const int position = (a.positions ? a.positions[b] : a.first_position) + t;
  if (static_cast<int>(threadIdx.x) < half)
    rotary_angle(position, threadIdx.x, a.log_theta, a.rotary, a.round, cosine[threadIdx.x], sine[threadIdx.x]);
  __syncthreads();
  // where the token's key/value rows go
  size_t kv_row = 0;
  void* k_dst = a.k_cache;
  void* v_dst = a.v_cache;
  if (a.k_bases != nullptr) {   // separately allocated sequences
    k_dst = const_cast<void*>(a.k_bases[b]);
    v_dst = const_cast<void*>(a.v_bases[b]);
    kv_row = static_cast<size_t>(position) * a.token_stride;
  } else {
    const int page = a.block_table ? a.block_table[static_cast<size_t>(b) * a.max_blocks + position / a.page_size] : b;
    kv_row = static_cast<size_t>(page) * a.page_stride + static_cast<size_t>(position % a.page_size) * a.token_stride;
  }
  const int stride = 8 * gridDim.y;
  for (int head = blockIdx.y * 8 + warp; head < heads; head += stride) {
    const bool is_query = head < a.q_heads;
    const int h = is_query ? head : head - a.q_heads;
    const size_t dense = (static_cast<size_t>(token) * a.kv_heads + h) * D;
    const size_t in0 = is_query ? static_cast<size_t>(token) * a.q_token + static_cast<size_t>(h) * a.q_head : dense;
    const void* in = is_query ? a.q_in : a.k_in;
    const float* norm = is_query ? a.q_norm : a.k_norm;
    float x[kRowOwn], value[kRowOwn];
#pragma unroll
    for (int i = 0; i < kRowOwn; i += kPer) {
      const int c = row_channel<kPer>(i, lane);
#pragma unroll
      for (int u = 0; u < kPer; ++u) x[i + u] = 0.0f;
      if (c < D) {
        load_in_vec<kPer>(in, in0 + c, a.in_is_bf16, x + i);
        if (!is_query) load_in_vec<kPer>(a.v_in, dense + c, a.in_is_bf16, value + i);
      }
    }
    const float inverse = rsqrtf(row_square_sum<kPer>(x, lane) / static_cast<float>(D) + a.epsilon);
#pragma unroll
    for (int i = 0; i < kRowOwn; i += kPer) {
      const int c = row_channel<kPer>(i, lane);
      if (c >= D) continue;
      float result[kPer];
#pragma unroll
      for (int u = 0; u < kPer; ++u) result[u] = rnd(x[i + u] * inverse * (1.0f + norm[c + u]), a.round);
      if (c < a.rotary) {   // kPer channels lie on one side of the half by the dispatch rule
        const int partner = c < half ? c + half : c - half;
        float p[kPer];
        load_in_vec<kPer>(in, in0 + partner, a.in_is_bf16, p);
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          float rotated = rnd(p[u] * inverse * (1.0f + norm[partner + u]), a.round);
          if (c < half) rotated = -rotated;
          const int f = (c < half ? c : c - half) + u;
          result[u] = rotate(result[u], rotated, cosine[f], sine[f], a.round);
        }
      }
      if (is_query) {
        store_out_vec<kPer>(a.q_out, (static_cast<size_t>(token) * a.q_heads + h) * D + c, a.q_out_is_bf16, result);
      } else {
        const size_t at = kv_row + static_cast<size_t>(h) * D + c;
        store_out_vec<kPer>(k_dst, at, a.kv_is_bf16, result);
#pragma unroll
        for (int u = 0; u < kPer; ++u) value[i + u] = rnd(value[i + u], a.round);
        store_out_vec<kPer>(v_dst, at, a.kv_is_bf16, value + i);
      }
    }
  }
}

}  // namespace

cudaError_t qk_prepare(cudaStream_t stream, const PrepareArgs& a) {
  const int tokens = a.batch * a.tokens, heads = a.q_heads + a.kv_heads;
  const auto aligned = [](const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
  const size_t in = a.in_is_bf16 ? 8 : 16, kv = a.kv_is_bf16 ? 8 : 16;
  // four-channel accesses: every row and the rotary halves start on a multiple of four elements
  // (separately allocated caches are only known on the device, so they take single channels)
  const bool vector = a.head_dim % 4 == 0 && a.rotary % 8 == 0 && a.q_token % 4 == 0 && a.q_head % 4 == 0 &&
                      a.token_stride % 4 == 0 && a.page_stride % 4 == 0 && a.k_bases == nullptr &&
                      aligned(a.q_in, in) && aligned(a.k_in, in) && aligned(a.v_in, in) &&
                      aligned(a.q_out, a.q_out_is_bf16 ? 8 : 16) && aligned(a.k_cache, kv) && aligned(a.v_cache, kv);
  // with fewer tokens than two per SM, a CTA for every eight heads of a token; else one CTA per token
  const int slabs = tokens < 2 * 148 ? (heads + 7) / 8 : 1;
  const dim3 grid(tokens, slabs);
  if (vector) qk_prepare_kernel<4><<<grid, 256, 0, stream>>>(a);
  else qk_prepare_kernel<1><<<grid, 256, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace pluto
