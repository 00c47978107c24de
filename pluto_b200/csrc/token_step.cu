// One token of one sequence through a decoder layer, each as a single launch: the generation loop
// of a small batch is bound by launches and by the latency of what they wait for, not by bytes.
//
//   cached_step_kernel   QwenAttentionLayer's cached forward (CachedAttentionStep,
//                        src/llm/layers/util/cached_attention_ops.cc:308-353) while the context is
//                        short: Q/K norm + RoPE, cache append, attention, output gate.
//   gdn_token_kernel     DeltaNetState::Step (cached_attention_ops.cc:355-442): convolution + SiLU,
//                        gates, recurrence, output norm and gate.
#include "common.cuh"
#include "engine.h"

namespace pluto {
namespace {

__device__ __forceinline__ float load_any(const void* p, size_t i, int is_bf16) {
  return is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]) : static_cast<const float*>(p)[i];
}
__device__ __forceinline__ void store_any(void* p, size_t i, int is_bf16, float v) {
  if (is_bf16) static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else static_cast<float*>(p)[i] = v;
}
__device__ __forceinline__ float rnd(float v, int round) { return round ? bf16_round(v) : v; }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ------------------------------------------------------------------------------------------------
// attention
// ------------------------------------------------------------------------------------------------
constexpr int kStepWarps = 16;

// kPer consecutive cache elements of a row.
template <int kPer, bool KV_BF16>
__device__ __forceinline__ void load_row(const void* base, size_t at, float (&v)[kPer]) {
  if (!KV_BF16) {
    const float* p = static_cast<const float*>(base) + at;
#pragma unroll
    for (int i = 0; i < kPer; i += 2) {
      const float2 f = *reinterpret_cast<const float2*>(p + i);
      v[i] = f.x; v[i + 1] = f.y;
    }
    return;
  }
  const __nv_bfloat16* p = static_cast<const __nv_bfloat16*>(base) + at;
  uint32_t w[kPer / 2];
  if (kPer == 8) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    w[0] = raw.x; w[1 % (kPer / 2)] = raw.y; w[2 % (kPer / 2)] = raw.z; w[3 % (kPer / 2)] = raw.w;
  } else if (kPer == 4) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    w[0] = raw.x; w[1 % (kPer / 2)] = raw.y;
  } else {
    w[0] = *reinterpret_cast<const uint32_t*>(p);
  }
#pragma unroll
  for (int i = 0; i < kPer; i += 2) { v[i] = bf16_lo(w[i / 2]); v[i + 1] = bf16_hi(w[i / 2]); }
}

// One CTA per query head, head width 32 * kPer, a lane owning kPer consecutive channels of a row.
// Every CTA prepares its query and its group's new key and value itself (the first head of a group
// writes the two into the cache); the scores of all tokens go to shared memory, so the softmax is
// two-pass fp32 as in the reference.  K and V are read once per query head: with at most
// kCachedStepTokens rows they come from L2.
template <int kPer, bool KV_BF16>
__global__ void __launch_bounds__(kStepWarps * 32) cached_step_kernel(CachedStepArgs a) {
  constexpr int D = 32 * kPer;
  __shared__ float cosine[128], sine[128], vec[3][D];   // query, new key, new value
  __shared__ float score[kCachedStepTokens];
  __shared__ float acc_s[kStepWarps][D];
  __shared__ float red[2][kStepWarps];
  const int head = blockIdx.x, group = a.q_heads / a.kv_heads, kv_head = head / group;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, c0 = lane * kPer;
  const int length = a.position + 1, half = a.rotary / 2;
  const size_t row0 = static_cast<size_t>(kv_head) * D + c0;

  pdl_wait();   // every input, the weights too: the kernel before this one may have written them
  pdl_launch_dependents();   // the next launch sets itself up meanwhile and waits for this grid in turn
  float w_norm[kPer];
  if (warp < 2) {
#pragma unroll
    for (int i = 0; i < kPer; ++i) w_norm[i] = 1.0f + (warp == 0 ? a.q_norm : a.k_norm)[c0 + i];
  }
  // The first rows of the cache and the gate of this thread's output channel are requested before
  // anything waits: at short contexts the kernel is a chain of memory round trips.
  constexpr int kAhead = 2;
  float k_ahead[kAhead][kPer], v_ahead[kAhead][kPer];
#pragma unroll
  for (int u = 0; u < kAhead; ++u) {
    const int t = warp + u * kStepWarps;
    if (t < a.position) {
      load_row<kPer, KV_BF16>(a.k_cache, static_cast<size_t>(t) * a.token_stride + row0, k_ahead[u]);
      load_row<kPer, KV_BF16>(a.v_cache, static_cast<size_t>(t) * a.token_stride + row0, v_ahead[u]);
    }
  }
  float gate = 0.0f;
  if (threadIdx.x < D) gate = load_any(a.q_gate, static_cast<size_t>(head) * 2 * D + D + threadIdx.x, a.in_is_bf16);
  if (static_cast<int>(threadIdx.x) < half) {
    const float angle = static_cast<float>(a.position) *
                        expf(static_cast<float>(threadIdx.x) * (-2.0f * a.log_theta / static_cast<float>(a.rotary)));
    cosine[threadIdx.x] = rnd(cosf(angle), a.round);
    sine[threadIdx.x] = rnd(sinf(angle), a.round);
  }
  // warp 0: query, warp 1: new key; R(x * inv * (1 + w)), then the rotation in qk_prepare.cu's steps
  float n[kPer];
  if (warp < 2) {
    const void* in = warp == 0 ? a.q_gate : a.k;
    const size_t in0 = warp == 0 ? static_cast<size_t>(head) * 2 * D : static_cast<size_t>(kv_head) * D;
    float sq = 0.0f;
#pragma unroll
    for (int i = 0; i < kPer; ++i) n[i] = load_any(in, in0 + c0 + i, a.in_is_bf16);
    // the sum of squares in qk_prepare.cu's order (four channels of every 128 per lane): the prepared
    // vectors of the two kernels are equal bit for bit
#pragma unroll
    for (int c = lane * 4; c < D; c += 128)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float x = load_any(in, in0 + c + u, a.in_is_bf16);
        sq += x * x;
      }
    const float inverse = rsqrtf(warp_sum(sq) / static_cast<float>(D) + a.epsilon);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      n[i] = rnd(n[i] * inverse * w_norm[i], a.round);
      vec[warp][c0 + i] = n[i];
    }
  } else if (warp == 2) {
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      vec[2][c0 + i] = rnd(load_any(a.v, static_cast<size_t>(kv_head) * D + c0 + i, a.in_is_bf16), a.round);
  }
  __syncthreads();
  if (warp < 2) {
    float result[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int c = c0 + i;
      result[i] = n[i];
      if (c < a.rotary) {
        const int f = c < half ? c : c - half;
        const float partner = c < half ? -vec[warp][c + half] : vec[warp][c - half];
        result[i] = rnd(rnd(n[i] * cosine[f], a.round) + rnd(partner * sine[f], a.round), a.round);
      }
    }
    __syncwarp();   // every partner has been read
#pragma unroll
    for (int i = 0; i < kPer; ++i) vec[warp][c0 + i] = result[i];
    if (warp == 1 && head % group == 0) {
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        store_any(a.k_cache, static_cast<size_t>(a.position) * a.token_stride + row0 + i, KV_BF16, result[i]);
    }
  } else if (warp == 2 && head % group == 0) {
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      store_any(a.v_cache, static_cast<size_t>(a.position) * a.token_stride + row0 + i, KV_BF16, vec[2][c0 + i]);
  }
  __syncthreads();

  float q[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) q[i] = vec[0][c0 + i];
  float top = -INFINITY;
  auto attend = [&](int t, const float (&k)[kPer]) {
    float dot = 0.0f;
#pragma unroll
    for (int i = 0; i < kPer; ++i) dot = fmaf(k[i], q[i], dot);
    dot = warp_sum(dot) * a.scale;
    if (lane == 0) score[t] = dot;
    top = fmaxf(top, dot);
  };
#pragma unroll
  for (int u = 0; u < kAhead; ++u)
    if (warp + u * kStepWarps < a.position) attend(warp + u * kStepWarps, k_ahead[u]);
#pragma unroll 8
  for (int t = warp + kAhead * kStepWarps; t < a.position; t += kStepWarps) {
    float k[kPer];
    load_row<kPer, KV_BF16>(a.k_cache, static_cast<size_t>(t) * a.token_stride + row0, k);
    attend(t, k);
  }
  if (warp == a.position % kStepWarps) {   // the new token, as the cache holds it
    float dot = 0.0f;
#pragma unroll
    for (int i = 0; i < kPer; ++i) dot = fmaf(rnd(vec[1][c0 + i], KV_BF16), q[i], dot);
    dot = warp_sum(dot) * a.scale;
    if (lane == 0) score[a.position] = dot;
    top = fmaxf(top, dot);
  }
  if (lane == 0) red[0][warp] = top;
  __syncthreads();
  top = red[0][0];
#pragma unroll
  for (int w = 1; w < kStepWarps; ++w) top = fmaxf(top, red[0][w]);
  float sum = 0.0f;
  for (int t = threadIdx.x; t < length; t += kStepWarps * 32) {
    const float p = expf(score[t] - top);
    score[t] = p;
    sum += p;
  }
  sum = warp_sum(sum);
  if (lane == 0) red[1][warp] = sum;
  __syncthreads();

  float acc[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) acc[i] = 0.0f;
#pragma unroll
  for (int u = 0; u < kAhead; ++u)
    if (warp + u * kStepWarps < a.position) {
      const float p = score[warp + u * kStepWarps];
#pragma unroll
      for (int i = 0; i < kPer; ++i) acc[i] = fmaf(p, v_ahead[u][i], acc[i]);
    }
#pragma unroll 8
  for (int t = warp + kAhead * kStepWarps; t < a.position; t += kStepWarps) {
    float v[kPer];
    load_row<kPer, KV_BF16>(a.v_cache, static_cast<size_t>(t) * a.token_stride + row0, v);
    const float p = score[t];
#pragma unroll
    for (int i = 0; i < kPer; ++i) acc[i] = fmaf(p, v[i], acc[i]);
  }
  if (warp == a.position % kStepWarps) {
#pragma unroll
    for (int i = 0; i < kPer; ++i) acc[i] = fmaf(score[a.position], rnd(vec[2][c0 + i], KV_BF16), acc[i]);
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i) acc_s[warp][c0 + i] = acc[i];
  __syncthreads();
  if (threadIdx.x >= D) return;
  // the warps' parts in double (a warp holds few terms at these lengths): the quotient is then good to
  // the last bit, and its rounding to bf16 falls where the exact result's would
  double parts = 0.0, total = 0.0;
#pragma unroll
  for (int w = 0; w < kStepWarps; ++w) {
    parts += static_cast<double>(acc_s[w][threadIdx.x]);
    total += static_cast<double>(red[1][w]);
  }
  float value = rnd(static_cast<float>(parts / total), a.round);
  value = rnd(value * rnd(1.0f / (1.0f + expf(-gate)), a.round), a.round);
  store_any(a.out, static_cast<size_t>(head) * D + threadIdx.x, a.out_is_bf16, value);
}

// ------------------------------------------------------------------------------------------------
// gated delta-net, widths 128.  One CTA of 16 warps per value head; warp w owns rows [8 w, 8 w + 8)
// of the state, a lane four columns of each (16-byte accesses, the state crosses HBM once each way:
// requested first, stored last).  The value heads of a key head share its q and k channels: each
// CTA convolves them for itself, they form a cluster, and the first of them replaces the window
// once all have read it.
// ------------------------------------------------------------------------------------------------
constexpr int kDim = 128, kTokenThreads = 512, kMaxTaps = 4;

__global__ void __launch_bounds__(kTokenThreads) gdn_token_kernel(GdnTokenArgs a) {
  const int h = blockIdx.x, group = a.value_heads / a.key_heads, kh = h / group;
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  __shared__ float qkv[3][kDim];           // convolved q, k, v
  __shared__ float4 column[16][kDim / 4];  // per-warp column sums
  __shared__ float delta_s[kDim], gates[2], red[4];

  pdl_wait();   // every input, the weights too: the kernel before this one may have written them
  pdl_launch_dependents();
  const int part = tid / kDim, i = tid % kDim;   // threads 0..383: one channel of q, k, v each
  const int channel = part == 2 ? 2 * a.key_heads * kDim + h * kDim + i : (part * a.key_heads + kh) * kDim + i;
  float w[kMaxTaps], norm = 0.0f;
  if (tid < 3 * kDim) {
#pragma unroll
    for (int tap = 0; tap < kMaxTaps; ++tap)
      w[tap] = tap < a.width ? a.conv_weight[static_cast<size_t>(channel) * a.width + tap] : 0.0f;
    if (part == 0) norm = a.norm_weight[i];
  }
  float4 S[8];
  float* state = a.state + static_cast<size_t>(h) * kDim * kDim + warp * 8 * kDim + lane * 4;
#pragma unroll
  for (int r = 0; r < 8; ++r) S[r] = *reinterpret_cast<const float4*>(state + r * kDim);

  float window[kMaxTaps];
  float z = 0.0f;
  if (tid < 3 * kDim) {
    const float* own = a.conv_state + static_cast<size_t>(channel) * a.width;
    float sum = 0.0f;
#pragma unroll
    for (int tap = 0; tap < kMaxTaps; ++tap) {
      if (tap + 1 < a.width) {
        window[tap] = own[tap + 1];
        sum += window[tap] * w[tap];
      } else if (tap + 1 == a.width) {
        window[tap] = rnd(load_any(a.qkv, channel, a.qkv_is_bf16), a.round);
        sum = rnd(sum + window[tap] * w[tap], a.round);
      }
    }
    qkv[part][i] = rnd(sum / (1.0f + expf(-sum)), a.round);
    if (part == 0) {   // the threads that finish the row
      z = load_any(a.z, static_cast<size_t>(h) * kDim + i, a.z_is_bf16);
    }
  } else if (tid == 3 * kDim) {
    const float alpha = load_any(a.a_in, h, a.ab_is_bf16) + a.dt_bias[h];
    const float softplus = fmaxf(alpha, 0.0f) + logf(1.0f + expf(-fabsf(alpha)));
    gates[0] = expf(-expf(a.a_log[h]) * softplus);
    gates[1] = rnd(1.0f / (1.0f + expf(-load_any(a.b_in, h, a.ab_is_bf16))), a.round);
  }
  if (group > 1) cluster_arrive();   // this CTA has read the shared windows
  __syncthreads();
  if (warp < 2) {   // L2 norms; the query also carries 1 / sqrt(128)
    float x[4], ss = 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      x[u] = qkv[warp][lane + 32 * u];
      ss += x[u] * x[u];
    }
    float f = rsqrtf(warp_sum(ss) + 1e-6f);
    if (warp == 0) f = f / sqrtf(static_cast<float>(kDim));
#pragma unroll
    for (int u = 0; u < 4; ++u) qkv[warp][lane + 32 * u] = x[u] * f;
  }
  __syncthreads();
  const float decay = gates[0], beta = gates[1];
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const float k = qkv[1][warp * 8 + r];
    S[r].x *= decay; S[r].y *= decay; S[r].z *= decay; S[r].w *= decay;
    sum.x = fmaf(S[r].x, k, sum.x); sum.y = fmaf(S[r].y, k, sum.y);
    sum.z = fmaf(S[r].z, k, sum.z); sum.w = fmaf(S[r].w, k, sum.w);
  }
  column[warp][lane] = sum;
  __syncthreads();
  const float* columns = reinterpret_cast<const float*>(column);
  if (tid < kDim) {
    float prediction = 0.0f;
#pragma unroll
    for (int w = 0; w < 16; ++w) prediction += columns[w * kDim + tid];
    delta_s[tid] = (qkv[2][tid] - prediction) * beta;
  }
  __syncthreads();
  const float4 delta = reinterpret_cast<const float4*>(delta_s)[lane];
  sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const float k = qkv[1][warp * 8 + r], q = qkv[0][warp * 8 + r];
    S[r].x = fmaf(k, delta.x, S[r].x); S[r].y = fmaf(k, delta.y, S[r].y);
    S[r].z = fmaf(k, delta.z, S[r].z); S[r].w = fmaf(k, delta.w, S[r].w);
    sum.x = fmaf(S[r].x, q, sum.x); sum.y = fmaf(S[r].y, q, sum.y);
    sum.z = fmaf(S[r].z, q, sum.z); sum.w = fmaf(S[r].w, q, sum.w);
    *reinterpret_cast<float4*>(state + r * kDim) = S[r];
  }
  column[warp][lane] = sum;
  __syncthreads();
  float core = 0.0f;
  if (tid < kDim) {
#pragma unroll
    for (int w = 0; w < 16; ++w) core += columns[w * kDim + tid];
    core = rnd(core, a.round);
    const float sq = warp_sum(core * core);
    if (lane == 0) red[warp] = sq;
  }
  __syncthreads();
  if (tid < kDim) {
    const float inverse = rsqrtf((red[0] + red[1] + red[2] + red[3]) / static_cast<float>(kDim) + a.epsilon);
    const float affine = rnd(rnd(core * inverse, a.round) * norm, a.round);
    store_any(a.out, static_cast<size_t>(h) * kDim + i, a.out_is_bf16, rnd(affine * (z / (1.0f + expf(-z))), a.round));
  }
  if (group > 1) cluster_wait();     // everyone has read the shared windows
  if (tid < 3 * kDim && (part == 2 || h % group == 0)) {
    float* own = a.conv_state + static_cast<size_t>(channel) * a.width;
#pragma unroll
    for (int tap = 0; tap < kMaxTaps; ++tap)
      if (tap < a.width) own[tap] = window[tap];
  }
}

}  // namespace

bool cached_step_supported(const CachedStepArgs& a) {
  return (a.head_dim == 64 || a.head_dim == 128 || a.head_dim == 256) && a.position < kCachedStepTokens &&
         a.token_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(a.k_cache) & 15u) == 0 &&
         (reinterpret_cast<uintptr_t>(a.v_cache) & 15u) == 0;
}

cudaError_t cached_step(cudaStream_t stream, const CachedStepArgs& a) {
  using Kernel = void (*)(CachedStepArgs);
  static const Kernel kernels[3][2] = {{cached_step_kernel<2, false>, cached_step_kernel<2, true>},
                                       {cached_step_kernel<4, false>, cached_step_kernel<4, true>},
                                       {cached_step_kernel<8, false>, cached_step_kernel<8, true>}};
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(a.q_heads);
  config.blockDim = dim3(kStepWarps * 32);
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernels[a.head_dim / 128][a.kv_is_bf16 ? 1 : 0], a);
}

bool gdn_token_supported(int key_heads, int value_heads, int key_dim, int value_dim, int width) {
  return key_dim == kDim && value_dim == kDim && width <= kMaxTaps && value_heads / key_heads <= 8;
}

cudaError_t gdn_token(cudaStream_t stream, const GdnTokenArgs& a) {
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = static_cast<unsigned>(a.value_heads / a.key_heads);
  attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(a.value_heads);
  config.blockDim = dim3(kTokenThreads);
  config.stream = stream;
  config.attrs = attributes;
  config.numAttrs = 2;
  return cudaLaunchKernelEx(&config, gdn_token_kernel, a);
}

}  // namespace pluto
