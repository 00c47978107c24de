// Elementwise pieces of the Qwen sequence-attention backward
// (src/llm/layers/qwen_attention.cc:120-239): the sigmoid output gate, the inverse partial RoPE
// followed by the per-head RMSNorm backward, and the deterministic reduction of the shared
// norm-weight gradient.  The attention core between them runs in attn_generic.cu
// (gqa_generic_bwd).  Head width <= 256.
#include "common.cuh"
#include "engine.h"

namespace pluto {
namespace {

__device__ __forceinline__ float rnd(float v, int round) { return round ? bf16_round(v) : v; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// GateBackwardKernel (:123-138): dc = dy * R(sigmoid(gate)); d_gate = dy * R(core) * s * (1 - s),
// s in fp32.  Also the row term of the softmax backward, delta = dc . core with the unrounded
// core (QueryBackwardKernel :153-155), so the core pass only reads it.
// One warp per (token, head), eight per CTA; a lane covers kPer consecutive channels per step of
// 32 * kPer (kPer = 4 with 16-byte accesses when the width and strides allow it).
template <int kPer>
__global__ void __launch_bounds__(256) gate_bwd_kernel(GateBwdArgs a, long long rows) {
  const long long row = static_cast<long long>(blockIdx.x) * 8 + threadIdx.x / 32;
  if (row >= rows) return;
  const int lane = threadIdx.x % 32, D = a.head_dim;
  const long long token = row / a.q_heads;
  const int h = static_cast<int>(row % a.q_heads);
  const int b = static_cast<int>(token / a.seq), s = static_cast<int>(token % a.seq);
  const size_t dense = static_cast<size_t>(row) * D;
  const __nv_bfloat16* gate = a.gate + static_cast<size_t>(token) * a.gate_token + static_cast<size_t>(h) * a.gate_head;
  float* d_gate = a.d_gate + static_cast<size_t>(token) * a.dgate_token + static_cast<size_t>(h) * a.dgate_head;
  float part = 0.0f;
  for (int c0 = lane * kPer; c0 < D; c0 += 32 * kPer) {
    float g[kPer], grad[kPer], core[kPer], dc[kPer], dg[kPer];
    if (kPer == 4) {
      const uint2 raw = *reinterpret_cast<const uint2*>(gate + c0);
      g[0] = bf16_lo(raw.x); g[1] = bf16_hi(raw.x); g[2] = bf16_lo(raw.y); g[3] = bf16_hi(raw.y);
      const float4 y = *reinterpret_cast<const float4*>(a.dy + dense + c0);
      const float4 c = *reinterpret_cast<const float4*>(a.core + dense + c0);
      grad[0] = y.x; grad[1] = y.y; grad[2] = y.z; grad[3] = y.w;
      core[0] = c.x; core[1] = c.y; core[2] = c.z; core[3] = c.w;
    } else {
      g[0] = __bfloat162float(gate[c0]);
      grad[0] = a.dy[dense + c0];
      core[0] = a.core[dense + c0];
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const float s = sigmoid(g[i]);
      dc[i] = grad[i] * rnd(s, a.round);
      dg[i] = grad[i] * rnd(core[i], a.round) * s * (1.0f - s);
      part = fmaf(dc[i], core[i], part);
    }
    if (kPer == 4) {
      *reinterpret_cast<float4*>(a.dc + dense + c0) = make_float4(dc[0], dc[1], dc[2], dc[3]);
      *reinterpret_cast<float4*>(d_gate + c0) = make_float4(dg[0], dg[1], dg[2], dg[3]);
    } else {
      a.dc[dense + c0] = dc[0];
      d_gate[c0] = dg[0];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) a.deltas[(static_cast<size_t>(b) * a.q_heads + h) * a.seq + s] = part;
}

// NormBackwardKernel (:196-226): rotate the gradient back with the rounded cos/sin of the forward,
// then the RMSNorm backward; `parts` (optional) receives one row per CTA of the sums of
// normalized_grad * x * inv, the norm-weight gradient.
// A CTA walks blocks of `per_block` tokens: their cos / sin tables go to shared memory, then every
// warp takes (token, head) rows, a lane owning kPer channels of every 32 * kPer.  HBM bound; the
// earlier form (a CTA per row with its own sines, the per-row parts written out and reduced from
// memory by 24 CTAs) took 64 + 71 us at 1000 tokens of 24 and 4 heads of 256, this 24 + 10.
constexpr int kBlockTokens = 8;   // tokens of one block when a token has a single head
template <int kPer>
__global__ void __launch_bounds__(256, 4) norm_bwd_kernel(NormBwdArgs a, int per_block) {
  constexpr int kOwn = 8;   // channels a lane owns at width 256
  __shared__ float cosine[kBlockTokens][128], sine[kBlockTokens][128];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int D = a.head_dim, half = a.rotary / 2, tokens = a.batch * a.tokens;
  auto channel = [&](int i) { return (i / kPer) * 32 * kPer + lane * kPer; };   // first of the kPer at i
  float weight[kOwn], sum[kOwn];
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    const int c = channel(i) + i % kPer;
    weight[i] = c < D ? 1.0f + a.weight[c] : 0.0f;
    sum[i] = 0.0f;
  }
  for (int first = blockIdx.x * per_block; first < tokens; first += gridDim.x * per_block) {
    const int count = min(per_block, tokens - first);
    __syncthreads();   // the previous block's rows are done with the tables
    for (int i = threadIdx.x; i < count * half; i += 256) {
      const int token = first + i / half, f = i % half;
      const int position = (a.positions ? a.positions[token / a.tokens] : 0) + token % a.tokens;
      const float angle = static_cast<float>(position) *
                          expf(static_cast<float>(f) * (-2.0f * a.log_theta / static_cast<float>(a.rotary)));
      cosine[i / half][f] = rnd(cosf(angle), a.round);
      sine[i / half][f] = rnd(sinf(angle), a.round);
    }
    __syncthreads();
    for (int row = warp; row < count * a.heads; row += 8) {
      const int own = row / a.heads, token = first + own, h = row % a.heads;
      const size_t dense = (static_cast<size_t>(token) * a.heads + h) * D;
      const __nv_bfloat16* in = a.x + static_cast<size_t>(token) * a.x_token + static_cast<size_t>(h) * a.x_head;
      float* out = a.dx + static_cast<size_t>(token) * a.dx_token + static_cast<size_t>(h) * a.dx_head;
      float x[kOwn], ng[kOwn];
      float sq = 0.0f;
#pragma unroll
      for (int i = 0; i < kOwn; i += kPer) {
        const int c = channel(i);
#pragma unroll
        for (int u = 0; u < kPer; ++u) x[i + u] = ng[i + u] = 0.0f;
        if (c >= D) continue;
        if (kPer == 4) {
          const uint2 raw = *reinterpret_cast<const uint2*>(in + c);
          x[i] = bf16_lo(raw.x); x[i + 1] = bf16_hi(raw.x); x[i + 2] = bf16_lo(raw.y); x[i + 3] = bf16_hi(raw.y);
          const float4 g = *reinterpret_cast<const float4*>(a.grad + dense + c);
          ng[i] = g.x; ng[i + 1] = g.y; ng[i + 2] = g.z; ng[i + 3] = g.w;
        } else {
          x[i] = __bfloat162float(in[c]);
          ng[i] = a.grad[dense + c];
        }
#pragma unroll
        for (int u = 0; u < kPer; ++u) sq += x[i + u] * x[i + u];
        if (c < a.rotary) {
          float p[kPer];
          const size_t partner = dense + (c < half ? c + half : c - half);
          if (kPer == 4) {
            const float4 g = *reinterpret_cast<const float4*>(a.grad + partner);
            p[0] = g.x; p[1] = g.y; p[2] = g.z; p[3] = g.w;
          } else {
            p[0] = a.grad[partner];
          }
#pragma unroll
          for (int u = 0; u < kPer; ++u) {
            const int f = (c < half ? c : c - half) + u;
            ng[i + u] = ng[i + u] * cosine[own][f] + (c < half ? p[u] * sine[own][f] : -p[u] * sine[own][f]);
          }
        }
      }
      const float inv = rsqrtf(warp_sum(sq) / static_cast<float>(D) + a.epsilon);
      float dot = 0.0f;
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        dot += ng[i] * weight[i] * x[i];
        sum[i] = fmaf(ng[i] * x[i], inv, sum[i]);
      }
      dot = warp_sum(dot);
      const float scale = inv * inv * inv / static_cast<float>(D);
#pragma unroll
      for (int i = 0; i < kOwn; i += kPer) {
        const int c = channel(i);
        if (c >= D) continue;
        float dx[kPer];
#pragma unroll
        for (int u = 0; u < kPer; ++u) dx[u] = inv * (ng[i + u] * weight[i + u]) - x[i + u] * scale * dot;
        if (kPer == 4) *reinterpret_cast<float4*>(out + c) = make_float4(dx[0], dx[1], dx[2], dx[3]);
        else out[c] = dx[0];
      }
    }
  }
  if (a.parts == nullptr) return;
  __shared__ float strip[8][256];
#pragma unroll
  for (int i = 0; i < kOwn; ++i)
    if (channel(i) + i % kPer < D) strip[warp][channel(i) + i % kPer] = sum[i];
  __syncthreads();
  if (static_cast<int>(threadIdx.x) < D) {
    float total = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) total += strip[i][threadIdx.x];
    a.parts[static_cast<size_t>(blockIdx.x) * D + threadIdx.x] = total;
  }
}

// dst[c] += sum over the strips of parts[strip, c], in a fixed order: a CTA per 32 columns, whose 32
// warps take contiguous runs of the strips and add the runs' sums in order.
__global__ void __launch_bounds__(1024) reduce_strips_kernel(const float* __restrict__ parts, int strips, int dim,
                                                             float* dst) {
  __shared__ float run_sum[32][32];
  const int lane = threadIdx.x % 32, run = threadIdx.x / 32, c = blockIdx.x * 32 + lane;
  const int length = (strips + 31) / 32;
  float sum = 0.0f;
  if (c < dim) {
#pragma unroll 8
    for (int s = run * length; s < min(strips, (run + 1) * length); ++s) sum += parts[static_cast<size_t>(s) * dim + c];
  }
  run_sum[run][lane] = sum;
  __syncthreads();
  if (run != 0 || c >= dim) return;
#pragma unroll
  for (int i = 1; i < 32; ++i) sum += run_sum[i][lane];
  dst[c] += sum;
}

}  // namespace

cudaError_t gqa_gate_bwd(cudaStream_t stream, const GateBwdArgs& a) {
  const long long rows = static_cast<long long>(a.batch) * a.seq * a.q_heads;
  const unsigned blocks = static_cast<unsigned>((rows + 7) / 8);
  const auto aligned = [](const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
  const bool vector = a.head_dim % 4 == 0 && a.gate_token % 4 == 0 && a.gate_head % 4 == 0 &&
                      a.dgate_token % 4 == 0 && a.dgate_head % 4 == 0 && aligned(a.gate, 8) &&
                      aligned(a.dy, 16) && aligned(a.core, 16) && aligned(a.dc, 16) &&
                      aligned(a.d_gate, 16);
  if (vector) gate_bwd_kernel<4><<<blocks, 256, 0, stream>>>(a, rows);
  else gate_bwd_kernel<1><<<blocks, 256, 0, stream>>>(a, rows);
  return cudaGetLastError();
}

namespace {
int norm_block_tokens(int heads) { return heads >= kBlockTokens ? 1 : kBlockTokens / heads; }
int norm_strips(long long rows, int heads) {   // CTAs of the norm backward, and rows of its partial sums
  const long long per_block = norm_block_tokens(heads), tokens = rows / heads;
  const long long blocks = (tokens + per_block - 1) / per_block;
  return static_cast<int>(blocks < 4 * 148 ? blocks : 4 * 148);
}
}  // namespace

size_t qk_prepare_bwd_workspace_bytes(long long rows, int heads, int head_dim) {
  return static_cast<size_t>(norm_strips(rows, heads)) * head_dim * sizeof(float);
}

cudaError_t qk_prepare_bwd(cudaStream_t stream, NormBwdArgs a, float* d_weight, void* workspace) {
  const long long rows = static_cast<long long>(a.batch) * a.tokens * a.heads;
  a.parts = d_weight ? static_cast<float*>(workspace) : nullptr;
  const int strips = norm_strips(rows, a.heads);
  const auto aligned = [](const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
  // four-channel accesses: every row and the rotary halves start on a multiple of four elements
  const bool vector = a.head_dim % 4 == 0 && a.rotary % 8 == 0 && a.x_token % 4 == 0 && a.x_head % 4 == 0 &&
                      a.dx_token % 4 == 0 && a.dx_head % 4 == 0 && aligned(a.x, 8) && aligned(a.grad, 16) &&
                      aligned(a.dx, 16);
  auto kernel = vector ? norm_bwd_kernel<4> : norm_bwd_kernel<1>;
  kernel<<<strips, 256, 0, stream>>>(a, norm_block_tokens(a.heads));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || d_weight == nullptr) return e;
  return reduce_strips_accumulate(stream, a.parts, strips, a.head_dim, d_weight);
}

cudaError_t reduce_strips_accumulate(cudaStream_t stream, const float* parts, int strips, int dim, float* dst) {
  reduce_strips_kernel<<<(dim + 31) / 32, 1024, 0, stream>>>(parts, strips, dim, dst);
  return cudaGetLastError();
}

}  // namespace pluto
