// Gated delta-net: the token-sequential recurrence with the state held on chip, plus the small
// operators either side of it.
//
// Reference kernels these stand in for:
//   DeltaRecurrenceKernel      src/llm/layers/util/cached_attention_ops.cc:205-251  (one token)
//   RecurrenceForward          src/llm/layers/sequence_delta_net.cc:55-102          (a sequence)
//   ConvolutionKernel          cached_attention_ops.cc:180-203,  ConvForward  sequence_delta_net.cc:31-51
//   DeltaOutputKernel          cached_attention_ops.cc:253-272,  OutputForward sequence_delta_net.cc:104-121
// The reference streams a [128 x 32] fp32 slice of the state through HBM for every token and, in
// the sequence layer, stores every intermediate state.  gdn_recurrent keeps a [dk x 32] slice in
// registers for the whole sequence: the state is read once and written once per launch, only the
// token vectors stream in.  The arithmetic per token is the reference's, in its order:
//     S <- g S;  delta = (v - S^T k) * beta;  S <- S + k (x) delta;  o = R(S^T q)
#include "common.cuh"
#include "engine.h"

namespace pluto {
namespace {

__device__ __forceinline__ float load_any(const void* p, size_t i, int is_bf16) {
  return is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i])
                 : static_cast<const float*>(p)[i];
}
__device__ __forceinline__ void store_any(void* p, size_t i, int is_bf16, float v) {
  if (is_bf16) static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else static_cast<float*>(p)[i] = v;
}
__device__ __forceinline__ float rnd(float v, int round) { return round ? bf16_round(v) : v; }

constexpr int kSlice = 32;    // value columns per CTA
constexpr int kRowGroups = 4; // each thread owns 32 key rows of one column
constexpr int kBlockT = 16;   // tokens staged per shared-memory block
constexpr int kRecThreads = kSlice * kRowGroups;  // 128

// grid (ceil(dv / 32), value heads, batch)
__global__ void __launch_bounds__(kRecThreads) gdn_recurrent_kernel(GdnArgs a) {
  const int slice = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int kh = h / (a.value_heads / a.key_heads);
  const int dk = a.key_dim, dv = a.value_dim;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  // lane = (column % 8) * 4 + row group, so the 4 partial sums of a column sit in one quad
  const int rg = lane & 3;
  const int col = slice * kSlice + warp * 8 + (lane >> 2);
  const bool col_ok = col < dv;

  __shared__ float sq[2][kBlockT][128];
  __shared__ float sk[2][kBlockT][128];
  __shared__ float sv[2][kBlockT][kSlice];
  __shared__ float sg[2][kBlockT], sb[2][kBlockT];

  float S[32];
  float* state = a.state + ((static_cast<size_t>(b) * a.value_heads + h) * dk) * dv;
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const int row = rg * 32 + r;
    S[r] = (col_ok && row < dk) ? state[static_cast<size_t>(row) * dv + col] : 0.0f;
  }

  auto stage = [&](int buf, int t0) {
    // q, k vectors of up to kBlockT tokens (normalised here), this slice of v, the two gates; a
    // single-token step stages one token, not sixteen
    const int n_tok = min(kBlockT, a.tokens - t0);
    for (int idx = threadIdx.x; idx < n_tok * 128; idx += kRecThreads) {
      const int tt = idx / 128, i = idx % 128, t = t0 + tt;
      float qv = 0.0f, kv = 0.0f;
      if (t < a.tokens && i < dk) {
        const size_t off = (static_cast<size_t>(b) * a.tokens + t) * a.qk_token + static_cast<size_t>(kh) * dk + i;
        qv = load_any(a.q, off, a.in_is_bf16);
        kv = load_any(a.k, off, a.in_is_bf16);
      }
      sq[buf][tt][i] = qv;
      sk[buf][tt][i] = kv;
    }
    for (int idx = threadIdx.x; idx < n_tok * kSlice; idx += kRecThreads) {
      const int tt = idx / kSlice, j = idx % kSlice, t = t0 + tt, c = slice * kSlice + j;
      float x = 0.0f;
      if (t < a.tokens && c < dv)
        x = load_any(a.v, (static_cast<size_t>(b) * a.tokens + t) * a.v_token + static_cast<size_t>(h) * dv + c,
                     a.in_is_bf16);
      sv[buf][tt][j] = x;
    }
    if (threadIdx.x < n_tok) {
      const int t = t0 + threadIdx.x;
      const size_t off = (static_cast<size_t>(b) * a.tokens + min(t, a.tokens - 1)) * a.value_heads + h;
      sg[buf][threadIdx.x] = a.g[off];
      sb[buf][threadIdx.x] = a.beta[off];
    }
  };
  auto normalise = [&](int buf, int t0) {
    // vectors 0 .. n_tok-1 are the queries, n_tok .. 2 n_tok - 1 the keys; lane covers 4 channels
    const int n_tok = min(kBlockT, a.tokens - t0);
    for (int v = warp; v < 2 * n_tok; v += 4) {
      const bool is_query = v < n_tok;
      float* vec = is_query ? sq[buf][v] : sk[buf][v - n_tok];
      float x[4], ss = 0.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i) { x[i] = vec[lane + 32 * i]; ss += x[i] * x[i]; }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      float f;
      if (a.normalize_qk) {
        f = rsqrtf(ss + 1e-6f);
        if (is_query) f = f / sqrtf(static_cast<float>(dk));
      } else {
        f = is_query ? a.q_scale : 1.0f;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) vec[lane + 32 * i] = x[i] * f;
    }
  };

  stage(0, 0);
  __syncthreads();
  normalise(0, 0);
  __syncthreads();
  const int blocks = (a.tokens + kBlockT - 1) / kBlockT;
  for (int blk = 0; blk < blocks; ++blk) {
    const int buf = blk & 1;
    if (blk + 1 < blocks) stage(buf ^ 1, (blk + 1) * kBlockT);
    const int count = min(kBlockT, a.tokens - blk * kBlockT);
    for (int tt = 0; tt < count; ++tt) {
      const float decay = sg[buf][tt], beta = sb[buf][tt];
      const float* kvec = &sk[buf][tt][rg * 32];
      const float* qvec = &sq[buf][tt][rg * 32];
      float prediction = 0.0f;
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        S[r] *= decay;
        prediction = fmaf(S[r], kvec[r], prediction);
      }
      prediction += __shfl_xor_sync(0xffffffffu, prediction, 1);
      prediction += __shfl_xor_sync(0xffffffffu, prediction, 2);
      const float delta = (sv[buf][tt][warp * 8 + (lane >> 2)] - prediction) * beta;
      float core = 0.0f;
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        S[r] = fmaf(kvec[r], delta, S[r]);
        core = fmaf(S[r], qvec[r], core);
      }
      core += __shfl_xor_sync(0xffffffffu, core, 1);
      core += __shfl_xor_sync(0xffffffffu, core, 2);
      if (rg == 0 && col_ok) {
        const int t = blk * kBlockT + tt;
        store_any(a.out, ((static_cast<size_t>(b) * a.tokens + t) * a.value_heads + h) * dv + col,
                  a.out_is_bf16, rnd(core, a.round));
      }
    }
    __syncthreads();
    if (blk + 1 < blocks) {
      normalise(buf ^ 1, (blk + 1) * kBlockT);
      __syncthreads();
    }
  }
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const int row = rg * 32 + r;
    if (col_ok && row < dk) state[static_cast<size_t>(row) * dv + col] = S[r];
  }
}

// g = exp(-exp(A_log) * softplus(a + dt_bias)),  beta = R(sigmoid(b));  one thread per (token, head)
__global__ void gdn_gates_kernel(const void* a_in, const void* b_in, const float* a_log,
                                 const float* dt_bias, int in_is_bf16, long long count, int heads,
                                 int round, float* g, float* beta) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int h = static_cast<int>(i % heads);
  const float alpha = load_any(a_in, i, in_is_bf16) + dt_bias[h];
  const float softplus = fmaxf(alpha, 0.0f) + logf(1.0f + expf(-fabsf(alpha)));
  g[i] = expf(-expf(a_log[h]) * softplus);
  beta[i] = rnd(sigmoid(load_any(b_in, i, in_is_bf16)), round);
}

// Causal depthwise convolution + SiLU over a sequence with an explicit history:
// `state` [B, channels, width] holds the last `width` inputs (oldest first; zero for a fresh
// sequence).  y_t = R(SiLU(R(sum_tap w[c][tap] * x[t + tap - width + 1]))) with inputs rounded
// first; on return the state holds the last `width` inputs of this call (the reference's
// shift register).  One thread per (batch, channel), sequential in t: windows wider than four
// taps, channel counts that are not a multiple of four, single tokens, and output over the input.
__global__ void gdn_conv_kernel(const void* input, const float* weight, int in_is_bf16, int batch,
                                int tokens, int channels, int width, int round, float* state,
                                void* output, int out_is_bf16) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<long long>(batch) * channels) return;
  const int b = static_cast<int>(i / channels), c = static_cast<int>(i % channels);
  float window[32], w[32];
  for (int tap = 0; tap < width; ++tap) {
    window[tap] = state[(static_cast<size_t>(b) * channels + c) * width + tap];
    w[tap] = weight[static_cast<size_t>(c) * width + tap];
  }
  for (int t = 0; t < tokens; ++t) {
    const size_t idx = (static_cast<size_t>(b) * tokens + t) * channels + c;
    float sum = 0.0f;
    for (int tap = 0; tap < width - 1; ++tap) {
      window[tap] = window[tap + 1];
      sum += window[tap] * w[tap];
    }
    const float current = rnd(load_any(input, idx, in_is_bf16), round);
    window[width - 1] = current;
    sum = rnd(sum + current * w[width - 1], round);
    store_any(output, idx, out_is_bf16, rnd(silu(sum), round));
  }
  for (int tap = 0; tap < width; ++tap)
    state[(static_cast<size_t>(b) * channels + c) * width + tap] = window[tap];
}

// Four consecutive elements of a bf16 or fp32 array (8- or 16-byte access).
template <bool BF16>
__device__ __forceinline__ float4 load_four(const void* p, size_t i) {
  if (BF16) {
    const uint2 raw = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p) + i);
    return make_float4(bf16_lo(raw.x), bf16_hi(raw.x), bf16_lo(raw.y), bf16_hi(raw.y));
  }
  return *reinterpret_cast<const float4*>(static_cast<const float*>(p) + i);
}
template <bool BF16>
__device__ __forceinline__ void store_four(void* p, size_t i, const float (&v)[4]) {
  if (BF16)
    *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p) + i) =
        make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
  else
    *reinterpret_cast<float4*>(static_cast<float*>(p) + i) = make_float4(v[0], v[1], v[2], v[3]);
}

// The same convolution cut along the tokens: a thread owns four channels of kConvSegment tokens,
// with the window in registers.  It is a stream (every input and output element once), so what
// counts is that there are enough threads to keep HBM busy: one thread per channel walked all
// tokens of a sequence by itself, 80 CTAs of dependent loads (565 us at 1000 tokens x 10240
// channels; 31 us in this form, 17 before the SiLU had an IEEE division).  Segment 0 is the only reader of the state, so it also writes the
// new one: it never races with a later segment, which takes its history from the input.
constexpr int kConvSegment = 16;
template <int W, bool IN_BF16, bool OUT_BF16>
__global__ void __launch_bounds__(128, 8) gdn_conv_segment_kernel(const void* __restrict__ input,
                                                               const float* __restrict__ weight, int tokens,
                                                               int channels, int round, float* state,
                                                               void* __restrict__ output) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (c >= channels) return;
  // (a bf16 input is rounded already, and a bf16 output is rounded by its store)
  auto rounded_in = [&](float v) { return IN_BF16 ? v : rnd(v, round); };
  const int b = blockIdx.z, t0 = blockIdx.y * kConvSegment, t1 = min(tokens, t0 + kConvSegment);
  const size_t seq = static_cast<size_t>(b) * tokens * channels + c;
  float* own_state = state + (static_cast<size_t>(b) * channels + c) * W;   // [4][W]
  float w[4][W], x[W][4];   // x[W-1] is the current token
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int tap = 0; tap < W; ++tap) w[i][tap] = weight[static_cast<size_t>(c + i) * W + tap];
#pragma unroll
  for (int tap = 1; tap < W; ++tap) {   // tokens t0 - W + tap
    const int t = t0 - W + tap;
    if (t >= 0) {
      const float4 v = load_four<IN_BF16>(input, seq + static_cast<size_t>(t) * channels);
      x[tap][0] = rounded_in(v.x); x[tap][1] = rounded_in(v.y);
      x[tap][2] = rounded_in(v.z); x[tap][3] = rounded_in(v.w);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) x[tap][i] = own_state[i * W + W + t];
    }
  }
#pragma unroll 4
  for (int t = t0; t < t1; ++t) {
    const size_t at = seq + static_cast<size_t>(t) * channels;
    const float4 v = load_four<IN_BF16>(input, at);
#pragma unroll
    for (int tap = 0; tap + 1 < W; ++tap)
#pragma unroll
      for (int i = 0; i < 4; ++i) x[tap][i] = x[tap + 1][i];
    x[W - 1][0] = rounded_in(v.x); x[W - 1][1] = rounded_in(v.y);
    x[W - 1][2] = rounded_in(v.z); x[W - 1][3] = rounded_in(v.w);
    float y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float sum = 0.0f;
#pragma unroll
      for (int tap = 0; tap + 1 < W; ++tap) sum += x[tap][i] * w[i][tap];
      sum = rnd(sum + x[W - 1][i] * w[i][W - 1], round);
      y[i] = OUT_BF16 ? silu(sum) : rnd(silu(sum), round);
    }
    store_four<OUT_BF16>(output, at, y);
  }
  if (t0 == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float kept[W];
#pragma unroll
      for (int tap = 0; tap < W; ++tap) {   // token tokens - W + tap, or an entry of the old window
        const int t = tokens - W + tap;
        kept[tap] = t >= 0 ? rounded_in(load_any(input, seq + static_cast<size_t>(t) * channels + i, IN_BF16))
                           : own_state[i * W + W + t];
      }
#pragma unroll
      for (int tap = 0; tap < W; ++tap) own_state[i * W + tap] = kept[tap];
    }
  }
}

// Per (token, head): RMSNorm * weight * SiLU(z) with the reference's rounding after every product;
// final_round = 0 leaves the last product unrounded before the store (OutputForward).
__device__ __forceinline__ float norm_gate(float x, float inverse, float weight, float gate, int round,
                                           int final_round) {
  const float normalized = rnd(x * inverse, round);
  const float affine = rnd(normalized * weight, round);
  return rnd(affine * silu(gate), round && final_round);
}

// One warp per row, eight rows per CTA, a lane owning four consecutive channels of every 128.  HBM
// bound; the earlier form (a CTA of 256 threads per row, half of them idle at width 128, two
// barriers) took 49 us where this takes 14 (48000 rows of 128).
template <int G, bool CORE_BF16, bool Z_BF16, bool OUT_BF16>   // G groups of 128 channels
__global__ void __launch_bounds__(256) gdn_output_rows_kernel(const void* __restrict__ core, const void* __restrict__ z,
                                                              const float* __restrict__ norm_weight, long long rows,
                                                              int dim, float epsilon, int round, int final_round,
                                                              void* __restrict__ output) {
  const long long row = static_cast<long long>(blockIdx.x) * 8 + threadIdx.x / 32;
  if (row >= rows) return;
  const int lane = threadIdx.x % 32;
  const size_t base = static_cast<size_t>(row) * dim;
  float4 x[G], gate[G];
  float sq = 0.0f;
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int c = i * 128 + lane * 4;
    x[i] = gate[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < dim) {
      x[i] = load_four<CORE_BF16>(core, base + c);
      gate[i] = load_four<Z_BF16>(z, base + c);
    }
    sq += x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  const float inverse = rsqrtf(sq / static_cast<float>(dim) + epsilon);
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int c = i * 128 + lane * 4;
    if (c >= dim) continue;
    const float4 w = *reinterpret_cast<const float4*>(norm_weight + c);
    const float y[4] = {norm_gate(x[i].x, inverse, w.x, gate[i].x, round, final_round),
                        norm_gate(x[i].y, inverse, w.y, gate[i].y, round, final_round),
                        norm_gate(x[i].z, inverse, w.z, gate[i].z, round, final_round),
                        norm_gate(x[i].w, inverse, w.w, gate[i].w, round, final_round)};
    store_four<OUT_BF16>(output, base + c, y);
  }
}

// The same for widths or addresses the four-channel accesses do not fit: grid = rows, 256 threads.
__global__ void __launch_bounds__(256) gdn_output_kernel(const void* core, const void* z,
                                                         const float* norm_weight, int core_is_bf16,
                                                         int z_is_bf16, int dim, float epsilon,
                                                         int round, int final_round, void* output,
                                                         int out_is_bf16) {
  const size_t row = blockIdx.x;
  const int c = threadIdx.x;
  const float x = c < dim ? load_any(core, row * dim + c, core_is_bf16) : 0.0f;
  __shared__ float red[8];
  float sq = x * x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if (c % 32 == 0) red[c / 32] = sq;
  __syncthreads();
  float total = 0.0f;
#pragma unroll
  for (int w = 0; w < 8; ++w) total += red[w];
  if (c >= dim) return;
  const float inverse = rsqrtf(total / static_cast<float>(dim) + epsilon);
  store_any(output, row * dim + c, out_is_bf16,
            norm_gate(x, inverse, norm_weight[c], load_any(z, row * dim + c, z_is_bf16), round, final_round));
}

bool aligned_to(const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; }

template <int W>
void launch_conv_segments(cudaStream_t stream, const void* input, const float* weight, int in_is_bf16, int batch,
                          int tokens, int channels, int round, float* state, void* output, int out_is_bf16) {
  const dim3 grid((channels / 4 + 127) / 128, (tokens + kConvSegment - 1) / kConvSegment, batch);
  auto kernel = in_is_bf16 ? (out_is_bf16 ? gdn_conv_segment_kernel<W, true, true> : gdn_conv_segment_kernel<W, true, false>)
                           : (out_is_bf16 ? gdn_conv_segment_kernel<W, false, true> : gdn_conv_segment_kernel<W, false, false>);
  kernel<<<grid, 128, 0, stream>>>(input, weight, tokens, channels, round, state, output);
}

}  // namespace

cudaError_t gdn_recurrent(cudaStream_t stream, const GdnArgs& a) {
  const dim3 grid((a.value_dim + kSlice - 1) / kSlice, a.value_heads, a.batch);
  gdn_recurrent_kernel<<<grid, kRecThreads, 0, stream>>>(a);
  return cudaGetLastError();
}

cudaError_t gdn_gates(cudaStream_t stream, const void* a_in, const void* b_in, const float* a_log,
                      const float* dt_bias, int in_is_bf16, long long tokens, int heads, int round,
                      float* g, float* beta) {
  const long long count = tokens * heads;
  gdn_gates_kernel<<<static_cast<unsigned>((count + 255) / 256), 256, 0, stream>>>(
      a_in, b_in, a_log, dt_bias, in_is_bf16, count, heads, round, g, beta);
  return cudaGetLastError();
}

cudaError_t gdn_conv(cudaStream_t stream, const void* input, const float* weight, int in_is_bf16,
                     int batch, int tokens, int channels, int width, int round, float* state,
                     void* output, int out_is_bf16) {
  // four-tap windows and shorter over several tokens: cut along the tokens (a single token has
  // nothing to cut, and grid.y / grid.z bound what one launch can hold; in place, a segment's history
  // would already be the segment before's output, so a thread then walks all tokens)
  const size_t elements = static_cast<size_t>(batch) * tokens * channels;
  const uintptr_t in0 = reinterpret_cast<uintptr_t>(input), out0 = reinterpret_cast<uintptr_t>(output);
  const bool apart = in0 + elements * (in_is_bf16 ? 2 : 4) <= out0 || out0 + elements * (out_is_bf16 ? 2 : 4) <= in0;
  if (apart && width >= 2 && width <= 4 && tokens > 1 && channels % 4 == 0 && batch <= 65535 &&
      (tokens + kConvSegment - 1) / kConvSegment <= 65535 && aligned_to(input, in_is_bf16 ? 8 : 16) &&
      aligned_to(output, out_is_bf16 ? 8 : 16)) {
    auto launch = width == 4 ? launch_conv_segments<4> : width == 3 ? launch_conv_segments<3> : launch_conv_segments<2>;
    launch(stream, input, weight, in_is_bf16, batch, tokens, channels, round, state, output, out_is_bf16);
    return cudaGetLastError();
  }
  const long long count = static_cast<long long>(batch) * channels;
  gdn_conv_kernel<<<static_cast<unsigned>((count + 127) / 128), 128, 0, stream>>>(
      input, weight, in_is_bf16, batch, tokens, channels, width, round, state, output, out_is_bf16);
  return cudaGetLastError();
}

cudaError_t gdn_output(cudaStream_t stream, const void* core, const void* z,
                       const float* norm_weight, int core_is_bf16, int z_is_bf16, long long rows,
                       int dim, float epsilon, int round, int final_round, void* output,
                       int out_is_bf16) {
  if (dim % 4 == 0 && aligned_to(core, core_is_bf16 ? 8 : 16) && aligned_to(z, z_is_bf16 ? 8 : 16) &&
      aligned_to(norm_weight, 16) && aligned_to(output, out_is_bf16 ? 8 : 16)) {
    using Kernel = void (*)(const void*, const void*, const float*, long long, int, float, int, int, void*);
#define OUTPUT_ROWS(G)                                                                                  \
    {gdn_output_rows_kernel<G, false, false, false>, gdn_output_rows_kernel<G, false, false, true>,     \
     gdn_output_rows_kernel<G, false, true, false>,  gdn_output_rows_kernel<G, false, true, true>,      \
     gdn_output_rows_kernel<G, true, false, false>,  gdn_output_rows_kernel<G, true, false, true>,      \
     gdn_output_rows_kernel<G, true, true, false>,   gdn_output_rows_kernel<G, true, true, true>}
    static const Kernel kernels[2][8] = {OUTPUT_ROWS(1), OUTPUT_ROWS(2)};
#undef OUTPUT_ROWS
    kernels[dim <= 128 ? 0 : 1][(core_is_bf16 ? 4 : 0) + (z_is_bf16 ? 2 : 0) + (out_is_bf16 ? 1 : 0)]
        <<<static_cast<unsigned>((rows + 7) / 8), 256, 0, stream>>>(core, z, norm_weight, rows, dim, epsilon, round,
                                                                    final_round, output);
    return cudaGetLastError();
  }
  gdn_output_kernel<<<static_cast<unsigned>(rows), 256, 0, stream>>>(
      core, z, norm_weight, core_is_bf16, z_is_bf16, dim, epsilon, round, final_round, output,
      out_is_bf16);
  return cudaGetLastError();
}

}  // namespace pluto
