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
#include "qk_rows.cuh"

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
// The arithmetic is that of prepare + split decode + merge, in their order, so that a result does not
// depend on the number of launches: the context is cut into decode_chunk_*'s chunks, a chunk into four
// token groups with an online softmax each, the groups meet in a chunk and the chunks in the row.  What
// the one launch saves is the launches and the round trips between them.
constexpr int kStepMaxChunks = 7;     // chunks of kCachedStepTokens tokens cut as one sequence is
constexpr int kStepSplit = 256;       // decode_chunk_*'s split_tokens for one sequence of this length
constexpr float kLog2e = 1.4426950408889634f;

// Four consecutive channels of a row of the call's input.
__device__ __forceinline__ void load_input(const void* p, size_t i, int is_bf16, float* v) {
#pragma unroll
  for (int u = 0; u < 4; ++u) v[u] = load_any(p, i + u, is_bf16);
}

// n = R(x * inv * (1 + w)) of one row of width D into `row` (shared memory), by one warp.
template <int D>
__device__ __forceinline__ void normalise_row(const void* in, size_t at, int is_bf16, const float* norm, float epsilon,
                                              int round, int lane, float* row) {
  float x[kRowOwn];
#pragma unroll
  for (int i = 0; i < kRowOwn; i += 4) {
    const int c = row_channel<4>(i, lane);
    if (c < D) load_input(in, at + c, is_bf16, x + i);
    else x[i] = x[i + 1] = x[i + 2] = x[i + 3] = 0.0f;
  }
  const float inverse = rsqrtf(row_square_sum<4>(x, lane) / static_cast<float>(D) + epsilon);
#pragma unroll
  for (int i = 0; i < kRowOwn; ++i) {
    const int c = row_channel<4>(i, lane);
    if (c < D) row[c] = rnd(x[i] * inverse * (1.0f + norm[c]), round);
  }
}
// Rotates that row in place, by the same warp.
template <int D>
__device__ __forceinline__ void rotate_row(float* row, const float* cosine, const float* sine, int rotary, int round,
                                           int lane) {
  const int half = rotary / 2;
  float result[D / 32];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < D / 32; ++i) {
    const int c = i * 32 + lane, f = c < half ? c : c - half;
    result[i] = row[c];
    if (c < rotary) result[i] = rotate(result[i], c < half ? -row[c + half] : row[c - half], cosine[f], sine[f], round);
  }
  __syncwarp();   // every partner has been read
#pragma unroll
  for (int i = 0; i < D / 32; ++i) row[i * 32 + lane] = result[i];
}
template <int D>
__device__ __forceinline__ void value_row(const void* in, size_t at, int is_bf16, int round, int lane, float* row) {
#pragma unroll
  for (int i = 0; i < D / 32; ++i) row[i * 32 + lane] = rnd(load_any(in, at + i * 32 + lane, is_bf16), round);
}

// The chunks' (maximum in log2 units, sum) in shared memory -> every chunk's weight; returns the row's sum.
__device__ __forceinline__ float chunk_weights(const float2* ml, int chunks, float (&weight)[kStepMaxChunks]) {
  float top = -INFINITY, total = 0.0f;
#pragma unroll
  for (int s = 0; s < kStepMaxChunks; ++s)
    if (s < chunks) top = fmaxf(top, ml[s].x);
#pragma unroll
  for (int s = 0; s < kStepMaxChunks; ++s) {
    weight[s] = s < chunks ? exp2f(ml[s].x - top) : 0.0f;
    if (s < chunks) total = __fadd_rn(total, __fmul_rn(ml[s].y, weight[s]));
  }
  return total;
}
// The reference's output stage (cached_attention_ops.cc:120-125): R(R(acc / l) * R(sigmoid(gate))).
__device__ __forceinline__ void store_gated(const CachedStepArgs& a, int head, int d, float value) {
  value = rnd(value, a.round);
  const float gate = load_any(a.q_gate, (static_cast<size_t>(head) * 2 + 1) * a.head_dim + d, a.in_is_bf16);
  store_any(a.out, static_cast<size_t>(head) * a.head_dim + d, a.out_is_bf16,
            rnd(value * rnd(sigmoid(gate), a.round), a.round));
}

// kCount (2, 4 or 8) consecutive cache elements of a row.
template <int kCount, bool KV_BF16>
__device__ __forceinline__ void load_cache(const void* base, size_t at, float (&v)[kCount]) {
  if (!KV_BF16) {
    const float* p = static_cast<const float*>(base) + at;
#pragma unroll
    for (int i = 0; i < kCount; i += 2) {
      const float2 f = *reinterpret_cast<const float2*>(p + i);
      v[i] = f.x; v[i + 1] = f.y;
    }
    return;
  }
  const __nv_bfloat16* p = static_cast<const __nv_bfloat16*>(base) + at;
  uint32_t w[kCount / 2];
  if (kCount == 8) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    w[0] = raw.x; w[1 % (kCount / 2)] = raw.y; w[2 % (kCount / 2)] = raw.z; w[3 % (kCount / 2)] = raw.w;
  } else if (kCount == 4) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    w[0] = raw.x; w[1 % (kCount / 2)] = raw.y;
  } else {
    w[0] = *reinterpret_cast<const uint32_t*>(p);
  }
#pragma unroll
  for (int i = 0; i < kCount; i += 2) { v[i] = bf16_lo(w[i / 2]); v[i + 1] = bf16_hi(w[i / 2]); }
}

// fp32 products, one CTA per query head: every CTA prepares its query and its group's new key and value
// itself (the first head of a group writes the two into the cache).  K is read by eight tokens per warp,
// four lanes each: a lane sums the channels 8 j .. 8 j + 7 of every 32, which are the chains that the
// decode kernel's lanes form, and the butterfly over a token's chains runs half in shuffles and half in
// the lane.  With at most kCachedStepTokens rows, K and V come from L2 for the heads of a group.
constexpr int kStepWarps = 16;
template <int D, bool KV_BF16>
__global__ void __launch_bounds__(kStepWarps * 32) cached_step_kernel(CachedStepArgs a) {
  constexpr int kPer = D / 32, kUnits = 4 * kStepMaxChunks;
  __shared__ float cosine[128], sine[128];
  __shared__ __align__(16) float query[D], new_key[D], new_value[D];
  __shared__ float score[kCachedStepTokens];
  __shared__ float2 weigh[kCachedStepTokens];        // (p, correction of what came before)
  __shared__ float unit_acc[kUnits][D];              // unit: a token group of a chunk
  __shared__ float2 unit_ml[kUnits], chunk_ml[kStepMaxChunks];
  const int head = blockIdx.x, group = a.q_heads / a.kv_heads, kv_head = head / group;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int length = a.position + 1, chunks = decode_chunk_count(length, kStepSplit);
  const size_t head_row = static_cast<size_t>(kv_head) * D;
  const int last_row = max(a.position - 1, 0);

  pdl_wait();   // every input, the weights too: the kernel before this one may have written them
  pdl_launch_dependents();   // the next launch sets itself up meanwhile and waits for this grid in turn
  // K of this lane's first token is requested before anything waits: at short contexts the kernel is a
  // chain of memory round trips
  const int own = warp * 8 + lane / 4, part = lane % 4 * 8;
  constexpr int kRaw = KV_BF16 ? 1 : 2;   // 16-byte pieces of eight elements
  auto load_key = [&](int t, uint4 (&raw)[kPer][kRaw]) {
    const size_t at = static_cast<size_t>(min(t, last_row)) * a.token_stride + head_row + part;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
#pragma unroll
      for (int u = 0; u < kRaw; ++u)
        raw[i][u] = KV_BF16 ? *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.k_cache) + at + i * 32)
                            : *reinterpret_cast<const uint4*>(static_cast<const float*>(a.k_cache) + at + i * 32 + u * 4);
  };
  uint4 keys[kPer][kRaw];
  load_key(own, keys);
  if (static_cast<int>(threadIdx.x) < a.rotary / 2)
    rotary_angle(a.position, threadIdx.x, a.log_theta, a.rotary, a.round, cosine[threadIdx.x], sine[threadIdx.x]);
  if (warp == 0)
    normalise_row<D>(a.q_gate, static_cast<size_t>(head) * 2 * D, a.in_is_bf16, a.q_norm, a.epsilon, a.round, lane, query);
  else if (warp == 1)
    normalise_row<D>(a.k, head_row, a.in_is_bf16, a.k_norm, a.epsilon, a.round, lane, new_key);
  else if (warp == 2)
    value_row<D>(a.v, head_row, a.in_is_bf16, a.round, lane, new_value);
  __syncthreads();   // (the rotary tables)
  if (warp < 2) rotate_row<D>(warp == 0 ? query : new_key, cosine, sine, a.rotary, a.round, lane);
  if (warp == 1 || warp == 2) {   // attended to as the cache holds them
    float* row = warp == 1 ? new_key : new_value;
    void* cache = warp == 1 ? a.k_cache : a.v_cache;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int c = i * 32 + lane;
      row[c] = rnd(row[c], KV_BF16);
      if (head % group == 0) store_any(cache, static_cast<size_t>(a.position) * a.token_stride + head_row + c, KV_BF16, row[c]);
    }
  }
  __syncthreads();

  for (int t0 = 0; t0 < length; t0 += 8 * kStepWarps) {   // (uniform: the shuffles want whole warps)
    const int t = t0 + own;
    if (t0 > 0) load_key(t, keys);
    float dot[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) dot[r] = 0.0f;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      float q[8], k[8];
      *reinterpret_cast<float4*>(q) = *reinterpret_cast<const float4*>(query + i * 32 + part);
      *reinterpret_cast<float4*>(q + 4) = *reinterpret_cast<const float4*>(query + i * 32 + part + 4);
      const uint32_t* raw = reinterpret_cast<const uint32_t*>(keys[i]);
#pragma unroll
      for (int r = 0; r < 8; ++r)
        k[r] = !KV_BF16 ? __uint_as_float(raw[r % (4 * kRaw)]) : r % 2 ? bf16_hi(raw[r / 2]) : bf16_lo(raw[r / 2]);
      if (t >= a.position) {   // the new token (and whatever past the end: not stored)
#pragma unroll
        for (int r = 0; r < 8; ++r) k[r] = new_key[i * 32 + part + r];
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) dot[r] = fmaf(k[r], q[r], dot[r]);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      dot[r] += __shfl_xor_sync(0xffffffffu, dot[r], 2);
      dot[r] += __shfl_xor_sync(0xffffffffu, dot[r], 1);
    }
    const float sum = ((dot[0] + dot[4]) + (dot[2] + dot[6])) + ((dot[1] + dot[5]) + (dot[3] + dot[7]));
    if (t < length && lane % 4 == 0) score[t] = __fmul_rn(sum, a.scale);
  }
  __syncthreads();

  for (int unit = warp; unit < 4 * chunks; unit += kStepWarps) {
    const int chunk = unit / 4, begin = decode_chunk_begin(chunk, kStepSplit) + unit % 4;
    const int end = min(length, decode_chunk_begin(chunk, kStepSplit) + decode_chunk_tokens(chunk, kStepSplit));
    const int count = begin < end ? (end - begin + 3) / 4 : 0;   // tokens begin, begin + 4, ... (64 at most)
    // the running maxima of the online softmax, all at once
    float top = -INFINITY;
#pragma unroll
    for (int k0 = 0; k0 < 64; k0 += 32) {
      const int t = begin + (k0 + lane) * 4;
      const float s = k0 + lane < count ? score[t] : -INFINITY;
      float m = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float below = __shfl_up_sync(0xffffffffu, m, o);
        if (lane >= o) m = fmaxf(m, below);
      }
      m = fmaxf(m, top);
      float before = __shfl_up_sync(0xffffffffu, m, 1);
      if (lane == 0) before = top;
      if (k0 + lane < count) weigh[t] = make_float2(expf(s - m), expf(before - m));
      top = __shfl_sync(0xffffffffu, m, 31);
    }
    __syncwarp();
    float acc[kPer], l = 0.0f;
#pragma unroll
    for (int i = 0; i < kPer; ++i) acc[i] = 0.0f;
#pragma unroll 8
    for (int k = 0; k < count; ++k) {
      const int t = begin + 4 * k;
      float v[kPer];
      // (the new token is the last one; its row of the cache may be another CTA's to write at this moment)
      load_cache<kPer, KV_BF16>(a.v_cache, static_cast<size_t>(min(t, last_row)) * a.token_stride + head_row + lane * kPer, v);
      if (t >= a.position) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) v[i] = new_value[lane * kPer + i];
      }
      const float2 w = weigh[t];
      l = fmaf(l, w.y, w.x);
#pragma unroll
      for (int i = 0; i < kPer; ++i) acc[i] = fmaf(w.x, v[i], __fmul_rn(acc[i], w.y));
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i) unit_acc[unit][lane * kPer + i] = acc[i];
    if (lane == 0) unit_ml[unit] = make_float2(top, l);
  }
  __syncthreads();
  auto chunk_top = [&](int s) {
    return fmaxf(fmaxf(unit_ml[4 * s].x, unit_ml[4 * s + 1].x), fmaxf(unit_ml[4 * s + 2].x, unit_ml[4 * s + 3].x));
  };
  if (static_cast<int>(threadIdx.x) < chunks) {
    const int s = threadIdx.x;
    const float top = chunk_top(s);
    float l = 0.0f;
#pragma unroll
    for (int w = 0; w < 4; ++w) l = fmaf(unit_ml[4 * s + w].y, expf(unit_ml[4 * s + w].x - top), l);
    chunk_ml[s] = make_float2(__fmul_rn(top, kLog2e), l);
  }
  __syncthreads();
  if (threadIdx.x >= D) return;
  float weight[kStepMaxChunks];
  const float total = chunk_weights(chunk_ml, chunks, weight);
  float acc = 0.0f;
#pragma unroll
  for (int s = 0; s < kStepMaxChunks; ++s) {
    if (s >= chunks) break;
    const float top = chunk_top(s);
    float sum = 0.0f;
#pragma unroll
    for (int w = 0; w < 4; ++w) sum = fmaf(unit_acc[4 * s + w][threadIdx.x], expf(unit_ml[4 * s + w].x - top), sum);
    acc = fmaf(sum, weight[s], acc);
  }
  store_gated(a, head, threadIdx.x, acc / total);
}

// Products on the tensor cores (mma.sync), where the decode kernel takes them: bf16 cache and rounded
// queries of width 64 or 128.  One CTA of eight warps per key/value head, whose query heads are the rows
// of the tile; a warp owns 16 tokens of every 64, so four warps make a chunk and the CTA walks two at a
// time.  P enters P V as a bf16 high part and a remainder.  A warp's K and V rows come by asynchronous
// copies into shared memory of its own; the first are requested before anything waits.
constexpr int kTcStepWarps = 8;
template <int D>
struct TcStepLayout {
  static constexpr int kPitch = D + 8;                              // bf16 elements: rows 16 bytes further round the banks
  static constexpr int kTileBytes = 16 * kPitch * 2;                // K or V of a warp
  static constexpr int kOwnBytes = 2 * kTileBytes;                  // both; later fp32 [16][D]
  static constexpr int kVectors = kTcStepWarps * kOwnBytes;         // fp32 [18][D]: queries, new key, new value
  static constexpr int kChunkAcc = kVectors + 18 * D * 4;           // fp32 [chunk][16][D]
  static constexpr int kMl = kChunkAcc + kStepMaxChunks * 16 * D * 4;   // float2 [16][chunks], then [warp][16]
  static constexpr int kTotal = kMl + (kStepMaxChunks + kTcStepWarps) * 16 * 8;
  static_assert(16 * D * 4 <= kOwnBytes, "a warp's accumulators fit its tiles");
};

__device__ __forceinline__ void step_ldmatrix(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void step_ldmatrix_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void step_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int D>
__global__ void __launch_bounds__(kTcStepWarps * 32) cached_step_tc_kernel(CachedStepArgs a) {
  using Layout = TcStepLayout<D>;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float cosine[64], sine[64];
  float* vectors = reinterpret_cast<float*>(smem + Layout::kVectors);
  float* chunk_acc = reinterpret_cast<float*>(smem + Layout::kChunkAcc);
  float2* chunk_ml = reinterpret_cast<float2*>(smem + Layout::kMl);
  float2* warp_ml = chunk_ml + kStepMaxChunks * 16;
  const int kv_head = blockIdx.x, group = a.q_heads / a.kv_heads;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, quarter = warp % 4;
  const int length = a.position + 1, chunks = decode_chunk_count(length, kStepSplit);
  const size_t head_row = static_cast<size_t>(kv_head) * D;
  uint8_t* own = smem + warp * Layout::kOwnBytes;
  float* own_acc = reinterpret_cast<float*>(own);
  const uint32_t k_tile = smem_u32(own), v_tile = k_tile + Layout::kTileBytes;

  pdl_wait();
  pdl_launch_dependents();
  // The cached rows of the 16 tokens from t0 on, the new token's and zeros past the end.
  auto request = [&](int t0) {
    constexpr int kPieces = D / 8;   // 16-byte pieces of a row
    for (int e = lane; e < 2 * 16 * kPieces; e += 32) {
      const int value = e / (16 * kPieces), r = e / kPieces % 16, c = e % kPieces * 8, t = t0 + r;
      const uint32_t to = (value ? v_tile : k_tile) + (r * Layout::kPitch + c) * 2;
      if (t < a.position) {
        const __nv_bfloat16* from = static_cast<const __nv_bfloat16*>(value ? a.v_cache : a.k_cache) +
                                    static_cast<size_t>(t) * a.token_stride + head_row + c;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
      } else if (t > a.position) {
        sts_b32x4(to, 0u, 0u, 0u, 0u);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int first = decode_chunk_begin(warp / 4, kStepSplit) + quarter * 16;
  if (first < length) request(first);
  if (static_cast<int>(threadIdx.x) < a.rotary / 2)
    rotary_angle(a.position, threadIdx.x, a.log_theta, a.rotary, a.round, cosine[threadIdx.x], sine[threadIdx.x]);
  for (int r = warp; r < group + 2; r += kTcStepWarps) {
    float* row = vectors + r * D;
    if (r < group)
      normalise_row<D>(a.q_gate, (static_cast<size_t>(kv_head) * group + r) * 2 * D, a.in_is_bf16, a.q_norm, a.epsilon,
                       a.round, lane, row);
    else if (r == group)
      normalise_row<D>(a.k, head_row, a.in_is_bf16, a.k_norm, a.epsilon, a.round, lane, row);
    else
      value_row<D>(a.v, head_row, a.in_is_bf16, a.round, lane, row);
  }
  __syncthreads();   // (the rotary tables)
  for (int r = warp; r < group + 2; r += kTcStepWarps) {
    float* row = vectors + r * D;
    if (r <= group) rotate_row<D>(row, cosine, sine, a.rotary, a.round, lane);
    if (r >= group) {
      void* cache = r == group ? a.k_cache : a.v_cache;
#pragma unroll
      for (int i = 0; i < D / 32; ++i)
        store_any(cache, static_cast<size_t>(a.position) * a.token_stride + head_row + i * 32 + lane, 1, row[i * 32 + lane]);
    }
  }
  __syncthreads();
  // A fragments of Q: rows = query heads of this KV head (rows >= group are zero).
  uint32_t qf[D / 16][4];
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // rows lane / 4, + 8; columns 0-7, 8-15 of the step
      const int r = lane / 4 + (i & 1) * 8, c = ks * 16 + (i >> 1) * 8 + (lane % 4) * 2;
      qf[ks][i] = r < group ? pack_bf16(vectors[r * D + c], vectors[r * D + c + 1]) : 0u;
    }
  const float scale_log2 = a.scale * kLog2e;
  for (int chunk0 = 0; chunk0 < chunks; chunk0 += kTcStepWarps / 4) {
    const int chunk = chunk0 + warp / 4, begin = decode_chunk_begin(chunk, kStepSplit);
    const int end = min(length, begin + decode_chunk_tokens(chunk, kStepSplit));
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f}, o[D / 8][4];
#pragma unroll
    for (int nb = 0; nb < D / 8; ++nb)
#pragma unroll
      for (int i = 0; i < 4; ++i) o[nb][i] = 0.0f;
    if (chunk0 > 0) __syncthreads();   // the chunks before have been read
    for (int t0 = begin + quarter * 16; t0 < end; t0 += 64) {
      if (t0 != first) request(t0);
      const int fresh = a.position - t0;   // the new token's row of the tile, where it has one
      if (fresh >= 0 && fresh < 16 && lane < D / 8) {
#pragma unroll
        for (int value = 0; value < 2; ++value) {
          const float* row = vectors + (group + value) * D + lane * 8;
          sts_b32x4((value ? v_tile : k_tile) + (fresh * Layout::kPitch + lane * 8) * 2, pack_bf16(row[0], row[1]),
                    pack_bf16(row[2], row[3]), pack_bf16(row[4], row[5]), pack_bf16(row[6], row[7]));
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      float s[2][4] = {};
#pragma unroll
      for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int kp = 0; kp < D / 32; ++kp) {
          uint32_t kf[4];
          step_ldmatrix(kf, k_tile + ((nb * 8 + lane % 8) * Layout::kPitch + kp * 32 + lane / 8 * 8) * 2);
          step_mma(s[nb], qf[2 * kp], kf[0], kf[1]);
          step_mma(s[nb], qf[2 * kp + 1], kf[2], kf[3]);
        }
      const int token0 = t0 + (lane % 4) * 2;
      float tile_max[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          s[nb][i] = token0 + nb * 8 + (i & 1) < end ? __fmul_rn(s[nb][i], scale_log2) : -INFINITY;
          tile_max[i >> 1] = fmaxf(tile_max[i >> 1], s[nb][i]);
        }
      uint32_t pf[4], pl[4];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        tile_max[r] = fmaxf(tile_max[r], __shfl_xor_sync(0xffffffffu, tile_max[r], 1));
        tile_max[r] = fmaxf(tile_max[r], __shfl_xor_sync(0xffffffffu, tile_max[r], 2));
        const float m_new = fmaxf(m_run[r], tile_max[r]);
        const float m_safe = m_new == -INFINITY ? 0.0f : m_new;
        const float correction = fast_exp2(m_run[r] - m_safe);
        const float p00 = fast_exp2(s[0][2 * r] - m_safe), p01 = fast_exp2(s[0][2 * r + 1] - m_safe);
        const float p10 = fast_exp2(s[1][2 * r] - m_safe), p11 = fast_exp2(s[1][2 * r + 1] - m_safe);
        float sum = p00 + p01 + p10 + p11;
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        l_run[r] = fmaf(l_run[r], correction, sum);
        m_run[r] = m_new;
        pf[r] = pack_bf16(p00, p01);      // tokens 0-7
        pf[2 + r] = pack_bf16(p10, p11);  // tokens 8-15
        pl[r] = pack_bf16(p00 - bf16_lo(pf[r]), p01 - bf16_hi(pf[r]));
        pl[2 + r] = pack_bf16(p10 - bf16_lo(pf[2 + r]), p11 - bf16_hi(pf[2 + r]));
#pragma unroll
        for (int nb = 0; nb < D / 8; ++nb) {
          o[nb][2 * r] *= correction;
          o[nb][2 * r + 1] *= correction;
        }
      }
#pragma unroll
      for (int np = 0; np < D / 16; ++np) {
        uint32_t vf[4];
        step_ldmatrix_trans(vf, v_tile + ((lane / 8 % 2 * 8 + lane % 8) * Layout::kPitch + np * 16 + lane / 16 * 8) * 2);
        step_mma(o[2 * np], pf, vf[0], vf[1]);
        step_mma(o[2 * np], pl, vf[0], vf[1]);
        step_mma(o[2 * np + 1], pf, vf[2], vf[3]);
        step_mma(o[2 * np + 1], pl, vf[2], vf[3]);
      }
      __syncwarp();   // the tiles have been read
    }
    if (chunk < chunks) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = lane / 4 + i * 8;
#pragma unroll
        for (int nb = 0; nb < D / 8; ++nb)
          *reinterpret_cast<float2*>(own_acc + r * D + nb * 8 + (lane % 4) * 2) = make_float2(o[nb][2 * i], o[nb][2 * i + 1]);
        if (lane % 4 == 0) warp_ml[warp * 16 + r] = make_float2(m_run[i], l_run[i]);
      }
    }
    __syncthreads();
    // the four token groups of a chunk, in order
    for (int e = threadIdx.x; e < kTcStepWarps / 4 * group * D; e += kTcStepWarps * 32) {
      const int which = e / (group * D), r = e / D % group, d = e % D, s = chunk0 + which;
      if (s >= chunks) break;
      const float2* ml = warp_ml + which * 64 + r;
      const float top = fmaxf(fmaxf(ml[0].x, ml[16].x), fmaxf(ml[32].x, ml[48].x));
      float acc = 0.0f, l = 0.0f;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float f = fast_exp2(ml[16 * w].x - top);
        const float* from = reinterpret_cast<const float*>(smem + (which * 4 + w) * Layout::kOwnBytes);
        acc = fmaf(from[r * D + d], f, acc);
        l = fmaf(ml[16 * w].y, f, l);
      }
      chunk_acc[(s * 16 + r) * D + d] = acc;
      if (d == 0) chunk_ml[r * kStepMaxChunks + s] = make_float2(top, l);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < group * D; e += kTcStepWarps * 32) {
    const int r = e / D, d = e % D;
    float weight[kStepMaxChunks], acc = 0.0f;
    const float total = chunk_weights(chunk_ml + r * kStepMaxChunks, chunks, weight);
#pragma unroll
    for (int s = 0; s < kStepMaxChunks; ++s)
      if (s < chunks) acc = fmaf(chunk_acc[(s * 16 + r) * D + d], weight[s], acc);
    store_gated(a, kv_head * group + r, d, acc / total);
  }
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
    qkv[part][i] = rnd(silu(sum), a.round);
    if (part == 0) {   // the threads that finish the row
      z = load_any(a.z, static_cast<size_t>(h) * kDim + i, a.z_is_bf16);
    }
  } else if (tid == 3 * kDim) {
    const float alpha = load_any(a.a_in, h, a.ab_is_bf16) + a.dt_bias[h];
    const float softplus = fmaxf(alpha, 0.0f) + logf(1.0f + expf(-fabsf(alpha)));
    gates[0] = expf(-expf(a.a_log[h]) * softplus);
    gates[1] = rnd(sigmoid(load_any(a.b_in, h, a.ab_is_bf16)), a.round);
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
    store_any(a.out, static_cast<size_t>(h) * kDim + i, a.out_is_bf16, rnd(affine * silu(z), a.round));
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

namespace {
template <typename Kernel>
cudaError_t launch_step(Kernel kernel, int ctas, int threads, size_t smem, cudaStream_t stream, const CachedStepArgs& a) {
  if (smem > 0) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
  }
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(ctas);
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, a);
}
}  // namespace

cudaError_t cached_step(cudaStream_t stream, const CachedStepArgs& a) {
  // the decode kernel's rule for its tensor-core form, less width 256
  const bool tc = a.kv_is_bf16 && a.round && a.head_dim <= 128 && a.q_heads / a.kv_heads <= 16 && a.capacity % 16 == 0;
  if (tc && a.head_dim == 128)
    return launch_step(cached_step_tc_kernel<128>, a.kv_heads, kTcStepWarps * 32, TcStepLayout<128>::kTotal, stream, a);
  if (tc) return launch_step(cached_step_tc_kernel<64>, a.kv_heads, kTcStepWarps * 32, TcStepLayout<64>::kTotal, stream, a);
  using Kernel = void (*)(CachedStepArgs);
  static const Kernel kernels[3][2] = {{cached_step_kernel<64, false>, cached_step_kernel<64, true>},
                                       {cached_step_kernel<128, false>, cached_step_kernel<128, true>},
                                       {cached_step_kernel<256, false>, cached_step_kernel<256, true>}};
  return launch_step(kernels[a.head_dim / 128][a.kv_is_bf16 ? 1 : 0], a.q_heads, kStepWarps * 32, 0, stream, a);
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
