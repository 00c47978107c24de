// Causal multi-head attention over a packed [rows, 3E] activation -- the exact-fp32 path.
//
// Mirrors the reference layer AttentionLayer (src/llm/layers/attention.cc:98-170 forward,
// :176-230 probabilities, :235-314 query-owned backward, :319-396 key/value-owned backward) for
// every shape it accepts: any head width up to 256, fp32 storage (the reference's "FP16" compute
// policy keeps fp32 activations) or bf16 storage, ragged sequence and head tiles.  All arithmetic
// is fp32 FFMA with expf, so the fp32 policy meets a 1e-4 tolerance against the scalar CPU
// layer; the bf16 tensor-core path in attn_fwd_sm100.cu takes over for head widths 64/128.
//
// Like the reference the backward is two single-writer passes with fixed-order reductions and no
// floating-point atomics, so repeated runs are bitwise identical.
#include <algorithm>

#include "common.cuh"
#include "engine.h"

namespace pluto {
namespace {

constexpr int kThreads = 256;  // 16 x 16 thread grid
constexpr float kSentinel = -3.402823466e+38f;

template <typename T>
__device__ __forceinline__ float load_as_float(const T* p);
template <>
__device__ __forceinline__ float load_as_float<float>(const float* p) { return *p; }
template <>
__device__ __forceinline__ float load_as_float<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}
template <typename T>
__device__ __forceinline__ void store_from_float(T* p, float v);
template <>
__device__ __forceinline__ void store_from_float<float>(float* p, float v) { *p = v; }
template <>
__device__ __forceinline__ void store_from_float<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16_rn(v);
}

// Tiles in shared memory have rows of kPitch floats: a multiple of four, so that every access below is
// 16 bytes wide, and four more than the width, so that the 16 rows or the 16 column quads that half a
// warp touches fall into all bank groups.
//
// What bounds these kernels is the shared-memory pipe: with scalar accesses a 4 x 4 block of products
// cost eight of them for 16 multiply-adds (16 sequences of 256 tokens, 6 heads of 64:
// 343 us forward and backward); with
// 16-byte accesses and four products per operand it is 12 wavefronts for 64, below what the 64
// multiply-adds take to issue (183 us).
template <int W>
constexpr int kPitch = W + 4;

// Four consecutive head columns of a row, from an address known to be aligned to the four.
__device__ __forceinline__ float4 load_four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_four(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  return make_float4(bf16_lo(raw.x), bf16_hi(raw.x), bf16_lo(raw.y), bf16_hi(raw.y));
}
__device__ __forceinline__ void store_four(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store_four(__nv_bfloat16* p, const float (&v)[4]) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
}
// Whether rows of D elements that start at `base` plus multiples of the strides can be accessed by fours.
template <typename T>
__device__ __forceinline__ bool by_fours(const T* base, size_t token, size_t head, int D) {
  return D % 4 == 0 && token % 4 == 0 && head % 4 == 0 && reinterpret_cast<uintptr_t>(base) % (4 * sizeof(T)) == 0;
}
// v into the columns [d, d + 4) of a row of D.
template <typename T>
__device__ __forceinline__ void store_columns(T* row, int d, int D, bool fours, const float (&v)[4]) {
  if (fours) {
    if (d < D) store_four(row + d, v);
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (d + i < D) store_from_float(row + d + i, v[i]);
}

// Copies rows [row0, row0+ROWS) x head columns [0, D) of one section into an fp32 shared tile; rows
// past the sequence end and columns past D become zero.
template <typename T, int ROWS, int DP>
__device__ __forceinline__ void load_tile(float (*tile)[kPitch<DP>], const T* base, size_t row_stride,
                                          int row0, int seq, int D, bool fours) {
  constexpr int kQuads = DP / 4;
#pragma unroll 4
  for (int idx = threadIdx.x; idx < ROWS * kQuads; idx += kThreads) {
    const int r = idx / kQuads, d = idx % kQuads * 4;
    const int row = row0 + r;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (row < seq && d < D) {
      const T* from = base + static_cast<size_t>(row) * row_stride + d;
      if (fours) {
        v = load_four(from);
      } else {
        v.x = load_as_float(from);
        if (d + 1 < D) v.y = load_as_float(from + 1);
        if (d + 2 < D) v.z = load_as_float(from + 2);
        if (d + 3 < D) v.w = load_as_float(from + 3);
      }
    }
    *reinterpret_cast<float4*>(&tile[r][d]) = v;
  }
}

// c[i][j] = sum_d a[ty+16i][d] * b[tx+16j][d].  Columns are taken by fours (the tiles are zero past D);
// a pair of columns advances in one two-lane multiply-add, and the two lanes meet at the end.
template <int MI, int NJ, int P>
__device__ __forceinline__ void mm_nt(float (&c)[MI][NJ], const float (*a)[P], const float (*b)[P], int D, int ty,
                                      int tx) {
  uint64_t sum[MI][NJ];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) sum[i][j] = 0;
#pragma unroll 2
  for (int d = 0; d < D; d += 4) {
    ulonglong2 av[MI], bv[NJ];
#pragma unroll
    for (int i = 0; i < MI; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(&a[ty + 16 * i][d]);
#pragma unroll
    for (int j = 0; j < NJ; ++j) bv[j] = *reinterpret_cast<const ulonglong2*>(&b[tx + 16 * j][d]);
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) sum[i][j] = f2_fma(av[i].y, bv[j].y, f2_fma(av[i].x, bv[j].x, sum[i][j]));
  }
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      float even, odd;
      f2_unpack(sum[i][j], even, odd);
      c[i][j] = even + odd;
    }
}

// A thread's columns of an output row: four consecutive ones of every 64.
__device__ __forceinline__ int own_column(int tx, int c) { return tx * 4 + (c & 3) + (c >> 2) * 64; }

// acc[i][c] += sum_k p[ty+16i][k] * b[k][own_column(c)], k < BN (p is zero where there is no key)
template <int MI, int DC, int BN, int P>
__device__ __forceinline__ void mm_nn(float (&acc)[MI][DC], const float (*p)[kPitch<BN>], const float (*b)[P], int ty,
                                      int tx) {
#pragma unroll 2
  for (int k = 0; k < BN; k += 4) {
    float pv[MI][4];
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(&p[ty + 16 * i][k]);
      pv[i][0] = v.x; pv[i][1] = v.y; pv[i][2] = v.z; pv[i][3] = v.w;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int c = 0; c < DC; c += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&b[k + u][own_column(tx, c)]);
#pragma unroll
        for (int i = 0; i < MI; ++i) {
          acc[i][c] = fmaf(pv[i][u], v.x, acc[i][c]);
          acc[i][c + 1] = fmaf(pv[i][u], v.y, acc[i][c + 1]);
          acc[i][c + 2] = fmaf(pv[i][u], v.z, acc[i][c + 2]);
          acc[i][c + 3] = fmaf(pv[i][u], v.w, acc[i][c + 3]);
        }
      }
  }
}

// acc[i][c] += sum_q p[q][MI ty + i] * b[q][own_column(c)], q < BN (transposed left operand)
template <int MI, int DC, int BN, int P>
__device__ __forceinline__ void mm_tn(float (&acc)[MI][DC], const float (*p)[kPitch<BN>], const float (*b)[P], int ty,
                                      int tx) {
  static_assert(MI == 4 || MI == 2, "rows a thread owns");
#pragma unroll 4
  for (int q = 0; q < BN; ++q) {
    float pv[MI];
    if constexpr (MI == 4) {
      const float4 v = *reinterpret_cast<const float4*>(&p[q][4 * ty]);
      pv[0] = v.x; pv[1] = v.y; pv[2] = v.z; pv[3] = v.w;
    } else {
      const float2 v = *reinterpret_cast<const float2*>(&p[q][2 * ty]);
      pv[0] = v.x; pv[1] = v.y;
    }
#pragma unroll
    for (int c = 0; c < DC; c += 4) {
      const float4 v = *reinterpret_cast<const float4*>(&b[q][own_column(tx, c)]);
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        acc[i][c] = fmaf(pv[i], v.x, acc[i][c]);
        acc[i][c + 1] = fmaf(pv[i], v.y, acc[i][c + 1]);
        acc[i][c + 2] = fmaf(pv[i], v.z, acc[i][c + 2]);
        acc[i][c + 3] = fmaf(pv[i], v.w, acc[i][c + 3]);
      }
    }
  }
}

__device__ __forceinline__ float group16_max(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float group16_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct Dims {
  int seq, heads, head_dim;
  int batch, batch0;   // sequences of this launch, and the first of them
  float scale;
};

// Block id -> (tile, head, sequence), tile slowest: CTAs that share an SM then walk different numbers
// of tiles (with the tile fastest, 148 SMs and 4 tiles put the longest ones together).  The kernels
// number the tiles so that the longest come first.
struct Unit { int tile, head, batch; };
__device__ __forceinline__ Unit block_unit(int heads, const Dims& dims) {
  const unsigned per_tile = static_cast<unsigned>(heads) * dims.batch, rest = blockIdx.x % per_tile;
  return {static_cast<int>(blockIdx.x / per_tile), static_cast<int>(rest % heads),
          static_cast<int>(rest / heads) + dims.batch0};
}

// Addressing of separate Q/K/V tensors for the forward kernel: element strides between tokens
// and between heads, and how many query heads share one key/value head.
struct Views {
  size_t q_token, q_head, kv_token, kv_head, out_token, out_head, gate_token, gate_head;
  int group;
};

// ------------------------------------------------------------------------------------------
// forward: a CTA per (query tile, head, sequence), see block_unit
// ------------------------------------------------------------------------------------------
template <typename T, int DP, int BM>
__global__ void __launch_bounds__(kThreads, DP == 64 ? 3 : 1)
attn_fwd_generic(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                 T* __restrict__ out, float* __restrict__ maxima,
                 float* __restrict__ normalizers, const T* __restrict__ gate,
                 float* __restrict__ core, int round_gate, Dims dims, Views views) {
  constexpr int BN = BM, MI = BM / 16, NJ = BN / 16, DC = DP / 16;
  extern __shared__ __align__(16) float smem[];
  float(*Qs)[kPitch<DP>] = reinterpret_cast<float(*)[kPitch<DP>]>(smem);
  float(*Ks)[kPitch<DP>] = Qs + BM;
  float(*Vs)[kPitch<DP>] = Ks + BN;
  float(*Ps)[kPitch<BN>] = reinterpret_cast<float(*)[kPitch<BN>]>(Vs + BN);

  const int S = dims.seq, H = dims.heads, D = dims.head_dim;
  const Unit unit = block_unit(H, dims);
  const int qt = (S + BM - 1) / BM - 1 - unit.tile, h = unit.head, b = unit.batch;
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  const T* q_base = q + static_cast<size_t>(b) * S * views.q_token + h * views.q_head;
  const T* k_base = k + static_cast<size_t>(b) * S * views.kv_token + (h / views.group) * views.kv_head;
  const T* v_base = v + static_cast<size_t>(b) * S * views.kv_token + (h / views.group) * views.kv_head;
  const bool q_fours = by_fours(q, views.q_token, views.q_head, D);
  const bool kv_fours = by_fours(k, views.kv_token, views.kv_head, D) && by_fours(v, views.kv_token, views.kv_head, D);
  const bool out_fours = by_fours(out, views.out_token, views.out_head, D) &&
                         (core == nullptr || by_fours(core, views.out_token, views.out_head, D));

  load_tile<T, BM, DP>(Qs, q_base, views.q_token, qt * BM, S, D, q_fours);
  float m[MI], l[MI], acc[MI][DC];
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    m[i] = kSentinel;
    l[i] = 0.0f;
#pragma unroll
    for (int c = 0; c < DC; ++c) acc[i][c] = 0.0f;
  }
  for (int kt = 0; kt <= qt; ++kt) {
    __syncthreads();  // previous tile fully consumed (and Q visible on the first pass)
    load_tile<T, BN, DP>(Ks, k_base, views.kv_token, kt * BN, S, D, kv_fours);
    load_tile<T, BN, DP>(Vs, v_base, views.kv_token, kt * BN, S, D, kv_fours);
    __syncthreads();
    float s[MI][NJ];
    mm_nt<MI, NJ, kPitch<DP>>(s, Qs, Ks, D, ty, tx);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int query = qt * BM + ty + 16 * i;
      float tile_max = kSentinel;
      bool valid[NJ];
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int key = kt * BN + tx + 16 * j;
        valid[j] = key <= query && key < S;
        s[i][j] = valid[j] ? s[i][j] * dims.scale : kSentinel;
        tile_max = fmaxf(tile_max, s[i][j]);
      }
      tile_max = group16_max(tile_max);
      const float next = fmaxf(m[i], tile_max);
      const float correction = expf(m[i] - next);
      float row_sum = 0.0f;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const float p = valid[j] ? expf(s[i][j] - next) : 0.0f;
        Ps[ty + 16 * i][tx + 16 * j] = p;
        row_sum += p;
      }
      row_sum = group16_sum(row_sum);
      l[i] = l[i] * correction + row_sum;
      m[i] = next;
#pragma unroll
      for (int c = 0; c < DC; ++c) acc[i][c] *= correction;
    }
    __syncthreads();
    mm_nn<MI, DC, BN, kPitch<DP>>(acc, Ps, Vs, ty, tx);
  }
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int query = qt * BM + ty + 16 * i;
    if (query >= S) continue;
    const float inv = 1.0f / l[i];
    const size_t o_off = (static_cast<size_t>(b) * S + query) * views.out_token + h * views.out_head;
    const T* g = gate ? gate + (static_cast<size_t>(b) * S + query) * views.gate_token + h * views.gate_head
                      : nullptr;
#pragma unroll
    for (int c = 0; c < DC; c += 4) {
      const int d = own_column(tx, c);
      float value[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) value[u] = acc[i][c + u] * inv;
      if (core) store_columns(core + o_off, d, D, out_fours, value);
      if (g) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (d + u >= D) continue;
          // R(R(core) * R(sigmoid(gate))), qwen_attention.cc:103-108
          float factor = sigmoid(load_as_float(g + d + u));
          if (round_gate) {
            factor = bf16_round(factor);
            value[u] = bf16_round(value[u]);
          }
          value[u] *= factor;
        }
      }
      store_columns(out + o_off, d, D, out_fours, value);
    }
    if (tx == 0 && maxima != nullptr) {
      const size_t stat = (static_cast<size_t>(b) * H + h) * S + query;
      maxima[stat] = m[i];
      normalizers[stat] = l[i];
    }
  }
}

// ------------------------------------------------------------------------------------------
// probabilities [B,H,S,S] from the saved statistics: grid (query tiles, heads, batch)
// ------------------------------------------------------------------------------------------
template <typename T, int DP, int BM>
__global__ void __launch_bounds__(kThreads)
attn_probs_generic(const T* __restrict__ qkv, const float* __restrict__ maxima,
                   const float* __restrict__ normalizers, float* __restrict__ probs, Dims dims) {
  constexpr int BN = BM, MI = BM / 16, NJ = BN / 16;
  extern __shared__ __align__(16) float smem[];
  float(*Qs)[kPitch<DP>] = reinterpret_cast<float(*)[kPitch<DP>]>(smem);
  float(*Ks)[kPitch<DP>] = Qs + BM;
  const int S = dims.seq, H = dims.heads, D = dims.head_dim, E = H * D;
  const int qt = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  const size_t stride = 3 * static_cast<size_t>(E);
  const T* base = qkv + static_cast<size_t>(b) * S * stride + static_cast<size_t>(h) * D;
  const bool fours = by_fours(qkv, stride, D, D);
  load_tile<T, BM, DP>(Qs, base, stride, qt * BM, S, D, fours);
  float m[MI], inv[MI];
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int query = qt * BM + ty + 16 * i;
    const size_t stat = (static_cast<size_t>(b) * H + h) * S + min(query, S - 1);
    m[i] = maxima[stat];
    inv[i] = 1.0f / normalizers[stat];
  }
  const int tiles = (S + BN - 1) / BN;
  for (int kt = 0; kt < tiles; ++kt) {
    __syncthreads();
    if (kt <= qt) load_tile<T, BN, DP>(Ks, base + E, stride, kt * BN, S, D, fours);
    __syncthreads();
    float s[MI][NJ];
    if (kt <= qt) mm_nt<MI, NJ, kPitch<DP>>(s, Qs, Ks, D, ty, tx);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int query = qt * BM + ty + 16 * i;
      if (query >= S) continue;
      float* row = probs + ((static_cast<size_t>(b) * H + h) * S + query) * S;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int key = kt * BN + tx + 16 * j;
        if (key >= S) continue;
        row[key] = (kt <= qt && key <= query) ? expf(s[i][j] * dims.scale - m[i]) * inv[i] : 0.0f;
      }
    }
  }
}

// Addressing for the backward passes: element strides of the separate tensors.  `group` query
// heads share one key/value head; the packed [rows, 3E] layout is the special case with all token
// strides 3E, head strides D and group 1.
struct BwdViews {
  size_t q_token, q_head, kv_token, kv_head;      // q, and k/v (indexed by key/value head)
  size_t o_token, o_head;                         // saved output (only when deltas are computed here)
  size_t g_token, g_head;                         // upstream gradient (fp32)
  size_t dq_token, dq_head, dkv_token, dkv_head;  // gradients (fp32)
  int group;
};

// ------------------------------------------------------------------------------------------
// backward, query-owned pass: deltas and dQ.  A CTA per (query tile, query head, sequence).
// With `out` null the deltas were written by the caller (gate backward) and are only read.
// ------------------------------------------------------------------------------------------
template <typename T, int DP, int BM>
__global__ void __launch_bounds__(kThreads)
attn_bwd_dq_generic(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                    const T* __restrict__ out, const float* __restrict__ d_out,
                    const float* __restrict__ maxima, const float* __restrict__ normalizers,
                    float* __restrict__ dq, float* __restrict__ deltas, Dims dims, BwdViews views) {
  constexpr int BN = BM, MI = BM / 16, NJ = BN / 16, DC = DP / 16;
  extern __shared__ __align__(16) float smem[];
  float(*Qs)[kPitch<DP>] = reinterpret_cast<float(*)[kPitch<DP>]>(smem);
  float(*Gs)[kPitch<DP>] = Qs + BM;  // upstream gradient dO
  float(*Ks)[kPitch<DP>] = Gs + BM;
  float(*Vs)[kPitch<DP>] = Ks + BN;
  float(*Ps)[kPitch<BN>] = reinterpret_cast<float(*)[kPitch<BN>]>(Vs + BN);

  const int S = dims.seq, H = dims.heads, D = dims.head_dim;
  const Unit unit = block_unit(H, dims);
  const int qt = (S + BM - 1) / BM - 1 - unit.tile, h = unit.head, b = unit.batch;
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  const T* q_base = q + static_cast<size_t>(b) * S * views.q_token + h * views.q_head;
  const T* k_base = k + static_cast<size_t>(b) * S * views.kv_token + (h / views.group) * views.kv_head;
  const T* v_base = v + static_cast<size_t>(b) * S * views.kv_token + (h / views.group) * views.kv_head;
  const bool q_fours = by_fours(q, views.q_token, views.q_head, D);
  const bool kv_fours = by_fours(k, views.kv_token, views.kv_head, D) && by_fours(v, views.kv_token, views.kv_head, D);
  const bool g_fours = by_fours(d_out, views.g_token, views.g_head, D);
  const bool dq_fours = by_fours(dq, views.dq_token, views.dq_head, D);
  const float* g_base = d_out + static_cast<size_t>(b) * S * views.g_token + h * views.g_head;

  load_tile<T, BM, DP>(Qs, q_base, views.q_token, qt * BM, S, D, q_fours);
  load_tile<float, BM, DP>(Gs, g_base, views.g_token, qt * BM, S, D, g_fours);
  if (out != nullptr)  // borrow Ks for the saved output
    load_tile<T, BM, DP>(Ks, out + static_cast<size_t>(b) * S * views.o_token + h * views.o_head,
                         views.o_token, qt * BM, S, D, by_fours(out, views.o_token, views.o_head, D));
  __syncthreads();
  float m[MI], inv[MI], delta[MI], acc[MI][DC];
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int r = ty + 16 * i;
    const int query = qt * BM + r;
    const size_t stat = (static_cast<size_t>(b) * H + h) * S + min(query, S - 1);
    if (out != nullptr) {
      float part = 0.0f;
      for (int d = tx; d < D; d += 16) part = fmaf(Gs[r][d], Ks[r][d], part);
      delta[i] = group16_sum(part);
      if (tx == 0 && query < S) deltas[stat] = delta[i];
    } else {
      delta[i] = deltas[stat];
    }
    m[i] = maxima[stat];
    inv[i] = 1.0f / normalizers[stat];
#pragma unroll
    for (int c = 0; c < DC; ++c) acc[i][c] = 0.0f;
  }
  for (int kt = 0; kt <= qt; ++kt) {
    __syncthreads();
    load_tile<T, BN, DP>(Ks, k_base, views.kv_token, kt * BN, S, D, kv_fours);
    load_tile<T, BN, DP>(Vs, v_base, views.kv_token, kt * BN, S, D, kv_fours);
    __syncthreads();
    float s[MI][NJ], dp[MI][NJ];
    mm_nt<MI, NJ, kPitch<DP>>(s, Qs, Ks, D, ty, tx);
    mm_nt<MI, NJ, kPitch<DP>>(dp, Gs, Vs, D, ty, tx);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int query = qt * BM + ty + 16 * i;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int key = kt * BN + tx + 16 * j;
        const bool valid = key <= query && key < S && query < S;
        const float p = valid ? expf(s[i][j] * dims.scale - m[i]) * inv[i] : 0.0f;
        Ps[ty + 16 * i][tx + 16 * j] = p * (dp[i][j] - delta[i]) * dims.scale;
      }
    }
    __syncthreads();
    mm_nn<MI, DC, BN, kPitch<DP>>(acc, Ps, Ks, ty, tx);
  }
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int query = qt * BM + ty + 16 * i;
    if (query >= S) continue;
    float* row = dq + (static_cast<size_t>(b) * S + query) * views.dq_token + h * views.dq_head;
#pragma unroll
    for (int c = 0; c < DC; c += 4) {
      const float value[4] = {acc[i][c], acc[i][c + 1], acc[i][c + 2], acc[i][c + 3]};
      store_columns(row, own_column(tx, c), D, dq_fours, value);
    }
  }
}

// ------------------------------------------------------------------------------------------
// backward, key/value-owned pass: dK and dV.  A CTA per (key tile, key/value head, sequence).  The
// query heads of the group and the query tiles are visited in a fixed order (single writer).
// ------------------------------------------------------------------------------------------
template <typename T, int DP, int BM>
__global__ void __launch_bounds__(kThreads)
attn_bwd_dkv_generic(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                     const float* __restrict__ d_out, const float* __restrict__ maxima,
                     const float* __restrict__ normalizers, const float* __restrict__ deltas,
                     float* __restrict__ dk_out, float* __restrict__ dv_out, Dims dims,
                     BwdViews views) {
  constexpr int BN = BM, MI = BM / 16, NJ = BN / 16, DC = DP / 16;
  extern __shared__ __align__(16) float smem[];
  float(*Qs)[kPitch<DP>] = reinterpret_cast<float(*)[kPitch<DP>]>(smem);
  float(*Gs)[kPitch<DP>] = Qs + BM;
  float(*Ks)[kPitch<DP>] = Gs + BM;
  float(*Vs)[kPitch<DP>] = Ks + BN;
  float(*Ps)[kPitch<BN>] = reinterpret_cast<float(*)[kPitch<BN>]>(Vs + BN);
  float(*Ss)[kPitch<BN>] = Ps + BM;  // dS

  const int S = dims.seq, H = dims.heads, D = dims.head_dim;
  const Unit unit = block_unit(H / views.group, dims);
  const int kt = unit.tile, kvh = unit.head, b = unit.batch;   // the first key tile sees the most queries
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  const T* k_base = k + static_cast<size_t>(b) * S * views.kv_token + kvh * views.kv_head;
  const T* v_base = v + static_cast<size_t>(b) * S * views.kv_token + kvh * views.kv_head;

  const bool q_fours = by_fours(q, views.q_token, views.q_head, D);
  const bool kv_fours = by_fours(k, views.kv_token, views.kv_head, D) && by_fours(v, views.kv_token, views.kv_head, D);
  const bool g_fours = by_fours(d_out, views.g_token, views.g_head, D);
  const bool dkv_fours = by_fours(dk_out, views.dkv_token, views.dkv_head, D) &&
                         by_fours(dv_out, views.dkv_token, views.dkv_head, D);

  load_tile<T, BN, DP>(Ks, k_base, views.kv_token, kt * BN, S, D, kv_fours);
  load_tile<T, BN, DP>(Vs, v_base, views.kv_token, kt * BN, S, D, kv_fours);
  float dk[MI][DC], dv[MI][DC];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int c = 0; c < DC; ++c) dk[i][c] = dv[i][c] = 0.0f;
  const int tiles = (S + BM - 1) / BM;
  for (int h = kvh * views.group; h < (kvh + 1) * views.group; ++h) {
    const T* q_base = q + static_cast<size_t>(b) * S * views.q_token + h * views.q_head;
    const float* g_base = d_out + static_cast<size_t>(b) * S * views.g_token + h * views.g_head;
    for (int qt = kt; qt < tiles; ++qt) {
      __syncthreads();
      load_tile<T, BM, DP>(Qs, q_base, views.q_token, qt * BM, S, D, q_fours);
      load_tile<float, BM, DP>(Gs, g_base, views.g_token, qt * BM, S, D, g_fours);
      __syncthreads();
      float s[MI][NJ], dp[MI][NJ];
      mm_nt<MI, NJ, kPitch<DP>>(s, Qs, Ks, D, ty, tx);
      mm_nt<MI, NJ, kPitch<DP>>(dp, Gs, Vs, D, ty, tx);
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int query = qt * BM + ty + 16 * i;
        const size_t stat = (static_cast<size_t>(b) * H + h) * S + min(query, S - 1);
        const float m = maxima[stat], inv = 1.0f / normalizers[stat], delta = deltas[stat];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const int key = kt * BN + tx + 16 * j;
          const bool valid = key <= query && key < S && query < S;
          const float p = valid ? expf(s[i][j] * dims.scale - m) * inv : 0.0f;
          Ps[ty + 16 * i][tx + 16 * j] = p;
          Ss[ty + 16 * i][tx + 16 * j] = p * (dp[i][j] - delta) * dims.scale;
        }
      }
      __syncthreads();
      mm_tn<MI, DC, BN, kPitch<DP>>(dv, Ps, Gs, ty, tx);
      mm_tn<MI, DC, BN, kPitch<DP>>(dk, Ss, Qs, ty, tx);
    }
  }
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int key = kt * BN + ty * MI + i;
    if (key >= S) continue;
    const size_t off = (static_cast<size_t>(b) * S + key) * views.dkv_token + kvh * views.dkv_head;
#pragma unroll
    for (int c = 0; c < DC; c += 4) {
      const int d = own_column(tx, c);
      const float dk4[4] = {dk[i][c], dk[i][c + 1], dk[i][c + 2], dk[i][c + 3]};
      const float dv4[4] = {dv[i][c], dv[i][c + 1], dv[i][c + 2], dv[i][c + 3]};
      store_columns(dk_out + off, d, D, dkv_fours, dk4);
      store_columns(dv_out + off, d, D, dkv_fours, dv4);
    }
  }
}

template <int DP, int BM>
constexpr size_t fwd_smem() { return sizeof(float) * (3 * BM * kPitch<DP> + BM * kPitch<BM>); }
template <int DP, int BM>
constexpr size_t probs_smem() { return sizeof(float) * (2 * BM * kPitch<DP>); }
template <int DP, int BM>
constexpr size_t dq_smem() { return sizeof(float) * (4 * BM * kPitch<DP> + BM * kPitch<BM>); }
template <int DP, int BM>
constexpr size_t dkv_smem() { return sizeof(float) * (4 * BM * kPitch<DP> + 2 * BM * kPitch<BM>); }

template <typename K>
cudaError_t opt_in(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(bytes));
}

// One CTA per (tile, head, sequence), as many sequences a launch as keep the block count in range.
template <typename Launch>
cudaError_t launch_units(int tiles, int heads, int batch, Dims dims, Launch launch) {
  const long long per_sequence = static_cast<long long>(tiles) * heads;
  const int step = static_cast<int>(std::max(1LL, std::min<long long>(batch, 0x7fffffffLL / per_sequence)));
  for (dims.batch0 = 0; dims.batch0 < batch; dims.batch0 += step) {
    dims.batch = std::min(step, batch - dims.batch0);
    launch(static_cast<unsigned>(per_sequence * dims.batch), dims);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <typename T, int DP, int BM>
cudaError_t launch_fwd(cudaStream_t stream, const void* q, const void* k, const void* v, void* out,
                       float* maxima, float* normalizers, const void* gate, float* core,
                       int round_gate, int batch, Dims dims, Views views) {
  auto kernel = attn_fwd_generic<T, DP, BM>;
  cudaError_t e = opt_in(kernel, fwd_smem<DP, BM>());
  if (e != cudaSuccess) return e;
  return launch_units((dims.seq + BM - 1) / BM, dims.heads, batch, dims, [&](unsigned grid, const Dims& d) {
    kernel<<<grid, kThreads, fwd_smem<DP, BM>(), stream>>>(
        static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v),
        static_cast<T*>(out), maxima, normalizers, static_cast<const T*>(gate), core, round_gate, d, views);
  });
}
template <typename T, int DP, int BM>
cudaError_t launch_probs(cudaStream_t stream, const void* qkv, const float* maxima,
                         const float* normalizers, float* probs, int batch, Dims dims) {
  auto kernel = attn_probs_generic<T, DP, BM>;
  cudaError_t e = opt_in(kernel, probs_smem<DP, BM>());
  if (e != cudaSuccess) return e;
  dim3 grid((dims.seq + BM - 1) / BM, dims.heads, batch);
  kernel<<<grid, kThreads, probs_smem<DP, BM>(), stream>>>(static_cast<const T*>(qkv), maxima,
                                                           normalizers, probs, dims);
  return cudaGetLastError();
}
template <typename T, int DP, int BM>
cudaError_t launch_bwd(cudaStream_t stream, const void* q, const void* k, const void* v,
                       const void* out, const float* d_out, const float* maxima,
                       const float* normalizers, float* dq_out, float* dk_out, float* dv_out,
                       float* deltas, int batch, Dims dims, BwdViews views) {
  auto dq = attn_bwd_dq_generic<T, DP, BM>;
  auto dkv = attn_bwd_dkv_generic<T, DP, BM>;
  cudaError_t e = opt_in(dq, dq_smem<DP, BM>());
  if (e != cudaSuccess) return e;
  e = opt_in(dkv, dkv_smem<DP, BM>());
  if (e != cudaSuccess) return e;
  const int tiles = (dims.seq + BM - 1) / BM;
  e = launch_units(tiles, dims.heads, batch, dims, [&](unsigned grid, const Dims& d) {
    dq<<<grid, kThreads, dq_smem<DP, BM>(), stream>>>(
        static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v),
        static_cast<const T*>(out), d_out, maxima, normalizers, dq_out, deltas, d, views);
  });
  if (e != cudaSuccess) return e;
  // Same-stream ordering makes every delta visible to the key/value-owned pass.
  return launch_units(tiles, dims.heads / views.group, batch, dims, [&](unsigned grid, const Dims& d) {
    dkv<<<grid, kThreads, dkv_smem<DP, BM>(), stream>>>(
        static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v), d_out, maxima,
        normalizers, deltas, dk_out, dv_out, d, views);
  });
}

}  // namespace

// Forward over separate Q/K/V tensors.  Strides are in elements; `group` query heads share one
// key/value head.  The packed [rows, 3E] layout of AttentionLayer is the special case
// q = qkv, k = qkv + E, v = qkv + 2E with token stride 3E (see c_api.cu).
cudaError_t attn_generic_fwd(cudaStream_t stream, const void* q, const void* k, const void* v,
                             void* out, float* maxima, float* normalizers, int batch, int seq,
                             int heads, int head_dim, size_t q_token, size_t q_head,
                             size_t kv_token, size_t kv_head, size_t out_token, size_t out_head,
                             int group, const void* gate, size_t gate_token, size_t gate_head,
                             float* core, int round_gate, bool bf16) {
  Dims dims{seq, heads, head_dim, batch, 0, 1.0f / sqrtf(static_cast<float>(head_dim))};
  Views views{q_token, q_head, kv_token, kv_head, out_token, out_head, gate_token, gate_head, group};
#define CALL_FWD(T, DP, BM) \
  launch_fwd<T, DP, BM>(stream, q, k, v, out, maxima, normalizers, gate, core, round_gate, \
                        batch, dims, views)
  if (bf16) {
    if (head_dim <= 64) return CALL_FWD(__nv_bfloat16, 64, 64);
    if (head_dim <= 128) return CALL_FWD(__nv_bfloat16, 128, 64);
    return CALL_FWD(__nv_bfloat16, 256, 32);
  }
  if (head_dim <= 64) return CALL_FWD(float, 64, 64);
  if (head_dim <= 128) return CALL_FWD(float, 128, 64);
  return CALL_FWD(float, 256, 32);
#undef CALL_FWD
}

cudaError_t attn_generic_probs(cudaStream_t stream, const void* qkv, const float* maxima,
                               const float* normalizers, float* probs, int batch, int seq,
                               int heads, int head_dim, bool bf16) {
  Dims dims{seq, heads, head_dim, batch, 0, 1.0f / sqrtf(static_cast<float>(head_dim))};
#define CALL_P(T, DP, BM) launch_probs<T, DP, BM>(stream, qkv, maxima, normalizers, probs, batch, dims)
  if (bf16) {
    if (head_dim <= 64) return CALL_P(__nv_bfloat16, 64, 64);
    if (head_dim <= 128) return CALL_P(__nv_bfloat16, 128, 64);
    return CALL_P(__nv_bfloat16, 256, 32);
  }
  if (head_dim <= 64) return CALL_P(float, 64, 64);
  if (head_dim <= 128) return CALL_P(float, 128, 64);
  return CALL_P(float, 256, 32);
#undef CALL_P
}

cudaError_t attn_generic_bwd(cudaStream_t stream, const void* qkv, const void* out,
                             const float* d_out, const float* maxima, const float* normalizers,
                             float* d_qkv, float* deltas, int batch, int seq, int heads,
                             int head_dim, bool bf16) {
  const size_t E = static_cast<size_t>(heads) * head_dim, D = head_dim;
  const size_t elem = bf16 ? 2 : 4;
  const char* base = static_cast<const char*>(qkv);
  GqaBwdArgs a{};
  a.q = base;
  a.k = base + E * elem;
  a.v = base + 2 * E * elem;
  a.out = out;
  a.d_out = d_out;
  a.maxima = maxima;
  a.normalizers = normalizers;
  a.deltas = deltas;
  a.dq = d_qkv;
  a.dk = d_qkv + E;
  a.dv = d_qkv + 2 * E;
  a.batch = batch; a.seq = seq; a.q_heads = heads; a.kv_heads = heads; a.head_dim = head_dim;
  a.q_token = a.kv_token = a.dq_token = a.dkv_token = 3 * E;
  a.q_head = a.kv_head = a.dq_head = a.dkv_head = a.o_head = a.g_head = D;
  a.o_token = a.g_token = E;
  a.bf16 = bf16;
  return gqa_generic_bwd(stream, a);
}

// Backward of the attention core over separate tensors with grouped query heads (the Qwen
// sequence layer): see GqaBwdArgs in engine.h.
cudaError_t gqa_generic_bwd(cudaStream_t stream, const GqaBwdArgs& a) {
  Dims dims{a.seq, a.q_heads, a.head_dim, a.batch, 0, 1.0f / sqrtf(static_cast<float>(a.head_dim))};
  BwdViews views{a.q_token, a.q_head, a.kv_token, a.kv_head, a.o_token, a.o_head, a.g_token,
                 a.g_head, a.dq_token, a.dq_head, a.dkv_token, a.dkv_head, a.q_heads / a.kv_heads};
#define CALL_B(T, DP, BM)                                                                        \
  launch_bwd<T, DP, BM>(stream, a.q, a.k, a.v, a.out, a.d_out, a.maxima, a.normalizers, a.dq, a.dk, \
                        a.dv, a.deltas, a.batch, dims, views)
  if (a.bf16) {
    if (a.head_dim <= 64) return CALL_B(__nv_bfloat16, 64, 64);
    if (a.head_dim <= 128) return CALL_B(__nv_bfloat16, 128, 64);
    return CALL_B(__nv_bfloat16, 256, 32);
  }
  if (a.head_dim <= 64) return CALL_B(float, 64, 64);
  if (a.head_dim <= 128) return CALL_B(float, 128, 64);
  return CALL_B(float, 256, 32);
#undef CALL_B
}

}  // namespace pluto
