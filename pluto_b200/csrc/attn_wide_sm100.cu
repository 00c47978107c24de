// Causal attention of head width 256 on the Blackwell tensor cores, forward and backward (the Qwen
// decoder's default width: 24 query heads over 4 key/value heads).  bf16 tensors, fp32
// accumulation; every fp32 quantity that becomes an operand of a second product (the
// probabilities P, the score gradient dS, the upstream gradient dO) enters it as a bf16 high part
// plus a bf16 remainder, 2^-17 relative, far below the layer's own bf16 rounding points: at 64 to 2048
// tokens its output and gradients differ from float64 by 2.5e-3 to 4.1e-3, to three digits what they
// differ by with the fp32 kernels in attn_generic.cu that this width ran on before (the unrounded core by
// 2e-6, there 3e-7).  At 1000 tokens those took 1078 us forward, 2258 dQ and 3798 dK/dV, these 44, 53
// and 99 + 11.
// Reference: src/llm/layers/qwen_attention.cc:68-119 (forward), :140-190 (backward).
//
// The width decides the layout.  An fp32 accumulator tile of 128 rows x 256 channels takes half of
// the SM's tensor memory, a bf16 tile of 128 rows x 256 channels 64 KB of its shared memory:
//   attn_fwd_wide      128 queries per CTA; two score buffers of 128 keys and O fill TMEM.  K passes
//                      through a ring of 16 KB slots as slabs of 64 channels, V as runs of 32 keys,
//                      in the order the products consume them.
//   attn_bwd_dq_wide   128 queries per CTA, 64 keys per step; Q as a TMEM operand, dO (high part and
//                      remainder) resident in shared memory.
//   attn_bwd_dkv_wide  128 keys per CTA, 64 queries per step.  dV and dK of all 256 channels would
//                      fill TMEM by themselves, so a CTA owns 128 channels of both and its twin the
//                      others; the scores are computed by both (11 products per step against 8).
//                      CTAs also split over the query heads of a key/value head while there are too
//                      few of them, and attn_bwd_sum_wide adds the parts up in a fixed order.
// Two threads share a row in all three: warpgroup g takes columns [w g, w g + w) of a step (w = half
// a step) and writes what it makes of them - high parts in the first half of its own columns,
// remainders in the second - over exactly the columns that it read, so the two never wait for each
// other there.  All waits are bounded; no TMA multicast.
#include "common.cuh"
#include "engine.h"

namespace pluto {
namespace {

constexpr int kD = 256;
constexpr int kRows = 128;                    // rows a CTA owns (TMEM lanes)
constexpr int kSlabBytes = kRows * 128;       // [128 rows x 64 bf16]
constexpr int kTileBytes = 4 * kSlabBytes;    // [128 rows x 256 bf16]
constexpr int kStep = 64;                     // opposite-side rows of a backward step
constexpr int kStepSlab = kStep * 128;        // [64 rows x 64 bf16]
constexpr int kStepBytes = 4 * kStepSlab;     // [64 rows x 256 bf16]
constexpr int kWideThreads = 384;             // warp 0 loads, warp 1 issues MMAs, warps 4-11 own rows
constexpr float kLog2e = 1.4426950408889634f;

// hi[i] = the bf16 high parts of values 2i, 2i+1; lo[i] = their remainders.
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(a, b);
  lo = pack_bf16(a - bf16_lo(hi), b - bf16_hi(hi));
}

// A staging tile of fp32 rows of kRowBytes in shared memory: 16-byte chunk c of row r lies at chunk
// position c ^ (r & 7), so that a warp writing one chunk of 32 rows spreads over the banks.
template <int kRowBytes>
__device__ __forceinline__ uint32_t staged_chunk(uint32_t base, int row, int chunk) {
  return base + row * kRowBytes + ((chunk ^ (row & 7)) << 4);
}
template <int kRowBytes>
__device__ __forceinline__ void stage_32(uint32_t base, int row, int chunk0, const uint32_t (&o)[32], float factor) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
    sts_b32x4(staged_chunk<kRowBytes>(base, row, chunk0 + i), __float_as_uint(__uint_as_float(o[4 * i]) * factor),
              __float_as_uint(__uint_as_float(o[4 * i + 1]) * factor),
              __float_as_uint(__uint_as_float(o[4 * i + 2]) * factor),
              __float_as_uint(__uint_as_float(o[4 * i + 3]) * factor));
}

// ------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------
constexpr int kFwdSlots = 9;
constexpr int kRunBytes = 32 * 128;           // [32 keys x 64 bf16] of V
constexpr float kRescaleThreshold = 8.0f;     // log2 units

struct WideFwdParams {
  int q_col0, k_col0, v_col0, q_head_cols;
  int seq, heads, group;
  float scale, scale_log2;
  __nv_bfloat16* out;
  size_t out_token, out_head;
  float *maxima, *normalizers, *core;
  const __nv_bfloat16* gate;
  size_t gate_token, gate_head;
  int round_gate;
  uint32_t* status;
};
struct WideFwdBarriers {
  uint64_t q_full, full[kFwdSlots], empty[kFwdSlots], s_full[2], p_full[2], pv_done[2];
  uint32_t tmem_base;
};
constexpr int kFwdExchange = 2 * 2 * kRows * 4;   // row maxima: two steps x two warpgroups
constexpr int kFwdSmem = 1024 + kTileBytes + kFwdSlots * kSlabBytes + kFwdExchange + sizeof(WideFwdBarriers);

__global__ void __launch_bounds__(kWideThreads, 1)
attn_fwd_wide(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
              const __grid_constant__ CUtensorMap map_v32, WideFwdParams p) {
  constexpr uint32_t kColO = 256;
  constexpr uint32_t kIdescS = umma_idesc_bf16(kRows, 128, false);
  constexpr uint32_t kIdescO = umma_idesc_bf16(kRows, kD, true);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* ring = smem + kTileBytes;
  const uint32_t exchange = smem_u32(ring + kFwdSlots * kSlabBytes);
  WideFwdBarriers* bar = reinterpret_cast<WideFwdBarriers*>(ring + kFwdSlots * kSlabBytes + kFwdExchange);

  const int warp = uniform_warp_index(), lane = threadIdx.x % 32;
  // (sequence, head) fastest, longest query tiles first
  const int q_tile = gridDim.y - 1 - blockIdx.y;
  const int head = blockIdx.x % p.heads, batch = blockIdx.x / p.heads;
  const int n_tiles = q_tile + 1;

  if (threadIdx.x == 0) {
    mbar_init(&bar->q_full, 1);
    for (int s = 0; s < kFwdSlots; ++s) {
      mbar_init(&bar->full[s], 1);
      mbar_init(&bar->empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar->s_full[s], 1);
      mbar_init(&bar->p_full[s], 8);   // one arrival per softmax warp
      mbar_init(&bar->pv_done[s], 1);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&bar->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bar->tmem_base;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&map_q);
      tma_prefetch_desc(&map_k);
      tma_prefetch_desc(&map_v32);
      const int kv_head = head / p.group;
      mbar_expect_tx(&bar->q_full, kTileBytes);
      for (int s = 0; s < 4; ++s)
        tma_load_3d(smem + s * kSlabBytes, &map_q, p.q_col0 + head * p.q_head_cols + s * 64, q_tile * kRows, batch,
                    &bar->q_full);
      // K_0, then K_j and V_{j-1} in turn, then the last V: the order of the products
      int n = 0;
      bool ok = true;
      auto slot = [&]() -> uint8_t* {
        const int st = n % kFwdSlots, use = n / kFwdSlots;
        if (use > 0) ok = mbar_wait(&bar->empty[st], (use - 1) & 1, p.status, 100);
        if (ok) mbar_expect_tx(&bar->full[st], kSlabBytes);
        return ring + st * kSlabBytes;
      };
      auto load_k = [&](int j) {
        for (int s = 0; s < 4 && ok; ++s) {
          uint8_t* dst = slot();
          if (!ok) return;
          tma_load_3d(dst, &map_k, p.k_col0 + kv_head * kD + s * 64, j * kRows, batch, &bar->full[n % kFwdSlots]);
          ++n;
        }
      };
      auto load_v = [&](int j) {
        for (int c = 0; c < 4 && ok; ++c) {
          uint8_t* dst = slot();
          if (!ok) return;
          for (int s = 0; s < 4; ++s)
            tma_load_3d(dst + s * kRunBytes, &map_v32, p.v_col0 + kv_head * kD + s * 64, j * kRows + c * 32, batch,
                        &bar->full[n % kFwdSlots]);
          ++n;
        }
      };
      load_k(0);
      for (int j = 1; j < n_tiles && ok; ++j) {
        load_k(j);
        if (ok) load_v(j - 1);
      }
      if (ok) load_v(n_tiles - 1);
      mbar_wait(&bar->q_full, 0, p.status, 101);   // no copy may be in flight when the CTA leaves
      for (int i = max(0, n - kFwdSlots); i < n; ++i)
        mbar_wait(&bar->full[i % kFwdSlots], (i / kFwdSlots) & 1, p.status, 102);
    }
  } else if (warp == 1) {
    int n = 0;
    const uint32_t ring_base = smem_u32(ring);
    const uint64_t q_desc = umma_desc_sw128(smem_u32(smem), 16, 1024);
    bool ok = __all_sync(0xffffffffu, mbar_wait(&bar->q_full, 0, p.status, 103));
    auto arrived = [&]() -> bool {
      const bool good = __all_sync(0xffffffffu, mbar_wait(&bar->full[n % kFwdSlots], (n / kFwdSlots) & 1, p.status, 104));
      tc_fence_after();
      return good;
    };
    auto issue_s = [&](int j) -> bool {   // S(j) = Q K_j^T
      for (int s = 0; s < 4; ++s, ++n) {
        if (!arrived()) return false;
        if (elect_one()) {
          const uint64_t k_desc = umma_desc_sw128(ring_base + (n % kFwdSlots) * kSlabBytes, 16, 1024);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            umma_ss(tmem + (j & 1) * 128, q_desc + ((s * kSlabBytes + i * 32) >> 4), k_desc + ((i * 32) >> 4), kIdescS,
                    s > 0 || i > 0);
          tc_commit(&bar->empty[n % kFwdSlots]);
          if (s == 3) tc_commit(&bar->s_full[j & 1]);
        }
        __syncwarp();
      }
      return true;
    };
    auto issue_pv = [&](int j) -> bool {   // O += P_hi V_j + P_lo V_j, 32 keys at a time
      if (!__all_sync(0xffffffffu, mbar_wait(&bar->p_full[j & 1], (j >> 1) & 1, p.status, 105))) return false;
      for (int c = 0; c < 4; ++c, ++n) {
        if (!arrived()) return false;
        if (elect_one()) {
          const uint64_t v_desc = umma_desc_sw128(ring_base + (n % kFwdSlots) * kSlabBytes, kRunBytes, 1024);
          const uint32_t own = tmem + (j & 1) * 128 + (c >> 1) * 64 + (c & 1) * 16;
#pragma unroll
          for (int i = 0; i < 4; ++i)   // key half i & 1; high part, then remainder
            umma_ts(tmem + kColO, own + (i >> 1) * 32 + (i & 1) * 8, v_desc + (((i & 1) * 2048) >> 4), kIdescO,
                    j > 0 || c > 0 || i > 0);
          tc_commit(&bar->empty[n % kFwdSlots]);
          if (c == 3) tc_commit(&bar->pv_done[j & 1]);
        }
        __syncwarp();
      }
      return true;
    };
    for (int j = 0; j < n_tiles && ok; ++j) {
      ok = issue_s(j);
      if (ok && j > 0) ok = issue_pv(j - 1);
    }
    if (ok) issue_pv(n_tiles - 1);
  } else if (warp >= 4) {
    const int g = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const int query = q_tile * kRows + row;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t o_addr = tmem + lane_base + kColO + g * 128;
    float m_used = -INFINITY, m_true = -INFINITY, l = 0.0f;
    bool ok = true;
    // (no early exit: the two warpgroups meet at a barrier in every step, whatever their waits say)
    for (int j = 0; j < n_tiles; ++j) {
      const uint32_t s_addr = tmem + lane_base + (j & 1) * 128 + g * 64;
      ok = ok && mbar_wait(&bar->s_full[j & 1], (j >> 1) & 1, p.status, 106);
      uint32_t s[2][32];
      float local = -INFINITY;
      if (ok) {
        tc_fence_after();
        tmem_ld32(s_addr, s[0]);
        tmem_ld32(s_addr + 32, s[1]);
        tmem_wait_ld();
        if (j == q_tile) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (g * 64 + c * 32 + i > row) s[c][i] = 0xff800000u;   // -inf above the diagonal
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            mx[(i >> 1) & 3] = max3(mx[(i >> 1) & 3], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
        local = fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]);
      }
      const uint32_t own = exchange + (j & 1) * 2 * kRows * 4 + row * 4;
      sts_f32(own + g * kRows * 4, local);
      named_barrier_sync(1, 256);
      if (!ok) continue;
      m_true = max3(m_true, local, lds_f32(own + (g ^ 1) * kRows * 4));
      // both threads of a row see the same maxima, so they rescale in the same steps
      const bool grow = (m_true - m_used) * p.scale_log2 > kRescaleThreshold;
      if (__any_sync(0xffffffffu, grow)) {
        const float factor = grow ? fast_exp2((m_used - m_true) * p.scale_log2) : 1.0f;
        if (grow) m_used = m_true;
        l *= factor;
        if (j > 0) {
          ok = mbar_wait(&bar->pv_done[(j - 1) & 1], ((j - 1) >> 1) & 1, p.status, 107);
          if (!ok) continue;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            tmem_ld32(o_addr + c * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
            tmem_st32(o_addr + c * 32, o);
          }
        }
      }
      const float neg_m = -m_used * p.scale_log2;
      float sum[2] = {0.0f, 0.0f};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = fast_exp2(fmaf(__uint_as_float(s[c][i]), p.scale_log2, neg_m));
          const float p1 = fast_exp2(fmaf(__uint_as_float(s[c][i + 1]), p.scale_log2, neg_m));
          split_pair(p0, p1, hi[i / 2], lo[i / 2]);
          // the sum of what the product sees: an error of a P then weighs V minus the result, not V
          sum[0] += bf16_lo(hi[i / 2]) + bf16_lo(lo[i / 2]);
          sum[1] += bf16_hi(hi[i / 2]) + bf16_hi(lo[i / 2]);
        }
        tmem_st16(s_addr + c * 16, hi);
        tmem_st16(s_addr + 32 + c * 16, lo);
      }
      l += sum[0] + sum[1];
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->p_full[j & 1]);
    }
    // The gate of the eight channels this thread will write of each of sixteen rows, requested while the
    // last product runs and kept in shared memory behind the staging tile, so that the store loop
    // below is a loop: unrolled, its 128 sigmoids are code that runs once and is fetched cold (13 us
    // per CTA), and with the loads inside, every row waits for its own.
    const int t256 = threadIdx.x - 128, c8 = t256 & 31;   // row t256 / 32 + 8 u, channels 8 c8 ..
    uint4 gates[16];
    if (p.gate) {
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int r = min(q_tile * kRows + (t256 >> 5) + 8 * u, p.seq - 1);
        gates[u] = *reinterpret_cast<const uint4*>(p.gate + (static_cast<size_t>(batch) * p.seq + r) * p.gate_token +
                                                   head * p.gate_head + c8 * 8);
      }
    }
    ok = ok && mbar_wait(&bar->pv_done[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1, p.status, 108);
    // l of the whole row; the rows then leave through shared memory (Q and the first slots are free
    // by now), coalesced, with the gate applied on the way
    const uint32_t own = exchange + (n_tiles & 1) * 2 * kRows * 4 + row * 4;
    sts_f32(own + g * kRows * 4, l);
    named_barrier_sync(1, 256);
    l += lds_f32(own + (g ^ 1) * kRows * 4);
    const uint32_t stage = smem_u32(smem), own_gate = stage + 2 * kTileBytes + t256 * 16;
    static_assert(kTileBytes + kFwdSlots * kSlabBytes >= 3 * kTileBytes, "staging tile and gate");
    if (ok) {
      if (p.gate) {
#pragma unroll
        for (int u = 0; u < 16; ++u) sts_b32x4(own_gate + u * 4096, gates[u].x, gates[u].y, gates[u].z, gates[u].w);
      }
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld32(o_addr + c * 32, o);
        tmem_wait_ld();
        // (a division: one rounding where a product with 1 / l has two; core is saved as fp32)
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) / l);
        stage_32<1024>(stage, row, g * 32 + c * 8, o, 1.0f);
      }
      if (g == 0 && query < p.seq && p.maxima) {
        const size_t stat = (static_cast<size_t>(batch) * p.heads + head) * p.seq + query;
        p.maxima[stat] = m_true * p.scale;
        p.normalizers[stat] = l * fast_exp2((m_used - m_true) * p.scale_log2);
      }
    }
    named_barrier_sync(1, 256);
    if (ok) {
#pragma unroll 1
      for (int u = 0; u < 16; ++u) {
        const int r = (t256 >> 5) + 8 * u;
        if (q_tile * kRows + r >= p.seq) continue;
        const size_t token = static_cast<size_t>(batch) * p.seq + q_tile * kRows + r;
        const size_t at = token * p.out_token + head * p.out_head + c8 * 8;
        const float4 a = lds_f32x4(staged_chunk<1024>(stage, r, 2 * c8));
        const float4 b = lds_f32x4(staged_chunk<1024>(stage, r, 2 * c8 + 1));
        float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        if (p.core) {
          *reinterpret_cast<float4*>(p.core + at) = a;
          *reinterpret_cast<float4*>(p.core + at + 4) = b;
        }
        if (p.gate) {
          const uint4 raw = lds_b32x4(own_gate + u * 4096);   // written by this thread
          const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float x = (i & 1) ? bf16_hi(w[i / 2]) : bf16_lo(w[i / 2]);
            float sigmoid = sigmoid_fast(x);
            if (p.round_gate) {
              sigmoid = bf16_round(sigmoid);
              v[i] = bf16_round(v[i]);
            }
            v[i] *= sigmoid;
          }
        }
        *reinterpret_cast<uint4*>(p.out + at) =
            make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------
// backward
// ------------------------------------------------------------------------------------------------
struct WideBwdParams {
  int q_col0, k_col0, v_col0;
  int seq, seq_pad, heads, group, heads_per_cta;
  float scale, scale_log2;
  const float2* stats;     // [(b*heads + h) * seq_pad + s] = (-(max*log2e + log2 l), delta); padding (-1e30, 0)
  float *dq, *dk, *dv;     // dk / dv: the outputs, or the partial sums [part][b][s][kv_head][D]
  size_t dq_token, dkv_token, part_stride;
  uint32_t* status;
};

// dO as bf16 high parts and remainders, and the row statistics.  One warp per padded (head, row):
// head-major, so the statistics are written in runs; a row of dO is a whole kilobyte either way.
__global__ void __launch_bounds__(256)
attn_bwd_prep_wide(const __nv_bfloat16* __restrict__ out, const float* __restrict__ d_out,
                   const float* __restrict__ maxima, const float* __restrict__ normalizers,
                   float* deltas, __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo,
                   float2* __restrict__ stats, int seq, int seq_pad, int heads, long long rows) {
  pdl_launch_dependents();
  const long long padded = static_cast<long long>(blockIdx.x) * 8 + threadIdx.x / 32;
  if (padded >= rows) return;
  const int lane = threadIdx.x % 32, s = static_cast<int>(padded % seq_pad);
  const long long unit = padded / seq_pad;   // (sequence, head)
  if (s >= seq) {
    if (lane == 0) stats[padded] = make_float2(-1.0e30f, 0.0f);
    return;
  }
  const long long b = unit / heads, h = unit % heads;
  const size_t base = ((static_cast<size_t>(b) * seq + s) * heads + h) * kD + lane * 8;
  const float4 g0 = *reinterpret_cast<const float4*>(d_out + base), g1 = *reinterpret_cast<const float4*>(d_out + base + 4);
  uint4 high, low;
  split_pair(g0.x, g0.y, high.x, low.x);
  split_pair(g0.z, g0.w, high.y, low.y);
  split_pair(g1.x, g1.y, high.z, low.z);
  split_pair(g1.z, g1.w, high.w, low.w);
  *reinterpret_cast<uint4*>(hi + base) = high;
  *reinterpret_cast<uint4*>(lo + base) = low;
  const size_t stat = static_cast<size_t>(unit) * seq + s;
  float delta = 0.0f;
  if (out != nullptr) {
    const uint4 o = *reinterpret_cast<const uint4*>(out + base);
    delta = g0.x * bf16_lo(o.x) + g0.y * bf16_hi(o.x) + g0.z * bf16_lo(o.y) + g0.w * bf16_hi(o.y) +
            g1.x * bf16_lo(o.z) + g1.y * bf16_hi(o.z) + g1.z * bf16_lo(o.w) + g1.w * bf16_hi(o.w);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) delta += __shfl_xor_sync(0xffffffffu, delta, off);
    if (lane == 0) deltas[stat] = delta;
  } else {
    delta = deltas[stat];
  }
  if (lane == 0) stats[padded] = make_float2(-(maxima[stat] * kLog2e + log2f(normalizers[stat])), delta);
}

struct WideDqBarriers {
  uint64_t do_full, q_full, rows_ready, k_full[2], k_empty[2], v_full[4], v_empty[4];
  uint64_t s_full, dp_full, loaded, ds_ready, done;
  uint32_t tmem_base;
};
constexpr int kDqSmem = 1024 + 2 * kTileBytes + 3 * kStepBytes + sizeof(WideDqBarriers);

// Tensor work of a step (64 keys): S 1, dP 2 (dO high part and remainder), dQ 2 (dS likewise) of
// [128 x 64 x 256].  The row threads read S and dP into registers at once, so dP(j+1) runs while
// they compute; dS(j) takes S's columns, so S(j+1) follows dQ(j).
__global__ void __launch_bounds__(kWideThreads, 1)
attn_bwd_dq_wide(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k64,
                 const __grid_constant__ CUtensorMap map_v64, const __grid_constant__ CUtensorMap map_hi,
                 const __grid_constant__ CUtensorMap map_lo, WideBwdParams p) {
  constexpr uint32_t kColS = 0, kColDP = 64, kColQ = 128, kColDQ = 256;
  constexpr uint32_t kIdescS = umma_idesc_bf16(kRows, kStep, false);
  constexpr uint32_t kIdescDQ = umma_idesc_bf16(kRows, kD, true);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* do_hi = smem;
  uint8_t* do_lo = do_hi + kTileBytes;
  uint8_t* k_ring = do_lo + kTileBytes;         // two stages; Q passes through them on its way into TMEM
  uint8_t* v_slabs = k_ring + 2 * kStepBytes;   // one step, slab by slab
  WideDqBarriers* bar = reinterpret_cast<WideDqBarriers*>(v_slabs + kStepBytes);

  const int warp = uniform_warp_index(), lane = threadIdx.x % 32;
  const int q_tile = gridDim.y - 1 - blockIdx.y;
  const int head = blockIdx.x % p.heads, batch = blockIdx.x / p.heads;
  const int kv_head = head / p.group;
  const int n_steps = min(2 * q_tile + 2, (p.seq + kStep - 1) / kStep);

  if (threadIdx.x == 0) {
    mbar_init(&bar->do_full, 1);
    mbar_init(&bar->q_full, 1);
    mbar_init(&bar->rows_ready, 8);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar->k_full[s], 1);
      mbar_init(&bar->k_empty[s], 1);
    }
    for (int s = 0; s < 4; ++s) {
      mbar_init(&bar->v_full[s], 1);
      mbar_init(&bar->v_empty[s], 1);
    }
    mbar_init(&bar->s_full, 1);
    mbar_init(&bar->dp_full, 1);
    mbar_init(&bar->loaded, 8);
    mbar_init(&bar->ds_ready, 8);
    mbar_init(&bar->done, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&bar->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bar->tmem_base;
  pdl_wait();   // the prep kernel's operands and statistics are complete from here on
  pdl_launch_dependents();

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&map_k64);
      tma_prefetch_desc(&map_v64);
      mbar_expect_tx(&bar->q_full, kTileBytes);
      for (int s = 0; s < 4; ++s)
        tma_load_3d(k_ring + s * kSlabBytes, &map_q, p.q_col0 + head * kD + s * 64, q_tile * kRows, batch, &bar->q_full);
      mbar_expect_tx(&bar->do_full, 2 * kTileBytes);
      for (int s = 0; s < 4; ++s) {
        tma_load_3d(do_hi + s * kSlabBytes, &map_hi, head * kD + s * 64, q_tile * kRows, batch, &bar->do_full);
        tma_load_3d(do_lo + s * kSlabBytes, &map_lo, head * kD + s * 64, q_tile * kRows, batch, &bar->do_full);
      }
      bool ok = true;
      int k_used = 0, v_used[4] = {0, 0, 0, 0};
      for (int j = 0; j < n_steps && ok; ++j) {
        for (int s = 0; s < 4 && ok; ++s) {
          if (j > 0) ok = mbar_wait(&bar->v_empty[s], (j - 1) & 1, p.status, 110);
          if (!ok) break;
          mbar_expect_tx(&bar->v_full[s], kStepSlab);
          tma_load_3d(v_slabs + s * kStepSlab, &map_v64, p.v_col0 + kv_head * kD + s * 64, j * kStep, batch,
                      &bar->v_full[s]);
          ++v_used[s];
        }
        if (j == 0 && ok) ok = mbar_wait(&bar->rows_ready, 0, p.status, 111);
        if (j >= 2 && ok) ok = mbar_wait(&bar->k_empty[j & 1], ((j >> 1) - 1) & 1, p.status, 112);
        if (!ok) break;
        mbar_expect_tx(&bar->k_full[j & 1], kStepBytes);
        for (int s = 0; s < 4; ++s)
          tma_load_3d(k_ring + (j & 1) * kStepBytes + s * kStepSlab, &map_k64, p.k_col0 + kv_head * kD + s * 64,
                      j * kStep, batch, &bar->k_full[j & 1]);
        ++k_used;
      }
      // no copy may be in flight when the CTA leaves
      mbar_wait(&bar->q_full, 0, p.status, 113);
      mbar_wait(&bar->do_full, 0, p.status, 113);
      for (int s = 0; s < 4; ++s)
        if (v_used[s] > 0) mbar_wait(&bar->v_full[s], (v_used[s] - 1) & 1, p.status, 114);
      for (int j = max(0, k_used - 2); j < k_used; ++j) mbar_wait(&bar->k_full[j & 1], (j >> 1) & 1, p.status, 114);
    }
  } else if (warp == 1) {
    const uint64_t hi_desc = umma_desc_sw128(smem_u32(do_hi), 16, 1024);
    const uint64_t lo_desc = umma_desc_sw128(smem_u32(do_lo), 16, 1024);
    const uint32_t k_base = smem_u32(k_ring), v_base = smem_u32(v_slabs);
    auto issue_dp = [&](int j) -> bool {   // dP(j) = (dO_hi + dO_lo) V_j^T
      for (int s = 0; s < 4; ++s) {
        if (!__all_sync(0xffffffffu, mbar_wait(&bar->v_full[s], j & 1, p.status, 115))) return false;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t v_desc = umma_desc_sw128(v_base + s * kStepSlab, 16, 1024);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t off = (s * kSlabBytes + i * 32) >> 4;
            umma_ss(tmem + kColDP, hi_desc + off, v_desc + ((i * 32) >> 4), kIdescS, s > 0 || i > 0);
            umma_ss(tmem + kColDP, lo_desc + off, v_desc + ((i * 32) >> 4), kIdescS, true);
          }
          tc_commit(&bar->v_empty[s]);
          if (s == 3) tc_commit(&bar->dp_full);
        }
        __syncwarp();
      }
      return true;
    };
    auto issue_s = [&](int j) -> bool {   // S(j) = Q K_j^T
      if (!__all_sync(0xffffffffu, mbar_wait(&bar->k_full[j & 1], (j >> 1) & 1, p.status, 116))) return false;
      tc_fence_after();
      if (elect_one()) {
        const uint64_t k_desc = umma_desc_sw128(k_base + (j & 1) * kStepBytes, 16, 1024);
#pragma unroll
        for (int ks = 0; ks < kD / 16; ++ks)
          umma_ts(tmem + kColS, tmem + kColQ + ks * 8, k_desc + (((ks / 4) * kStepSlab + (ks % 4) * 32) >> 4), kIdescS,
                  ks > 0);
        tc_commit(&bar->s_full);
      }
      __syncwarp();
      return true;
    };
    bool ok = __all_sync(0xffffffffu, mbar_wait(&bar->do_full, 0, p.status, 117));
    if (ok) ok = issue_dp(0);
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&bar->rows_ready, 0, p.status, 118));
    if (ok) ok = issue_s(0);
    for (int j = 0; j < n_steps && ok; ++j) {
      if (j + 1 < n_steps) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bar->loaded, j & 1, p.status, 119));
        if (ok) ok = issue_dp(j + 1);
        if (!ok) break;
      }
      ok = __all_sync(0xffffffffu, mbar_wait(&bar->ds_ready, j & 1, p.status, 120));
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint64_t k_mn = umma_desc_sw128(k_base + (j & 1) * kStepBytes, kStepSlab, 1024);
#pragma unroll
        for (int ks = 0; ks < kStep / 16; ++ks)
#pragma unroll
          for (int part = 0; part < 2; ++part)
            umma_ts(tmem + kColDQ, tmem + kColS + (ks >> 1) * 32 + part * 16 + (ks & 1) * 8, k_mn + ks * (2048 >> 4),
                    kIdescDQ, j > 0 || ks > 0 || part > 0);
        tc_commit(&bar->k_empty[j & 1]);
      }
      __syncwarp();
      if (j + 1 < n_steps) ok = issue_s(j + 1);
    }
    if (ok && elect_one()) tc_commit(&bar->done);
    __syncwarp();
  } else if (warp >= 4) {
    const int g = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const int query = q_tile * kRows + row;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    bool ok = mbar_wait(&bar->q_full, 0, p.status, 121);
    if (ok) {   // this thread's half of its query row into TMEM
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        uint32_t w[32];
        load_swizzled_row(smem_u32(k_ring) + (2 * g + s) * kSlabBytes, row, w);
        tmem_st32(tmem + lane_base + kColQ + (2 * g + s) * 32, w);
      }
      tmem_wait_st();
      fence_proxy_async();
      tc_fence_before();
    }
    __syncwarp();
    if (ok && lane == 0) mbar_arrive(&bar->rows_ready);
    const float2 st = p.stats[(static_cast<size_t>(batch) * p.heads + head) * p.seq_pad + min(query, p.seq_pad - 1)];
    const float shift = st.x, delta = st.y;
    const uint32_t s_addr = tmem + lane_base + kColS + g * 32, dp_addr = tmem + lane_base + kColDP + g * 32;
    for (int j = 0; j < n_steps && ok; ++j) {
      ok = mbar_wait(&bar->s_full, j & 1, p.status, 122) && mbar_wait(&bar->dp_full, j & 1, p.status, 123);
      if (!ok) break;
      tc_fence_after();
      uint32_t s[32], dp[32];
      tmem_ld32(s_addr, s);
      tmem_ld32(dp_addr, dp);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->loaded);
      const int key0 = j * kStep + g * 32;
      const bool masked = j >= 2 * q_tile;
      uint32_t hi[16], lo[16];
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float p0 = fast_exp2(fmaf(__uint_as_float(s[i]), p.scale_log2, shift));
        float p1 = fast_exp2(fmaf(__uint_as_float(s[i + 1]), p.scale_log2, shift));
        if (masked) {
          if (key0 + i > query) p0 = 0.0f;
          if (key0 + i + 1 > query) p1 = 0.0f;
        }
        split_pair(p0 * (__uint_as_float(dp[i]) - delta), p1 * (__uint_as_float(dp[i + 1]) - delta), hi[i / 2], lo[i / 2]);
      }
      tmem_st16(s_addr, hi);
      tmem_st16(s_addr + 16, lo);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->ds_ready);
    }
    ok = ok && mbar_wait(&bar->done, 0, p.status, 124);
    // dQ leaves through the dO tiles, scaled
    const uint32_t stage = smem_u32(smem);
    if (ok) {
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld32(tmem + lane_base + kColDQ + g * 128 + c * 32, o);
        tmem_wait_ld();
        stage_32<1024>(stage, row, g * 32 + c * 8, o, p.scale);
      }
    }
    named_barrier_sync(1, 256);
    if (ok) {
#pragma unroll 4
      for (int e = threadIdx.x - 128; e < kRows * 64; e += 256) {
        const int r = e >> 6, c = e & 63;
        if (q_tile * kRows + r >= p.seq) continue;
        const size_t token = static_cast<size_t>(batch) * p.seq + q_tile * kRows + r;
        *reinterpret_cast<float4*>(p.dq + token * p.dq_token + head * kD + c * 4) =
            lds_f32x4(staged_chunk<1024>(stage, r, c));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

constexpr int kDkvSlots = 5;
struct WideDkvBarriers {
  uint64_t v_full, k_full, rows_ready, full[kDkvSlots], empty[kDkvSlots], s_full, stored, done;
  uint32_t tmem_base;
};
constexpr int kDkvStats = 2 * kStep * 8;   // two steps of (shift, delta)
constexpr int kDkvSmem = 1024 + kTileBytes + kDkvSlots * kStepBytes + kDkvStats + sizeof(WideDkvBarriers);

// grid (2 channel halves x (batch x query heads / heads_per_cta), key tiles).  The ring carries
// Q, dO_hi and dO_lo of a step as items 3i, 3i+1, 3i+2; item n lies in slot (n + 2) % 5, so that the
// first three leave slots 0 and 1 to K on its way into TMEM.
__global__ void __launch_bounds__(kWideThreads, 1)
attn_bwd_dkv_wide(const __grid_constant__ CUtensorMap map_q64, const __grid_constant__ CUtensorMap map_k,
                  const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_hi64,
                  const __grid_constant__ CUtensorMap map_lo64, WideBwdParams p) {
  constexpr uint32_t kColS = 0, kColDP = 64, kColDV = 128, kColDK = 256, kColK = 384;
  constexpr uint32_t kIdescS = umma_idesc_bf16(kRows, kStep, false);
  constexpr uint32_t kIdescAcc = umma_idesc_bf16(kRows, 128, true);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* v_smem = smem;
  uint8_t* ring = v_smem + kTileBytes;
  uint8_t* stat_ring = ring + kDkvSlots * kStepBytes;
  WideDkvBarriers* bar = reinterpret_cast<WideDkvBarriers*>(stat_ring + kDkvStats);

  const int warp = uniform_warp_index(), lane = threadIdx.x % 32;
  const int half = blockIdx.x & 1, k_tile = blockIdx.y;   // the first key tile sees the most queries
  const int head_sets = p.heads / p.heads_per_cta;
  const int set = (blockIdx.x >> 1) % head_sets, batch = (blockIdx.x >> 1) / head_sets;
  const int head0 = set * p.heads_per_cta, kv_head = head0 / p.group;
  const int part = (head0 % p.group) / p.heads_per_cta;
  const int per_head = (p.seq + kStep - 1) / kStep - 2 * k_tile;   // steps of one query head
  const int n_steps = p.heads_per_cta * per_head;

  if (threadIdx.x == 0) {
    mbar_init(&bar->v_full, 1);
    mbar_init(&bar->k_full, 1);
    mbar_init(&bar->rows_ready, 8);
    for (int s = 0; s < kDkvSlots; ++s) {
      mbar_init(&bar->full[s], 1);
      mbar_init(&bar->empty[s], 1);
    }
    mbar_init(&bar->s_full, 1);
    mbar_init(&bar->stored, 8);
    mbar_init(&bar->done, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&bar->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bar->tmem_base;
  // The dQ kernel lets this grid start as soon as every one of its CTAs has seen the prep kernel
  // complete; nothing it writes is read here, so its last CTAs and this grid's first share the chip.
  pdl_launch_dependents();

  // Item n's slot, and which use of the slot's barriers it is (slots 0 and 1 come in a round later).
  auto slot_of = [](int n) { return (n + 2) % kDkvSlots; };
  auto use_of = [](int n) { return (n + 2) / kDkvSlots - ((n + 2) % kDkvSlots < 2 ? 1 : 0); };

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(&bar->k_full, kTileBytes);
      for (int s = 0; s < 4; ++s)
        tma_load_3d(ring + s * kSlabBytes, &map_k, p.k_col0 + kv_head * kD + s * 64, k_tile * kRows, batch, &bar->k_full);
      mbar_expect_tx(&bar->v_full, kTileBytes);
      for (int s = 0; s < 4; ++s)
        tma_load_3d(v_smem + s * kSlabBytes, &map_v, p.v_col0 + kv_head * kD + s * 64, k_tile * kRows, batch, &bar->v_full);
      bool ok = true;
      int n = 0;
      for (int i = 0; i < n_steps && ok; ++i) {
        const int head = head0 + i / per_head, q0 = (2 * k_tile + i % per_head) * kStep;
        for (int item = 0; item < 3 && ok; ++item) {
          const int st = slot_of(n), use = use_of(n);
          if (n == 3) ok = mbar_wait(&bar->rows_ready, 0, p.status, 130);
          if (use > 0 && ok) ok = mbar_wait(&bar->empty[st], (use - 1) & 1, p.status, 131);
          if (!ok) break;
          mbar_expect_tx(&bar->full[st], kStepBytes + (item == 0 ? kStep * 8 : 0));
          const CUtensorMap* map = item == 0 ? &map_q64 : item == 1 ? &map_hi64 : &map_lo64;
          const int col = item == 0 ? p.q_col0 + head * kD : head * kD;
          for (int s = 0; s < 4; ++s)
            tma_load_3d(ring + st * kStepBytes + s * kStepSlab, map, col + s * 64, q0, batch, &bar->full[st]);
          if (item == 0)   // the other half of stat_ring belongs to the step before, this one to a finished step
            bulk_load(stat_ring + (i & 1) * kStep * 8,
                      p.stats + (static_cast<size_t>(batch) * p.heads + head) * p.seq_pad + q0, kStep * 8, &bar->full[st]);
          ++n;
        }
      }
      mbar_wait(&bar->k_full, 0, p.status, 132);
      mbar_wait(&bar->v_full, 0, p.status, 132);
      for (int i = max(0, n - kDkvSlots); i < n; ++i) mbar_wait(&bar->full[slot_of(i)], use_of(i) & 1, p.status, 133);
    }
  } else if (warp == 1) {
    const uint32_t ring_base = smem_u32(ring);
    const uint64_t v_desc = umma_desc_sw128(smem_u32(v_smem), 16, 1024);
    auto arrived = [&](int n) -> bool {
      const bool good = __all_sync(0xffffffffu, mbar_wait(&bar->full[slot_of(n)], use_of(n) & 1, p.status, 134));
      tc_fence_after();
      return good;
    };
    bool ok = __all_sync(0xffffffffu, mbar_wait(&bar->v_full, 0, p.status, 135) &&
                                          mbar_wait(&bar->rows_ready, 0, p.status, 136));
    for (int i = 0; i < n_steps && ok; ++i) {
      const uint32_t slot[3] = {ring_base + slot_of(3 * i) * kStepBytes, ring_base + slot_of(3 * i + 1) * kStepBytes,
                                ring_base + slot_of(3 * i + 2) * kStepBytes};
      ok = arrived(3 * i);
      if (!ok) break;
      if (elect_one()) {   // S^T = K Q^T
        const uint64_t q_desc = umma_desc_sw128(slot[0], 16, 1024);
#pragma unroll
        for (int ks = 0; ks < kD / 16; ++ks)
          umma_ts(tmem + kColS, tmem + kColK + ks * 8, q_desc + (((ks / 4) * kStepSlab + (ks % 4) * 32) >> 4), kIdescS,
                  ks > 0);
      }
      __syncwarp();
#pragma unroll
      for (int part_of = 0; part_of < 2; ++part_of) {   // dP^T = V (dO_hi + dO_lo)^T
        ok = ok && arrived(3 * i + 1 + part_of);
        if (ok && elect_one()) {
          const uint64_t do_desc = umma_desc_sw128(slot[1 + part_of], 16, 1024);
#pragma unroll
          for (int ks = 0; ks < kD / 16; ++ks)
            umma_ss(tmem + kColDP, v_desc + (((ks / 4) * kSlabBytes + (ks % 4) * 32) >> 4),
                    do_desc + (((ks / 4) * kStepSlab + (ks % 4) * 32) >> 4), kIdescS, part_of > 0 || ks > 0);
          if (part_of == 1) tc_commit(&bar->s_full);
        }
        __syncwarp();
      }
      if (!ok) break;
      ok = __all_sync(0xffffffffu, mbar_wait(&bar->stored, i & 1, p.status, 137));
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        // this CTA's 128 channels, MN-major: 16 queries per instruction
        const uint32_t columns = half * 2 * kStepSlab;
        const uint64_t q_mn = umma_desc_sw128(slot[0] + columns, kStepSlab, 1024);
        const uint64_t hi_mn = umma_desc_sw128(slot[1] + columns, kStepSlab, 1024);
        const uint64_t lo_mn = umma_desc_sw128(slot[2] + columns, kStepSlab, 1024);
#pragma unroll
        for (int ks = 0; ks < kStep / 16; ++ks) {
          const uint32_t own = (ks >> 1) * 32 + (ks & 1) * 8;
          const uint32_t off = ks * (2048 >> 4);
          const bool more = i > 0 || ks > 0;
          umma_ts(tmem + kColDV, tmem + kColS + own, hi_mn + off, kIdescAcc, more);          // P_hi dO_hi
          umma_ts(tmem + kColDV, tmem + kColS + own, lo_mn + off, kIdescAcc, true);          // P_hi dO_lo
          umma_ts(tmem + kColDV, tmem + kColS + own + 16, hi_mn + off, kIdescAcc, true);     // P_lo dO_hi
          umma_ts(tmem + kColDK, tmem + kColDP + own, q_mn + off, kIdescAcc, more);          // dS_hi Q
          umma_ts(tmem + kColDK, tmem + kColDP + own + 16, q_mn + off, kIdescAcc, true);     // dS_lo Q
        }
        tc_commit(&bar->empty[slot_of(3 * i)]);
        tc_commit(&bar->empty[slot_of(3 * i + 1)]);
        tc_commit(&bar->empty[slot_of(3 * i + 2)]);
      }
      __syncwarp();
    }
    if (ok && elect_one()) tc_commit(&bar->done);
    __syncwarp();
  } else if (warp >= 4) {
    const int g = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const int key = k_tile * kRows + row;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    bool ok = mbar_wait(&bar->k_full, 0, p.status, 138);
    if (ok) {   // this thread's half of its key row into TMEM
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        uint32_t w[32];
        load_swizzled_row(smem_u32(ring) + (2 * g + s) * kSlabBytes, row, w);
        tmem_st32(tmem + lane_base + kColK + (2 * g + s) * 32, w);
      }
      tmem_wait_st();
      fence_proxy_async();
      tc_fence_before();
    }
    __syncwarp();
    if (ok && lane == 0) mbar_arrive(&bar->rows_ready);
    const uint32_t s_addr = tmem + lane_base + kColS + g * 32, dp_addr = tmem + lane_base + kColDP + g * 32;
    for (int i = 0; i < n_steps && ok; ++i) {
      ok = mbar_wait(&bar->s_full, i & 1, p.status, 139) &&
           mbar_wait(&bar->full[slot_of(3 * i)], use_of(3 * i) & 1, p.status, 140);   // the statistics landed
      if (!ok) break;
      tc_fence_after();
      uint32_t s[32], dp[32];
      tmem_ld32(s_addr, s);
      tmem_ld32(dp_addr, dp);
      tmem_wait_ld();
      const int local = i % per_head, query0 = (2 * k_tile + local) * kStep + g * 32;
      const bool masked = local < 2;
      const uint32_t stats = smem_u32(stat_ring) + (i & 1) * kStep * 8 + g * 32 * 8;
      uint32_t hi[16], lo[16];
#pragma unroll
      for (int c = 0; c < 32; c += 2) {
        const float4 st = lds_f32x4(stats + c * 8);   // (shift, delta) of two queries, the same for the whole warp
        float p0 = fast_exp2(fmaf(__uint_as_float(s[c]), p.scale_log2, st.x));
        float p1 = fast_exp2(fmaf(__uint_as_float(s[c + 1]), p.scale_log2, st.z));
        if (masked) {
          if (query0 + c < key) p0 = 0.0f;
          if (query0 + c + 1 < key) p1 = 0.0f;
        }
        split_pair(p0, p1, hi[c / 2], lo[c / 2]);
        dp[c] = __float_as_uint(p0 * (__uint_as_float(dp[c]) - st.y));
        dp[c + 1] = __float_as_uint(p1 * (__uint_as_float(dp[c + 1]) - st.w));
      }
      tmem_st16(s_addr, hi);
      tmem_st16(s_addr + 16, lo);
#pragma unroll
      for (int c = 0; c < 32; c += 2)
        split_pair(__uint_as_float(dp[c]), __uint_as_float(dp[c + 1]), hi[c / 2], lo[c / 2]);
      tmem_st16(dp_addr, hi);
      tmem_st16(dp_addr + 16, lo);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->stored);
    }
    ok = ok && mbar_wait(&bar->done, 0, p.status, 141);
    // dV (warpgroup 0) and dK (warpgroup 1) leave through the ring: [128 rows x 128] fp32 each
    const uint32_t stage = smem_u32(ring) + g * kRows * 512;
    if (ok) {
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld32(tmem + lane_base + (g == 0 ? kColDV : kColDK) + c * 32, o);
        tmem_wait_ld();
        stage_32<512>(stage, row, c * 8, o, g == 0 ? 1.0f : p.scale);
      }
    }
    named_barrier_sync(1, 256);
    if (ok) {
      float* dst = (g == 0 ? p.dv : p.dk) + part * p.part_stride + kv_head * kD + half * 128;
#pragma unroll 4
      for (int e = (threadIdx.x - 128) & 127; e < kRows * 32; e += 128) {
        const int r = e >> 5, c = e & 31;
        if (k_tile * kRows + r >= p.seq) continue;
        const size_t token = static_cast<size_t>(batch) * p.seq + k_tile * kRows + r;
        *reinterpret_cast<float4*>(dst + token * p.dkv_token + c * 4) = lds_f32x4(staged_chunk<512>(stage, r, c));
      }
    }
  }
  if (threadIdx.x == 0) pdl_wait();   // this grid completes after the dQ kernel, whatever follows it
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// dk / dv [token][width] (token stride dkv_token) = sum over parts, in order.  One thread per four
// channels; grid.y picks dK or dV.
__global__ void __launch_bounds__(256)
attn_bwd_sum_wide(const float* __restrict__ part_dk, const float* __restrict__ part_dv, int parts, size_t part_stride,
                  int width, long long count, float* __restrict__ dk, float* __restrict__ dv, size_t dkv_token) {
  pdl_wait();
  const long long i = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) * 4;
  if (i >= count) return;
  const float* src = blockIdx.y == 0 ? part_dk : part_dv;
  float4 sum = *reinterpret_cast<const float4*>(src + i);
  for (int part = 1; part < parts; ++part) {
    const float4 v = *reinterpret_cast<const float4*>(src + part * part_stride + i);
    sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
  }
  float* dst = (blockIdx.y == 0 ? dk : dv) + (i / width) * dkv_token + i % width;
  *reinterpret_cast<float4*>(dst) = sum;
}

int padded_rows(int seq) { return (seq + kStep - 1) / kStep * kStep; }

template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                           Args&&... args) {
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, args...);
}

template <typename K>
cudaError_t opt_in(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace

cudaError_t attn_fwd_wide_tc(cudaStream_t stream, const AttnFwdArgs& a) {
  CUtensorMap map_q, map_k, map_v;
  if (a.head_dim != kD || !make_token_map(&map_q, a.q, a.q_cols, a.seq, a.batch, a.q_token, kRows) ||
      !make_token_map(&map_k, a.k, a.kv_cols, a.seq, a.batch, a.kv_token, kRows) ||
      !make_token_map(&map_v, a.v, a.kv_cols, a.seq, a.batch, a.kv_token, 32))
    return cudaErrorInvalidValue;
  WideFwdParams p;
  p.q_col0 = a.q_col0; p.k_col0 = a.k_col0; p.v_col0 = a.v_col0; p.q_head_cols = a.q_head_cols;
  p.seq = a.seq; p.heads = a.heads; p.group = a.group;
  p.scale = 1.0f / sqrtf(static_cast<float>(kD));
  p.scale_log2 = p.scale * kLog2e;
  p.out = static_cast<__nv_bfloat16*>(a.out);
  p.out_token = a.out_token; p.out_head = a.out_head;
  p.maxima = a.maxima; p.normalizers = a.normalizers; p.core = a.core;
  p.gate = static_cast<const __nv_bfloat16*>(a.gate);
  p.gate_token = a.gate_token; p.gate_head = a.gate_head;
  p.round_gate = a.round_gate;
  p.status = a.status;
  if (cudaError_t e = opt_in(attn_fwd_wide, kFwdSmem); e != cudaSuccess) return e;
  attn_fwd_wide<<<dim3(a.heads * a.batch, (a.seq + kRows - 1) / kRows), kWideThreads, kFwdSmem, stream>>>(map_q, map_k,
                                                                                                          map_v, p);
  return cudaGetLastError();
}

// The upstream gradient's high parts and remainders, the statistics, and dK / dV partial sums for as
// many parts as a group can have query heads.
size_t attn_bwd_wide_workspace_bytes(int batch, int seq, int heads) {
  const size_t rows = static_cast<size_t>(batch) * seq * heads;
  return rows * kD * 4 + static_cast<size_t>(batch) * heads * padded_rows(seq) * sizeof(float2) + 256 + 2 * rows * kD * 4;
}

cudaError_t attn_bwd_wide_tc(cudaStream_t stream, const GqaBwdTcArgs& a) {
  const int seq_pad = padded_rows(a.seq), tiles = (a.seq + kRows - 1) / kRows, group = a.q_heads / a.kv_heads;
  const size_t rows = static_cast<size_t>(a.batch) * a.seq * a.q_heads;
  auto* hi = static_cast<__nv_bfloat16*>(a.workspace);
  auto* lo = hi + rows * kD;
  float2* stats = reinterpret_cast<float2*>(lo + rows * kD);
  const size_t stat_rows = static_cast<size_t>(a.batch) * a.q_heads * seq_pad;
  float* parts = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(stats + stat_rows) + 255) & ~static_cast<uintptr_t>(255));
  attn_bwd_prep_wide<<<static_cast<unsigned>((stat_rows + 7) / 8), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(a.out), a.d_out, a.maxima, a.normalizers, a.deltas, hi, lo, stats, a.seq, seq_pad,
      a.q_heads, static_cast<long long>(stat_rows));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int E = a.q_heads * kD;
  CUtensorMap q128, q64, k128, k64, v128, v64, hi128, hi64, lo128, lo64;
  if (!make_token_map(&q128, a.q, a.q_cols, a.seq, a.batch, a.q_token, kRows) ||
      !make_token_map(&q64, a.q, a.q_cols, a.seq, a.batch, a.q_token, kStep) ||
      !make_token_map(&k128, a.k, a.kv_cols, a.seq, a.batch, a.kv_token, kRows) ||
      !make_token_map(&k64, a.k, a.kv_cols, a.seq, a.batch, a.kv_token, kStep) ||
      !make_token_map(&v128, a.v, a.kv_cols, a.seq, a.batch, a.kv_token, kRows) ||
      !make_token_map(&v64, a.v, a.kv_cols, a.seq, a.batch, a.kv_token, kStep) ||
      !make_token_map(&hi128, hi, E, a.seq, a.batch, E, kRows) || !make_token_map(&hi64, hi, E, a.seq, a.batch, E, kStep) ||
      !make_token_map(&lo128, lo, E, a.seq, a.batch, E, kRows) || !make_token_map(&lo64, lo, E, a.seq, a.batch, E, kStep))
    return cudaErrorInvalidValue;
  WideBwdParams p;
  p.q_col0 = a.q_col0; p.k_col0 = a.k_col0; p.v_col0 = a.v_col0;
  p.seq = a.seq; p.seq_pad = seq_pad; p.heads = a.q_heads; p.group = group;
  p.scale = 1.0f / sqrtf(static_cast<float>(kD));
  p.scale_log2 = p.scale * kLog2e;
  p.stats = stats;
  p.dq = a.dq; p.dq_token = a.dq_token;
  p.status = a.status;
  if ((e = opt_in(attn_bwd_dq_wide, kDqSmem)) != cudaSuccess) return e;
  if ((e = opt_in(attn_bwd_dkv_wide, kDkvSmem)) != cudaSuccess) return e;
  p.heads_per_cta = 1;
  p.dk = a.dk; p.dv = a.dv; p.dkv_token = a.dkv_token; p.part_stride = 0;
  // a CTA walks as many query heads of its group as still leaves two CTAs per SM
  const long long units = 2LL * tiles * a.batch * a.q_heads;
  for (int n = group; n > 1; --n)
    if (group % n == 0 && units / n >= 2 * 148) {
      p.heads_per_cta = n;
      break;
    }
  const int n_parts = group / p.heads_per_cta, width = a.kv_heads * kD;
  const size_t part_floats = static_cast<size_t>(a.batch) * a.seq * width;
  if (n_parts > 1) {
    p.dk = parts;
    p.dv = parts + n_parts * part_floats;
    p.part_stride = part_floats;
    p.dkv_token = width;
  }
  e = launch_chained(attn_bwd_dq_wide, dim3(a.q_heads * a.batch, tiles), kWideThreads, kDqSmem, stream, q128, k64, v64,
                     hi128, lo128, p);
  if (e != cudaSuccess) return e;
  e = launch_chained(attn_bwd_dkv_wide, dim3(2 * a.batch * (a.q_heads / p.heads_per_cta), tiles), kWideThreads, kDkvSmem,
                     stream, q64, k128, v128, hi64, lo64, p);
  if (e != cudaSuccess || n_parts == 1) return e;
  return launch_chained(attn_bwd_sum_wide, dim3(static_cast<unsigned>((part_floats / 4 + 255) / 256), 2), 256, 0, stream,
                        static_cast<const float*>(p.dk), static_cast<const float*>(p.dv), n_parts, part_floats, width,
                        static_cast<long long>(part_floats), a.dk, a.dv, a.dkv_token);
}

}  // namespace pluto
