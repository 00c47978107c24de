// Causal attention of head width 256 on the Blackwell tensor cores, forward and backward (the Qwen
// decoder's default width: 24 query heads over 4 key/value heads).  bf16 tensors; every fp32 quantity
// that becomes an operand of a second product (the probabilities P, the score gradient dS, the upstream
// gradient dO) enters it as three bf16 parts, 24 bits, and of the products of two such quantities only
// those below 2^-24 are left out.  The tensor cores truncate when they accumulate (2^-26 of the sum per
// instruction, always towards zero), so no accumulator lives longer than a step: the parts go in from the
// smallest to the largest, and the step's tile is added in fp32 registers; sums over 256
// channels are made in two halves.  Relative error against float64 at 64 to 2048 tokens, N(0, 1) and
// N(0, 1/4) inputs: unrounded core 0.8e-7 to 2.1e-7, dQ 2.5e-7 to 4.0e-7, dK 3.0e-7 to 4.4e-7, dV 1.7e-7 to
// 3.4e-7; the fp32 kernels in attn_generic.cu 0.9e-7 to 3.8e-7, 3.6e-7 to 5.4e-7, 0.5e-6 to 2.1e-6 and 0.4e-6
// to 2.1e-6.  (With two parts and accumulators that live as long as the row: 1.5e-6 to 2.4e-6, 4e-6, 0.4e-5
// to 1.3e-5, 0.4e-5 to 1.8e-5.)  At 1000 tokens of 24 heads the fp32 kernels took 1078 us forward, 2258 dQ and
// 3798 dK/dV, these take 69 with a gate (59 without), 83 and 116 + 10 (the two-part ones 44, 52 and 99 + 11).
// Reference: src/llm/layers/qwen_attention.cc:68-119 (forward), :140-190 (backward).
//
// The width decides the layout.  A bf16 tile of 128 rows x 256 channels takes 64 KB of the SM's shared
// memory or a quarter of its tensor memory, an fp32 tile half of the latter:
//   attn_fwd_wide      128 queries per CTA, 64 keys per step; two score buffers.  K passes through a ring
//                      of 16 KB slots as slabs of 64 channels, V as runs of 32 keys, in the order the
//                      products consume them.
//   attn_bwd_dq_wide   128 queries per CTA, 64 keys per step; Q and the last part of dO are TMEM operands,
//                      the other two parts resident in shared memory.  dQ of a step is made in quarters of
//                      64 channels that two column blocks hold in turn.
//   attn_bwd_dkv_wide  128 keys per CTA, 32 queries per step; V is a TMEM operand, K resident in shared
//                      memory.  dV and dK of all 256 channels would fill TMEM by themselves, so a CTA owns
//                      128 channels of both and its twin the others; the scores are computed by both.
//                      CTAs also split over the query heads of a key/value head while there are too
//                      few of them, and attn_bwd_sum_wide adds the parts up in a fixed order.
// Two threads share a row in all three: warpgroup g takes columns [w g, w g + w) of a step (w = half
// a step) and writes the first two parts of what it makes of them over exactly the columns that it read
// (the third into columns of its own), so the two never wait for each other there; each keeps half of the
// row's fp32 accumulator.  The row threads take over registers of the copy and MMA warps for it.
// All waits are bounded; no TMA multicast.
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

// Two values as three bf16 parts each: part[0] + part[1] + part[2] is the value to 24 bits.
struct Thirds { uint32_t part[3]; };
__device__ __forceinline__ Thirds split_pair(float a, float b) {
  Thirds t;
  t.part[0] = pack_bf16(a, b);
  a -= bf16_lo(t.part[0]);
  b -= bf16_hi(t.part[0]);
  t.part[1] = pack_bf16(a, b);
  t.part[2] = pack_bf16(a - bf16_lo(t.part[1]), b - bf16_hi(t.part[1]));
  return t;
}

// 384 threads have 168 registers each at launch; the copy and MMA warps keep 40.
__device__ __forceinline__ void take_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 224;"); }
__device__ __forceinline__ void give_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 40;"); }

// The sums of 32 columns each of two accumulators: a product over 256 channels is made in two halves, since
// what an accumulator loses grows with the number of instructions that add to it.
__device__ __forceinline__ void load_halves(uint32_t first, uint32_t second, uint32_t (&v)[32]) {
  uint32_t other[32];
  tmem_ld32(first, v);
  tmem_ld32(second, other);
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(other[i]));
}

// acc = acc * factor + the 32 accumulator columns at `from` of this thread's row.
__device__ __forceinline__ void add_columns(uint32_t from, float factor, float* acc) {
  uint32_t o[32];
  tmem_ld32(from, o);
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < 32; ++i) acc[i] = fmaf(acc[i], factor, __uint_as_float(o[i]));
}

// A staging tile of fp32 rows of kRowBytes in shared memory: 16-byte chunk c of row r lies at chunk
// position c ^ (r & 7), so that a warp writing one chunk of 32 rows spreads over the banks.
template <int kRowBytes>
__device__ __forceinline__ uint32_t staged_chunk(uint32_t base, int row, int chunk) {
  return base + row * kRowBytes + ((chunk ^ (row & 7)) << 4);
}
template <int kRowBytes>
__device__ __forceinline__ void stage_32(uint32_t base, int row, int chunk0, const float* v) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
    sts_b32x4(staged_chunk<kRowBytes>(base, row, chunk0 + i), __float_as_uint(v[4 * i]), __float_as_uint(v[4 * i + 1]),
              __float_as_uint(v[4 * i + 2]), __float_as_uint(v[4 * i + 3]));
}

// ------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------
constexpr int kFwdSlots = 9;
constexpr int kSlotBytes = 16384;             // K: two slabs of [64 keys x 64 bf16]; V: four of [32 keys x 64 bf16]
constexpr int kRunBytes = 32 * 128;           // [32 keys x 64 bf16] of V

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
  uint64_t q_full, full[kFwdSlots], empty[kFwdSlots], s_full[2], p_full[2], o_full, o_free;
  uint32_t tmem_base;
};
constexpr int kFwdExchange = 2 * 2 * kRows * 4;   // row maxima: two steps x two warpgroups
constexpr int kFwdSmem = 1024 + kTileBytes + kFwdSlots * kSlotBytes + kFwdExchange + sizeof(WideFwdBarriers);

// Tensor work of a step (64 keys): S 1, PV 3 (the parts of P) of [128 x 64 x 256].  S(j + 1) runs while
// the row threads make P(j) of S(j); behind PV(j - 1), whose tile they add while S(j + 1) still runs.
__global__ void __launch_bounds__(kWideThreads, 1)
attn_fwd_wide(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k64,
              const __grid_constant__ CUtensorMap map_v32, WideFwdParams p) {
  constexpr uint32_t kColS = 0, kColO = 256;   // scores (two buffers of two halves of the channels), step of O
  constexpr uint32_t kIdescS = umma_idesc_bf16(kRows, kStep, false);
  constexpr uint32_t kIdescO = umma_idesc_bf16(kRows, kD, true);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* ring = smem + kTileBytes;
  const uint32_t exchange = smem_u32(ring + kFwdSlots * kSlotBytes);
  WideFwdBarriers* bar = reinterpret_cast<WideFwdBarriers*>(ring + kFwdSlots * kSlotBytes + kFwdExchange);

  const int warp = uniform_warp_index(), lane = threadIdx.x % 32;
  // (sequence, head) fastest, longest query tiles first
  const int q_tile = gridDim.y - 1 - blockIdx.y;
  const int head = blockIdx.x % p.heads, batch = blockIdx.x / p.heads;
  const int n_steps = min(2 * q_tile + 2, (p.seq + kStep - 1) / kStep);

  if (threadIdx.x == 0) {
    mbar_init(&bar->q_full, 1);
    for (int s = 0; s < kFwdSlots; ++s) {
      mbar_init(&bar->full[s], 1);
      mbar_init(&bar->empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar->s_full[s], 1);
      mbar_init(&bar->p_full[s], 8);   // one arrival per row warp
    }
    mbar_init(&bar->o_full, 1);
    mbar_init(&bar->o_free, 8);
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
    give_registers();
    if (lane == 0) {
      tma_prefetch_desc(&map_q);
      tma_prefetch_desc(&map_k64);
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
        if (ok) mbar_expect_tx(&bar->full[st], kSlotBytes);
        return ring + st * kSlotBytes;
      };
      auto load_k = [&](int j) {
        for (int h = 0; h < 2 && ok; ++h) {
          uint8_t* dst = slot();
          if (!ok) return;
          for (int s = 0; s < 2; ++s)
            tma_load_3d(dst + s * kStepSlab, &map_k64, p.k_col0 + kv_head * kD + (2 * h + s) * 64, j * kStep, batch,
                        &bar->full[n % kFwdSlots]);
          ++n;
        }
      };
      auto load_v = [&](int j) {
        for (int h = 0; h < 2 && ok; ++h) {
          uint8_t* dst = slot();
          if (!ok) return;
          for (int s = 0; s < 4; ++s)
            tma_load_3d(dst + s * kRunBytes, &map_v32, p.v_col0 + kv_head * kD + s * 64, j * kStep + h * 32, batch,
                        &bar->full[n % kFwdSlots]);
          ++n;
        }
      };
      load_k(0);
      for (int j = 1; j < n_steps && ok; ++j) {
        load_k(j);
        if (ok) load_v(j - 1);
      }
      if (ok) load_v(n_steps - 1);
      mbar_wait(&bar->q_full, 0, p.status, 101);   // no copy may be in flight when the CTA leaves
      for (int i = max(0, n - kFwdSlots); i < n; ++i)
        mbar_wait(&bar->full[i % kFwdSlots], (i / kFwdSlots) & 1, p.status, 102);
    }
  } else if (warp == 1) {
    give_registers();
    int n = 0;
    const uint32_t ring_base = smem_u32(ring);
    const uint64_t q_desc = umma_desc_sw128(smem_u32(smem), 16, 1024);
    bool ok = __all_sync(0xffffffffu, mbar_wait(&bar->q_full, 0, p.status, 103));
    auto arrived = [&](int item) -> bool {
      const bool good =
          __all_sync(0xffffffffu, mbar_wait(&bar->full[item % kFwdSlots], (item / kFwdSlots) & 1, p.status, 104));
      tc_fence_after();
      return good;
    };
    auto issue_s = [&](int j) -> bool {   // S(j) = Q K_j^T
      for (int h = 0; h < 2; ++h, ++n) {
        if (!arrived(n)) return false;
        if (elect_one()) {
          const uint64_t k_desc = umma_desc_sw128(ring_base + (n % kFwdSlots) * kSlotBytes, 16, 1024);
#pragma unroll
          for (int i = 0; i < 8; ++i)
            umma_ss(tmem + kColS + (j & 1) * 128 + h * kStep, q_desc + (((2 * h + i / 4) * kSlabBytes + i % 4 * 32) >> 4),
                    k_desc + ((i / 4 * kStepSlab + i % 4 * 32) >> 4), kIdescS, i > 0);
          tc_commit(&bar->empty[n % kFwdSlots]);
          if (h == 1) tc_commit(&bar->s_full[j & 1]);
        }
        __syncwarp();
      }
      return true;
    };
    auto issue_pv = [&](int j) -> bool {   // O(j) = P V_j, the parts of P from the last to the first
      if (!__all_sync(0xffffffffu, mbar_wait(&bar->p_full[j & 1], (j >> 1) & 1, p.status, 105))) return false;
      if (j > 0 && !__all_sync(0xffffffffu, mbar_wait(&bar->o_free, (j - 1) & 1, p.status, 105))) return false;
      if (!arrived(n) || !arrived(n + 1)) return false;
      if (elect_one()) {
        const uint64_t v_desc[2] = {umma_desc_sw128(ring_base + (n % kFwdSlots) * kSlotBytes, kRunBytes, 1024),
                                    umma_desc_sw128(ring_base + ((n + 1) % kFwdSlots) * kSlotBytes, kRunBytes, 1024)};
        const uint32_t own = tmem + kColS + (j & 1) * 128;
#pragma unroll
        for (int part = 2; part >= 0; --part)
#pragma unroll
          for (int ks = 0; ks < kStep / 16; ++ks)
            umma_ts(tmem + kColO, own + (part == 2 ? kStep : part * 16) + (ks >> 1) * 32 + (ks & 1) * 8,
                    v_desc[ks >> 1] + (((ks & 1) * 2048) >> 4), kIdescO, part < 2 || ks > 0);
        tc_commit(&bar->empty[n % kFwdSlots]);
        tc_commit(&bar->empty[(n + 1) % kFwdSlots]);
        tc_commit(&bar->o_full);
      }
      __syncwarp();
      n += 2;
      return true;
    };
    if (ok) ok = issue_s(0);
    for (int j = 0; j < n_steps && ok; ++j) {
      if (j + 1 < n_steps) ok = issue_s(j + 1);
      if (ok) ok = issue_pv(j);
    }
  } else if (warp >= 4) {
    take_registers();
    const int g = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const int query = q_tile * kRows + row;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t o_addr = tmem + lane_base + kColO + g * 128;
    float m_true = -INFINITY, l = 0.0f;
    // The exponent's offset is a whole number, at least the row's maximum so far in log2 units: it enters
    // every exponent without a rounding, and a step's correction is a power of two.
    float offset = -INFINITY, correction = 0.0f;
    float acc[128];
#pragma unroll
    for (int i = 0; i < 128; ++i) acc[i] = 0.0f;
    bool ok = true;
    auto add_step = [&](int j) {   // acc = acc * correction + O(j)
      ok = ok && mbar_wait(&bar->o_full, j & 1, p.status, 107);
      if (!ok) return;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 4; ++c) add_columns(o_addr + c * 32, correction, acc + c * 32);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->o_free);
    };
    // (no early exit: the two warpgroups meet at a barrier in every step, whatever their waits say)
    for (int j = 0; j < n_steps; ++j) {
      const uint32_t s_addr = tmem + lane_base + kColS + (j & 1) * 128 + g * 32;
      ok = ok && mbar_wait(&bar->s_full[j & 1], (j >> 1) & 1, p.status, 106);
      uint32_t s[32];
      float local = -INFINITY;
      if (ok) {
        tc_fence_after();
        load_halves(s_addr, s_addr + kStep, s);
        if (j >= 2 * q_tile) {
          const int key0 = j * kStep + g * 32;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + i > query) s[i] = 0xff800000u;   // -inf above the diagonal
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          mx[(i >> 1) & 3] = max3(mx[(i >> 1) & 3], __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
        local = fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]);
      }
      const uint32_t own = exchange + (j & 1) * 2 * kRows * 4 + row * 4;
      sts_f32(own + g * kRows * 4, local);
      named_barrier_sync(1, 256);
      if (!ok) continue;
      m_true = max3(m_true, local, lds_f32(own + (g ^ 1) * kRows * 4));
      const float next = fmaxf(offset, ceilf(m_true * p.scale_log2));
      const float factor = fast_exp2(offset - next);
      offset = next;
      float sum[2] = {0.0f, 0.0f};
#pragma unroll
      for (int c = 0; c < 2; ++c) {   // 16 columns at a time: parts 0 and 1 over one half's columns, part 2 over the other's
        uint32_t part[3][8];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float p0 = fast_exp2(fmaf(__uint_as_float(s[c * 16 + i]), p.scale_log2, -offset));
          const float p1 = fast_exp2(fmaf(__uint_as_float(s[c * 16 + i + 1]), p.scale_log2, -offset));
          sum[0] += p0;
          sum[1] += p1;
          const Thirds t = split_pair(p0, p1);
          part[0][i / 2] = t.part[0]; part[1][i / 2] = t.part[1]; part[2][i / 2] = t.part[2];
        }
        tmem_st8(s_addr + c * 8, part[0]);
        tmem_st8(s_addr + 16 + c * 8, part[1]);
        tmem_st8(s_addr + kStep + c * 8, part[2]);
      }
      l = fmaf(l, factor, sum[0] + sum[1]);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->p_full[j & 1]);
      if (j > 0) add_step(j - 1);
      correction = factor;
    }
    add_step(n_steps - 1);
    // l of the whole row; the rows then leave through shared memory (Q and the first slots are free
    // by now), coalesced, with the gate applied on the way.  The gate of the eight channels that a thread
    // writes of each of sixteen rows waits in shared memory behind the staging tile, so that the store
    // loop below is a loop: unrolled, its 128 sigmoids are code that runs once and is fetched cold (13 us
    // per CTA), and with the loads inside, every row waits for its own.
    const uint32_t own = exchange + (n_steps & 1) * 2 * kRows * 4 + row * 4;
    sts_f32(own + g * kRows * 4, l);
    named_barrier_sync(1, 256);
    l += lds_f32(own + (g ^ 1) * kRows * 4);
    const int t256 = threadIdx.x - 128, c8 = t256 & 31;   // row t256 / 32 + 8 u, channels 8 c8 ..
    const uint32_t stage = smem_u32(smem), own_gate = stage + 2 * kTileBytes + t256 * 16;
    static_assert(kTileBytes + kFwdSlots * kSlotBytes >= 3 * kTileBytes, "staging tile and gate");
    if (ok) {
      // (a division: one rounding where a product with 1 / l has two; core is saved as fp32)
#pragma unroll
      for (int i = 0; i < 128; ++i) acc[i] /= l;
#pragma unroll
      for (int c = 0; c < 4; ++c) stage_32<1024>(stage, row, g * 32 + c * 8, acc + c * 32);
      if (p.gate) {
        uint4 gates[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const int r = min(q_tile * kRows + (t256 >> 5) + 8 * u, p.seq - 1);
          gates[u] = *reinterpret_cast<const uint4*>(p.gate + (static_cast<size_t>(batch) * p.seq + r) * p.gate_token +
                                                     head * p.gate_head + c8 * 8);
        }
#pragma unroll
        for (int u = 0; u < 16; ++u) sts_b32x4(own_gate + u * 4096, gates[u].x, gates[u].y, gates[u].z, gates[u].w);
      }
      if (g == 0 && query < p.seq && p.maxima) {
        const size_t stat = (static_cast<size_t>(batch) * p.heads + head) * p.seq + query;
        p.maxima[stat] = m_true * p.scale;
        p.normalizers[stat] = l * fast_exp2(fmaf(-m_true, p.scale_log2, offset));
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
            float factor = sigmoid(x);
            if (p.round_gate) {
              factor = bf16_round(factor);
              v[i] = bf16_round(v[i]);
            }
            v[i] *= factor;
          }
        }
        *reinterpret_cast<uint4*>(p.out + at) =
            make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
      }
    }
  } else {
    give_registers();   // (every warp of a warpgroup gives its registers back)
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

// dO as three bf16 parts, and the row statistics.  One warp per padded (head, row):
// head-major, so the statistics are written in runs; a row of dO is a whole kilobyte either way.
__global__ void __launch_bounds__(256)
attn_bwd_prep_wide(const __nv_bfloat16* __restrict__ out, const float* __restrict__ d_out,
                   const float* __restrict__ maxima, const float* __restrict__ normalizers,
                   float* deltas, __nv_bfloat16* __restrict__ parts, size_t part_stride, float2* __restrict__ stats, int seq, int seq_pad,
                   int heads, long long rows) {
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
  const Thirds t[4] = {split_pair(g0.x, g0.y), split_pair(g0.z, g0.w), split_pair(g1.x, g1.y), split_pair(g1.z, g1.w)};
#pragma unroll
  for (int i = 0; i < 3; ++i)
    *reinterpret_cast<uint4*>(parts + i * part_stride + base) = make_uint4(t[0].part[i], t[1].part[i], t[2].part[i], t[3].part[i]);
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
  uint64_t do_full, q_full, q_stored, last_full, last_stored, k_full[2], k_empty[2], v_full, v_empty;
  uint64_t s_full, s_read, dp_full, ds_ready, dq_full[2], dq_free[2];
  uint32_t tmem_base;
};
constexpr int kDqSmem = 1024 + 2 * kTileBytes + 3 * kStepBytes + sizeof(WideDqBarriers);

// Tensor work of a step (64 keys): S 1, dP 3 (the parts of dO), dQ 3 (the parts of dS) of
// [128 x 64 x 256].  Two blocks of 64 columns hold the halves of S, then those of dP, then the parts of
// dS: the row threads take S into registers and make P of it while dP runs, and S(j + 1) follows the last
// quarter of dQ(j) and runs while that quarter is added.
__global__ void __launch_bounds__(kWideThreads, 1)
attn_bwd_dq_wide(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k64,
                 const __grid_constant__ CUtensorMap map_v64, const __grid_constant__ CUtensorMap map_do0,
                 const __grid_constant__ CUtensorMap map_do1, const __grid_constant__ CUtensorMap map_do2,
                 WideBwdParams p) {
  constexpr uint32_t kColQ = 0, kColLast = 128, kColDQ = 256, kColA = 384, kColB = 448;
  constexpr uint32_t kIdescS = umma_idesc_bf16(kRows, kStep, false);
  constexpr uint32_t kIdescDQ = umma_idesc_bf16(kRows, 64, true);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* do_smem = smem;                      // the first two parts
  uint8_t* k_ring = do_smem + 2 * kTileBytes;   // two stages; Q and dO's third part pass through them into TMEM
  uint8_t* v_smem = k_ring + 2 * kStepBytes;    // one step
  WideDqBarriers* bar = reinterpret_cast<WideDqBarriers*>(v_smem + kStepBytes);

  const int warp = uniform_warp_index(), lane = threadIdx.x % 32;
  const int q_tile = gridDim.y - 1 - blockIdx.y;
  const int head = blockIdx.x % p.heads, batch = blockIdx.x / p.heads;
  const int kv_head = head / p.group;
  const int n_steps = min(2 * q_tile + 2, (p.seq + kStep - 1) / kStep);

  if (threadIdx.x == 0) {
    mbar_init(&bar->do_full, 1);
    mbar_init(&bar->q_full, 1);
    mbar_init(&bar->q_stored, 8);
    mbar_init(&bar->last_full, 1);
    mbar_init(&bar->last_stored, 8);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar->k_full[s], 1);
      mbar_init(&bar->k_empty[s], 1);
      mbar_init(&bar->dq_full[s], 1);
      mbar_init(&bar->dq_free[s], 4);   // the warps of one warpgroup
    }
    mbar_init(&bar->v_full, 1);
    mbar_init(&bar->v_empty, 1);
    mbar_init(&bar->s_full, 1);
    mbar_init(&bar->s_read, 8);
    mbar_init(&bar->dp_full, 1);
    mbar_init(&bar->ds_ready, 8);
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
    give_registers();
    if (lane == 0) {
      tma_prefetch_desc(&map_k64);
      tma_prefetch_desc(&map_v64);
      mbar_expect_tx(&bar->q_full, kTileBytes);
      for (int s = 0; s < 4; ++s)
        tma_load_3d(k_ring + s * kSlabBytes, &map_q, p.q_col0 + head * kD + s * 64, q_tile * kRows, batch, &bar->q_full);
      mbar_expect_tx(&bar->do_full, 2 * kTileBytes);
      for (int s = 0; s < 4; ++s) {
        tma_load_3d(do_smem + s * kSlabBytes, &map_do0, head * kD + s * 64, q_tile * kRows, batch, &bar->do_full);
        tma_load_3d(do_smem + kTileBytes + s * kSlabBytes, &map_do1, head * kD + s * 64, q_tile * kRows, batch,
                    &bar->do_full);
      }
      int k_used = 0, v_used = 0;
      bool last_used = false;
      bool ok = mbar_wait(&bar->q_stored, 0, p.status, 110);
      if (ok) {
        mbar_expect_tx(&bar->last_full, kTileBytes);
        for (int s = 0; s < 4; ++s)
          tma_load_3d(k_ring + s * kSlabBytes, &map_do2, head * kD + s * 64, q_tile * kRows, batch, &bar->last_full);
        last_used = true;
      }
      for (int j = 0; j < n_steps && ok; ++j) {
        if (j > 0) ok = mbar_wait(&bar->v_empty, (j - 1) & 1, p.status, 110);
        if (!ok) break;
        mbar_expect_tx(&bar->v_full, kStepBytes);
        for (int s = 0; s < 4; ++s)
          tma_load_3d(v_smem + s * kStepSlab, &map_v64, p.v_col0 + kv_head * kD + s * 64, j * kStep, batch, &bar->v_full);
        ++v_used;
        if (j == 0) ok = mbar_wait(&bar->last_stored, 0, p.status, 111);
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
      if (last_used) mbar_wait(&bar->last_full, 0, p.status, 113);
      if (v_used > 0) mbar_wait(&bar->v_full, (v_used - 1) & 1, p.status, 114);
      for (int j = max(0, k_used - 2); j < k_used; ++j) mbar_wait(&bar->k_full[j & 1], (j >> 1) & 1, p.status, 114);
    }
  } else if (warp == 1) {
    give_registers();
    const uint64_t do_desc = umma_desc_sw128(smem_u32(do_smem), 16, 1024);
    const uint64_t v_desc = umma_desc_sw128(smem_u32(v_smem), 16, 1024);
    const uint32_t k_base = smem_u32(k_ring);
    bool ok = __all_sync(0xffffffffu, mbar_wait(&bar->do_full, 0, p.status, 117) &&
                                          mbar_wait(&bar->last_stored, 0, p.status, 118));
    for (int j = 0; j < n_steps && ok; ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bar->k_full[j & 1], (j >> 1) & 1, p.status, 116));
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {   // S(j) = Q K_j^T
        const uint64_t k_desc = umma_desc_sw128(k_base + (j & 1) * kStepBytes, 16, 1024);
#pragma unroll
        for (int ks = 0; ks < kD / 16; ++ks)
          umma_ts(tmem + (ks < 8 ? kColA : kColB), tmem + kColQ + ks * 8,
                  k_desc + (((ks / 4) * kStepSlab + (ks % 4) * 32) >> 4), kIdescS, ks % 8 > 0);
        tc_commit(&bar->s_full);
      }
      __syncwarp();
      ok = __all_sync(0xffffffffu, mbar_wait(&bar->v_full, j & 1, p.status, 115) &&
                                       mbar_wait(&bar->s_read, j & 1, p.status, 115));
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {   // dP(j) = dO V_j^T, the parts of dO from the last to the first
#pragma unroll
        for (int part = 2; part >= 0; --part)
#pragma unroll
          for (int ks = 0; ks < kD / 16; ++ks) {
            const uint32_t to = tmem + (ks < 8 ? kColA : kColB);
            const uint64_t v = v_desc + (((ks / 4) * kStepSlab + (ks % 4) * 32) >> 4);
            if (part == 2) umma_ts(to, tmem + kColLast + ks * 8, v, kIdescS, ks % 8 > 0);
            else umma_ss(to, do_desc + ((part * kTileBytes + (ks / 4) * kSlabBytes + (ks % 4) * 32) >> 4), v, kIdescS, true);
          }
        tc_commit(&bar->v_empty);
        tc_commit(&bar->dp_full);
      }
      __syncwarp();
      ok = __all_sync(0xffffffffu, mbar_wait(&bar->ds_ready, j & 1, p.status, 120));
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int slab = 0; slab < 4; ++slab) {   // 64 channels of dQ(j) = dS K_j
        const int block = slab & 1, use = 2 * j + (slab >> 1);
        if (use > 0) ok = ok && __all_sync(0xffffffffu, mbar_wait(&bar->dq_free[block], (use - 1) & 1, p.status, 119));
        if (ok && elect_one()) {
          tc_fence_after();
          const uint64_t k_mn = umma_desc_sw128(k_base + (j & 1) * kStepBytes + slab * kStepSlab, kStepSlab, 1024);
#pragma unroll
          for (int part = 2; part >= 0; --part)
#pragma unroll
            for (int ks = 0; ks < kStep / 16; ++ks)
              umma_ts(tmem + kColDQ + block * 64,
                      tmem + (part == 2 ? kColB : kColA + part * 16) + (ks >> 1) * 32 + (ks & 1) * 8,
                      k_mn + ks * (2048 >> 4), kIdescDQ, part < 2 || ks > 0);
          tc_commit(&bar->dq_full[block]);
          if (slab == 3) tc_commit(&bar->k_empty[j & 1]);
        }
        __syncwarp();
      }
    }
  } else if (warp >= 4) {
    take_registers();
    const int g = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const int query = q_tile * kRows + row;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    // this thread's half of its query row, then of its row of dO's third part, into TMEM
    auto store_half_row = [&](uint32_t column) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        uint32_t w[32];
        load_swizzled_row(smem_u32(k_ring) + (2 * g + s) * kSlabBytes, row, w);
        tmem_st32(tmem + lane_base + column + (2 * g + s) * 32, w);
      }
      tmem_wait_st();
      fence_proxy_async();
      tc_fence_before();
    };
    bool ok = mbar_wait(&bar->q_full, 0, p.status, 121);
    if (ok) store_half_row(kColQ);
    __syncwarp();
    if (ok && lane == 0) mbar_arrive(&bar->q_stored);
    ok = ok && mbar_wait(&bar->last_full, 0, p.status, 121);
    if (ok) store_half_row(kColLast);
    __syncwarp();
    if (ok && lane == 0) mbar_arrive(&bar->last_stored);
    const float2 st = p.stats[(static_cast<size_t>(batch) * p.heads + head) * p.seq_pad + min(query, p.seq_pad - 1)];
    const float shift = st.x, delta = st.y;
    const uint32_t a_addr = tmem + lane_base + kColA + g * 32, b_addr = tmem + lane_base + kColB + g * 32;
    float acc[128];   // channels of slabs g and g + 2
#pragma unroll
    for (int i = 0; i < 128; ++i) acc[i] = 0.0f;
    for (int j = 0; j < n_steps && ok; ++j) {
      ok = mbar_wait(&bar->s_full, j & 1, p.status, 122);
      if (!ok) break;
      tc_fence_after();
      uint32_t prob[32];
      load_halves(a_addr, b_addr, prob);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->s_read);
      const int key0 = j * kStep + g * 32;
      const bool masked = j >= 2 * q_tile;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        float x = fast_exp2(fmaf(__uint_as_float(prob[i]), p.scale_log2, shift));
        if (masked && key0 + i > query) x = 0.0f;
        prob[i] = __float_as_uint(x);
      }
      ok = mbar_wait(&bar->dp_full, j & 1, p.status, 123);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {   // 16 columns at a time into registers, P (dP - delta) in place of P
        uint32_t first[16], second[16];
        tmem_ld16(a_addr + c * 16, first);
        tmem_ld16(b_addr + c * 16, second);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          prob[c * 16 + i] = __float_as_uint(__uint_as_float(prob[c * 16 + i]) *
                                             (__uint_as_float(first[i]) + __uint_as_float(second[i]) - delta));
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {   // parts 0 and 1 over one half's columns, part 2 over the other's
        uint32_t part[3][8];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const Thirds t = split_pair(__uint_as_float(prob[c * 16 + i]), __uint_as_float(prob[c * 16 + i + 1]));
          part[0][i / 2] = t.part[0]; part[1][i / 2] = t.part[1]; part[2][i / 2] = t.part[2];
        }
        tmem_st8(a_addr + c * 8, part[0]);
        tmem_st8(a_addr + 16 + c * 8, part[1]);
        tmem_st8(b_addr + c * 8, part[2]);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->ds_ready);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ok = ok && mbar_wait(&bar->dq_full[g], h, p.status, 124);   // two uses a step: the parity is h
        if (ok) {
          tc_fence_after();
          add_columns(tmem + lane_base + kColDQ + g * 64, 1.0f, acc + h * 64);
          add_columns(tmem + lane_base + kColDQ + g * 64 + 32, 1.0f, acc + h * 64 + 32);
          tc_fence_before();
        }
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(&bar->dq_free[g]);
      }
    }
    // dQ leaves through the dO tiles, scaled (the last product that read them is long complete)
    const uint32_t stage = smem_u32(smem);
    named_barrier_sync(1, 256);
    if (ok) {
#pragma unroll
      for (int i = 0; i < 128; ++i) acc[i] *= p.scale;
#pragma unroll
      for (int c = 0; c < 4; ++c) stage_32<1024>(stage, row, (g + (c >> 1) * 2) * 16 + (c & 1) * 8, acc + c * 32);
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
  } else {
    give_registers();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

constexpr int kDkvSlots = 5;                  // Q of even and odd steps, the three parts of dO
struct WideDkvBarriers {
  uint64_t v_full, k_full, rows_ready, full[kDkvSlots], empty[kDkvSlots], s_full, p_stored, dp_full, ds_stored, acc_full[2], acc_free[2];
  uint32_t tmem_base;
};
constexpr int kDkvStats = 2 * kStep * 8;      // (shift, delta) of two steps
constexpr int kDkvSmem = 1024 + kTileBytes + kDkvSlots * kStepBytes + kDkvStats + sizeof(WideDkvBarriers);

// grid (2 channel halves x (batch x query heads / heads_per_cta), key tiles).  Tensor work of a step (64
// queries): S 1, dP 3 of [128 x 64 x 256]; dV 6 (the products of parts above 2^-24), dK 3 of
// [128 x 128 x 64], in the order dP(i), dV(i), S(i + 1), dK(i): the row threads make P(i) while dP(i) runs and
// dS(i) while dV(i) and S(i + 1) do.  dV and dK are made in the same columns, one added up by warpgroup 0 and
// the other by warpgroup 1.  Q lies in slot i & 1, part k of dO in slot 2 + k, and a part's
// slot is free as soon as its last product with P has run; V passes through the slots of parts 1 and 2 on
// its way into TMEM.
__global__ void __launch_bounds__(kWideThreads, 1)
attn_bwd_dkv_wide(const __grid_constant__ CUtensorMap map_q64, const __grid_constant__ CUtensorMap map_k,
                  const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do0,
                  const __grid_constant__ CUtensorMap map_do1, const __grid_constant__ CUtensorMap map_do2,
                  WideBwdParams p) {
  constexpr uint32_t kColSA = 0, kColSB = 64, kColDPA = 128, kColDPB = 192, kColAcc = 256, kColV = 384;
  constexpr uint32_t kIdescS = umma_idesc_bf16(kRows, kStep, false);
  constexpr uint32_t kIdescAcc = umma_idesc_bf16(kRows, 128, true);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* k_smem = smem;
  uint8_t* slots = k_smem + kTileBytes;
  uint8_t* stat_ring = slots + kDkvSlots * kStepBytes;
  WideDkvBarriers* bar = reinterpret_cast<WideDkvBarriers*>(stat_ring + kDkvStats);

  const int warp = uniform_warp_index(), lane = threadIdx.x % 32;
  const int half = blockIdx.x & 1, k_tile = blockIdx.y;   // the first key tile sees the most queries
  const int head_sets = p.heads / p.heads_per_cta;
  const int set = (blockIdx.x >> 1) % head_sets, batch = (blockIdx.x >> 1) / head_sets;
  const int head0 = set * p.heads_per_cta, kv_head = head0 / p.group;
  const int part_index = (head0 % p.group) / p.heads_per_cta;
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
    mbar_init(&bar->p_stored, 8);
    mbar_init(&bar->dp_full, 1);
    mbar_init(&bar->ds_stored, 8);
    for (int s = 0; s < 2; ++s) {   // dV, dK: one warpgroup each
      mbar_init(&bar->acc_full[s], 1);
      mbar_init(&bar->acc_free[s], 4);
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
  // The dQ kernel lets this grid start as soon as every one of its CTAs has seen the prep kernel
  // complete; nothing it writes is read here, so its last CTAs and this grid's first share the chip.
  pdl_launch_dependents();

  if (warp == 0) {
    give_registers();
    if (lane == 0) {
      mbar_expect_tx(&bar->v_full, kTileBytes);
      for (int s = 0; s < 4; ++s)
        tma_load_3d(slots + 3 * kStepBytes + s * kSlabBytes, &map_v, p.v_col0 + kv_head * kD + s * 64, k_tile * kRows,
                    batch, &bar->v_full);
      mbar_expect_tx(&bar->k_full, kTileBytes);
      for (int s = 0; s < 4; ++s)
        tma_load_3d(k_smem + s * kSlabBytes, &map_k, p.k_col0 + kv_head * kD + s * 64, k_tile * kRows, batch, &bar->k_full);
      bool ok = true;
      int uses[kDkvSlots] = {0, 0, 0, 0, 0};
      auto load = [&](int st, const CUtensorMap* map, int i, int col) {   // the next use of a slot, by step i
        const int head = head0 + i / per_head, q0 = (2 * k_tile + i % per_head) * kStep;
        if (uses[st] > 0) ok = ok && mbar_wait(&bar->empty[st], (uses[st] - 1) & 1, p.status, 131);
        if (!ok) return;
        mbar_expect_tx(&bar->full[st], kStepBytes + (st < 2 ? kStep * 8 : 0));
        for (int s = 0; s < 4; ++s)
          tma_load_3d(slots + st * kStepBytes + s * kStepSlab, map, col + head * kD + s * 64, q0, batch, &bar->full[st]);
        if (st < 2)   // the statistics come with Q
          bulk_load(stat_ring + st * kStep * 8, p.stats + (static_cast<size_t>(batch) * p.heads + head) * p.seq_pad + q0,
                    kStep * 8, &bar->full[st]);
        ++uses[st];
      };
      load(0, &map_q64, 0, p.q_col0);
      load(2, &map_do0, 0, 0);
      ok = mbar_wait(&bar->rows_ready, 0, p.status, 130);
      for (int i = 0; i < n_steps && ok; ++i) {
        load(4, &map_do2, i, 0);
        load(3, &map_do1, i, 0);
        if (i > 0) load(2, &map_do0, i, 0);
        if (i + 1 < n_steps) load((i + 1) & 1, &map_q64, i + 1, p.q_col0);
      }
      mbar_wait(&bar->k_full, 0, p.status, 132);   // no copy may be in flight when the CTA leaves
      mbar_wait(&bar->v_full, 0, p.status, 132);
      for (int s = 0; s < kDkvSlots; ++s)
        if (uses[s] > 0) mbar_wait(&bar->full[s], (uses[s] - 1) & 1, p.status, 133);
    }
  } else if (warp == 1) {
    give_registers();
    const uint32_t slot_base = smem_u32(slots);
    const uint64_t k_desc = umma_desc_sw128(smem_u32(k_smem), 16, 1024);
    auto arrived = [&](int st, int use) -> bool {
      const bool good = __all_sync(0xffffffffu, mbar_wait(&bar->full[st], use & 1, p.status, 134));
      tc_fence_after();
      return good;
    };
    auto issue_s = [&](int i) -> bool {   // S(i)^T = K Q^T
      if (!arrived(i & 1, i >> 1)) return false;
      if (elect_one()) {
        const uint64_t q_desc = umma_desc_sw128(slot_base + (i & 1) * kStepBytes, 16, 1024);
#pragma unroll
        for (int ks = 0; ks < kD / 16; ++ks)
          umma_ss(tmem + (ks < 8 ? kColSA : kColSB), k_desc + (((ks / 4) * kSlabBytes + (ks % 4) * 32) >> 4),
                  q_desc + (((ks / 4) * kStepSlab + (ks % 4) * 32) >> 4), kIdescS, ks % 8 > 0);
        tc_commit(&bar->s_full);
      }
      __syncwarp();
      return true;
    };
    bool ok = __all_sync(0xffffffffu, mbar_wait(&bar->k_full, 0, p.status, 135) &&
                                          mbar_wait(&bar->rows_ready, 0, p.status, 136));
    if (ok) ok = issue_s(0);
    const uint32_t columns = half * 2 * kStepSlab;   // this CTA's 128 channels, MN-major: 16 queries per instruction
    for (int i = 0; i < n_steps && ok; ++i) {
#pragma unroll
      for (int part = 2; part >= 0; --part) {   // dP(i)^T = V dO^T, the parts of dO from the last to the first
        ok = ok && arrived(2 + part, i);
        if (ok && elect_one()) {
          const uint64_t do_desc = umma_desc_sw128(slot_base + (2 + part) * kStepBytes, 16, 1024);
#pragma unroll
          for (int ks = 0; ks < kD / 16; ++ks)
            umma_ts(tmem + (ks < 8 ? kColDPA : kColDPB), tmem + kColV + ks * 8,
                    do_desc + (((ks / 4) * kStepSlab + (ks % 4) * 32) >> 4), kIdescS, part < 2 || ks % 8 > 0);
          if (part == 0) tc_commit(&bar->dp_full);
        }
        __syncwarp();
      }
      if (!ok) break;
      ok = __all_sync(0xffffffffu, mbar_wait(&bar->p_stored, i & 1, p.status, 137));
      if (ok && i > 0) ok = __all_sync(0xffffffffu, mbar_wait(&bar->acc_free[1], (i - 1) & 1, p.status, 137));
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {   // dV(i) = P dO, from the smallest products to the largest
        uint64_t do_mn[3];
#pragma unroll
        for (int part = 0; part < 3; ++part)
          do_mn[part] = umma_desc_sw128(slot_base + (2 + part) * kStepBytes + columns, kStepSlab, 1024);
        constexpr int kOrder[6][2] = {{0, 2}, {2, 0}, {1, 1}, {0, 1}, {1, 0}, {0, 0}};   // (part of P, part of dO)
#pragma unroll
        for (int k = 0; k < 6; ++k) {
#pragma unroll
          for (int ks = 0; ks < kStep / 16; ++ks)
            umma_ts(tmem + kColAcc,
                    tmem + (kOrder[k][0] == 2 ? kColSB : kColSA + kOrder[k][0] * 16) + (ks >> 1) * 32 + (ks & 1) * 8,
                    do_mn[kOrder[k][1]] + ks * (2048 >> 4), kIdescAcc, k > 0 || ks > 0);
          if (k == 0) tc_commit(&bar->empty[4]);
          if (k == 3) tc_commit(&bar->empty[3]);
          if (k == 5) tc_commit(&bar->empty[2]);
        }
        tc_commit(&bar->acc_full[0]);
      }
      __syncwarp();
      if (i + 1 < n_steps) ok = issue_s(i + 1);   // over P(i), behind its products
      if (ok)
        ok = __all_sync(0xffffffffu, mbar_wait(&bar->acc_free[0], i & 1, p.status, 137) &&
                                         mbar_wait(&bar->ds_stored, i & 1, p.status, 137));
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {   // dK(i) = dS Q
        const uint64_t q_mn = umma_desc_sw128(slot_base + (i & 1) * kStepBytes + columns, kStepSlab, 1024);
#pragma unroll
        for (int part = 2; part >= 0; --part)
#pragma unroll
          for (int ks = 0; ks < kStep / 16; ++ks)
            umma_ts(tmem + kColAcc, tmem + (part == 2 ? kColDPB : kColDPA + part * 16) + (ks >> 1) * 32 + (ks & 1) * 8,
                    q_mn + ks * (2048 >> 4), kIdescAcc, part < 2 || ks > 0);
        tc_commit(&bar->acc_full[1]);
        tc_commit(&bar->empty[i & 1]);
      }
      __syncwarp();
    }
  } else if (warp >= 4) {
    take_registers();
    const int g = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const int key = k_tile * kRows + row;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    bool ok = mbar_wait(&bar->v_full, 0, p.status, 138);
    if (ok) {   // this thread's half of its value row into TMEM
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        uint32_t w[32];
        load_swizzled_row(smem_u32(slots) + 3 * kStepBytes + (2 * g + s) * kSlabBytes, row, w);
        tmem_st32(tmem + lane_base + kColV + (2 * g + s) * 32, w);
      }
      tmem_wait_st();
      fence_proxy_async();
      tc_fence_before();
    }
    __syncwarp();
    if (ok && lane == 0) mbar_arrive(&bar->rows_ready);
    const uint32_t own = tmem + lane_base + g * 32;
    float acc[128];   // this CTA's channels of dV (warpgroup 0) or dK (warpgroup 1)
#pragma unroll
    for (int i = 0; i < 128; ++i) acc[i] = 0.0f;
    for (int i = 0; i < n_steps && ok; ++i) {
      ok = mbar_wait(&bar->s_full, i & 1, p.status, 139) &&
           mbar_wait(&bar->full[i & 1], (i >> 1) & 1, p.status, 140);   // the statistics landed
      if (!ok) break;
      tc_fence_after();
      uint32_t prob[32];
      load_halves(own + kColSA, own + kColSB, prob);
      const int local = i % per_head, query0 = (2 * k_tile + local) * kStep + g * 32;
      const bool masked = local < 2;
      const uint32_t stats = smem_u32(stat_ring) + ((i & 1) * kStep + g * 32) * 8;
#pragma unroll
      for (int c = 0; c < 2; ++c) {   // 16 columns at a time; parts 0 and 1 over one half's columns, part 2 over the other's
        uint32_t part[3][8];
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
          const int at = c * 16 + k;
          const float4 st = lds_f32x4(stats + at * 8);   // (shift, delta) of two queries, the same for the whole warp
          float p0 = fast_exp2(fmaf(__uint_as_float(prob[at]), p.scale_log2, st.x));
          float p1 = fast_exp2(fmaf(__uint_as_float(prob[at + 1]), p.scale_log2, st.z));
          if (masked) {
            if (query0 + at < key) p0 = 0.0f;
            if (query0 + at + 1 < key) p1 = 0.0f;
          }
          const Thirds t = split_pair(p0, p1);
          part[0][k / 2] = t.part[0]; part[1][k / 2] = t.part[1]; part[2][k / 2] = t.part[2];
          prob[at] = __float_as_uint(p0);
          prob[at + 1] = __float_as_uint(p1);
        }
        tmem_st8(own + kColSA + c * 8, part[0]);
        tmem_st8(own + kColSA + 16 + c * 8, part[1]);
        tmem_st8(own + kColSB + c * 8, part[2]);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->p_stored);
      ok = mbar_wait(&bar->dp_full, i & 1, p.status, 139);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t first[16], second[16];
        tmem_ld16(own + kColDPA + c * 16, first);
        tmem_ld16(own + kColDPB + c * 16, second);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
          const int at = c * 16 + k;
          const float4 st = lds_f32x4(stats + at * 8);
          prob[at] = __float_as_uint(__uint_as_float(prob[at]) *
                                     (__uint_as_float(first[k]) + __uint_as_float(second[k]) - st.y));
          prob[at + 1] = __float_as_uint(__uint_as_float(prob[at + 1]) *
                                         (__uint_as_float(first[k + 1]) + __uint_as_float(second[k + 1]) - st.w));
        }
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t part[3][8];
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
          const Thirds t = split_pair(__uint_as_float(prob[c * 16 + k]), __uint_as_float(prob[c * 16 + k + 1]));
          part[0][k / 2] = t.part[0]; part[1][k / 2] = t.part[1]; part[2][k / 2] = t.part[2];
        }
        tmem_st8(own + kColDPA + c * 8, part[0]);
        tmem_st8(own + kColDPA + 16 + c * 8, part[1]);
        tmem_st8(own + kColDPB + c * 8, part[2]);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->ds_stored);
      ok = mbar_wait(&bar->acc_full[g], i & 1, p.status, 141);
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 4; ++c) add_columns(tmem + lane_base + kColAcc + c * 32, 1.0f, acc + c * 32);
        tc_fence_before();
      }
      __syncwarp();
      if (ok && lane == 0) mbar_arrive(&bar->acc_free[g]);
    }
    // dV and dK leave through the slots: [128 rows x 128] fp32 each
    const uint32_t stage = smem_u32(slots) + g * kRows * 512;
    named_barrier_sync(1, 256);   // (dK's products read them: warpgroup 1 has seen the last complete)
    if (ok) {
      const float factor = g == 0 ? 1.0f : p.scale;
#pragma unroll
      for (int i = 0; i < 128; ++i) acc[i] *= factor;
#pragma unroll
      for (int c = 0; c < 4; ++c) stage_32<512>(stage, row, c * 8, acc + c * 32);
    }
    named_barrier_sync(1, 256);
    if (ok) {
      float* dst = (g == 0 ? p.dv : p.dk) + part_index * p.part_stride + kv_head * kD + half * 128;
#pragma unroll 4
      for (int e = (threadIdx.x - 128) & 127; e < kRows * 32; e += 128) {
        const int r = e >> 5, c = e & 31;
        if (k_tile * kRows + r >= p.seq) continue;
        const size_t token = static_cast<size_t>(batch) * p.seq + k_tile * kRows + r;
        *reinterpret_cast<float4*>(dst + token * p.dkv_token + c * 4) = lds_f32x4(staged_chunk<512>(stage, r, c));
      }
    }
  } else {
    give_registers();
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
      !make_token_map(&map_k, a.k, a.kv_cols, a.seq, a.batch, a.kv_token, kStep) ||
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

// The upstream gradient's three parts, the statistics, and dK / dV partial sums for as many parts as a
// group can have query heads.
size_t attn_bwd_wide_workspace_bytes(int batch, int seq, int heads) {
  const size_t rows = static_cast<size_t>(batch) * seq * heads;
  return rows * kD * 6 + static_cast<size_t>(batch) * heads * padded_rows(seq) * sizeof(float2) + 256 + 2 * rows * kD * 4;
}

cudaError_t attn_bwd_wide_tc(cudaStream_t stream, const GqaBwdTcArgs& a) {
  const int seq_pad = padded_rows(a.seq), tiles = (a.seq + kRows - 1) / kRows, group = a.q_heads / a.kv_heads;
  const size_t rows = static_cast<size_t>(a.batch) * a.seq * a.q_heads;
  auto* upstream = static_cast<__nv_bfloat16*>(a.workspace);
  float2* stats = reinterpret_cast<float2*>(upstream + 3 * rows * kD);
  const size_t stat_rows = static_cast<size_t>(a.batch) * a.q_heads * seq_pad;
  float* parts = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(stats + stat_rows) + 255) & ~static_cast<uintptr_t>(255));
  attn_bwd_prep_wide<<<static_cast<unsigned>((stat_rows + 7) / 8), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(a.out), a.d_out, a.maxima, a.normalizers, a.deltas, upstream, rows * kD, stats,
      a.seq, seq_pad, a.q_heads, static_cast<long long>(stat_rows));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int E = a.q_heads * kD;
  CUtensorMap q128, q64, k128, k64, v128, v64, do128[3], do64[3];
  if (!make_token_map(&q128, a.q, a.q_cols, a.seq, a.batch, a.q_token, kRows) ||
      !make_token_map(&q64, a.q, a.q_cols, a.seq, a.batch, a.q_token, kStep) ||
      !make_token_map(&k128, a.k, a.kv_cols, a.seq, a.batch, a.kv_token, kRows) ||
      !make_token_map(&k64, a.k, a.kv_cols, a.seq, a.batch, a.kv_token, kStep) ||
      !make_token_map(&v128, a.v, a.kv_cols, a.seq, a.batch, a.kv_token, kRows) ||
      !make_token_map(&v64, a.v, a.kv_cols, a.seq, a.batch, a.kv_token, kStep))
    return cudaErrorInvalidValue;
  for (int part = 0; part < 3; ++part) {
    const __nv_bfloat16* from = upstream + part * rows * kD;
    if (!make_token_map(&do128[part], from, E, a.seq, a.batch, E, kRows) ||
        !make_token_map(&do64[part], from, E, a.seq, a.batch, E, kStep))
      return cudaErrorInvalidValue;
  }
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
                     do128[0], do128[1], do128[2], p);
  if (e != cudaSuccess) return e;
  e = launch_chained(attn_bwd_dkv_wide, dim3(2 * a.batch * (a.q_heads / p.heads_per_cta), tiles), kWideThreads, kDkvSmem,
                     stream, q64, k128, v128, do64[0], do64[1], do64[2], p);
  if (e != cudaSuccess || n_parts == 1) return e;
  return launch_chained(attn_bwd_sum_wide, dim3(static_cast<unsigned>((part_floats / 4 + 255) / 256), 2), 256, 0, stream,
                        static_cast<const float*>(p.dk), static_cast<const float*>(p.dv), n_parts, part_floats, width,
                        static_cast<long long>(part_floats), a.dk, a.dv, a.dkv_token);
}

}  // namespace pluto
