// Grouped-query attention decode: one new query token per sequence against a KV cache.
//
// Stands in for FullAttentionKernel and the cached AttentionProbabilitiesKernel of the reference
// (src/llm/layers/util/cached_attention_ops.cc:83-126, :131-178), which run one program per query
// head (24-40 CTAs), re-read each KV head once per query head and keep the cache in fp32.  Here:
//   * the cache is read exactly once: all query heads of a KV head are the rows of one MMA tile;
//   * the sequence is split across CTAs (split-KV); every CTA produces a partial (max, sum,
//     accumulator), the token groups of a CTA merge through shared memory.  Small problems are cut
//     into at most sixteen parts per sequence that form a cluster and merge through distributed
//     shared memory (one launch); large ones into fixed chunks that a second kernel merges.  The
//     order is fixed either way (deterministic, no atomics);
//   * K/V tiles travel global -> shared as tiled TMA loads (no multicast) over a 4-D map of the
//     page pool (column, kv head, token in page, page): one elected thread issues a handful of
//     box copies per 64-token stage into a 3-stage ring guarded by mbarriers, 128-byte swizzled
//     so ldmatrix is bank-conflict free.  (Per-row bulk copies were tried first: at 256 bytes
//     per instruction the copy engine's per-instruction cost capped the kernel near 2 TB/s.)
//   * the arithmetic is bf16 mma.sync (m16n8k16) with fp32 accumulation -- the kernel is bound by
//     HBM bandwidth, the tensor path only has to stay out of the way.
// The cache is a page pool: token t of sequence b lives in page block_table[b][t / page_size]
// (or page b when there is no table: one contiguous region per sequence).
//
// A plain fp32 kernel covers every other case (fp32 cache, head widths other than 64/128/256,
// unrounded operands) with the same split/merge structure.
#include "common.cuh"
#include "engine.h"

namespace pluto {
namespace {

constexpr int kDecodeStages = 3;
constexpr int kMaxClusterParts = 16;
// Tokens per pipeline stage: 32 KB of K and V at head widths 128 and 256 (16 KB at 64), so that two
// CTAs share an SM and one's set-up, first loads and output run under the other's stream (one CTA per
// SM with 64-token stages at head width 256 took 238 us where this takes 142, at 60 sequences of up
// to 4000 tokens, 4 KV heads).
template <int D>
constexpr int kTile = D == 256 ? 32 : 64;
template <int D>
constexpr int kTokenWarps = kTile<D> / 16;   // 16 tokens of every tile each

// Sequence length as the kernels use it: the device value clamped into what the host sized the
// grid and the workspace for, [0, decode_chunk_capacity(splits, split_tokens)].  A value outside is a caller error; it
// is reported through the status word and the launch stays inside its buffers.
__device__ __forceinline__ int bounded_length(const DecodeArgs& a, int b, uint32_t site) {
  const int length = a.seq_lens ? a.seq_lens[b] : a.one_length;
  const long long limit = decode_chunk_capacity(a.splits, a.split_tokens);
  if (length < 0 || length > limit) {
    report_status(a.status, site, kBadLength);
    return length < 0 ? 0 : static_cast<int>(limit);
  }
  return length;
}

__device__ __forceinline__ const char* kv_row(const DecodeArgs& a, bool value, int b, int t,
                                              int kv_head, size_t element) {
  const void* base = value ? a.v_base : a.k_base;
  if (a.k_bases != nullptr) {   // separately allocated sequences
    const void* own = (value ? a.v_bases : a.k_bases)[b];
    return static_cast<const char*>(own) +
           (static_cast<size_t>(t) * a.token_stride + static_cast<size_t>(kv_head) * a.head_dim) * element;
  }
  int page = a.block_table ? a.block_table[static_cast<size_t>(b) * a.max_blocks + t / a.page_size]
                           : b;
  if (a.block_table && a.num_pages > 0 && (page < 0 || page >= a.num_pages)) {
    report_status(a.status, 35, kBadPage);   // the tiled-TMA path reads zeros there instead
    page = 0;
  }
  const size_t offset = static_cast<size_t>(page) * a.page_stride +
                        static_cast<size_t>(t % a.page_size) * a.token_stride +
                        static_cast<size_t>(kv_head) * a.head_dim;
  return static_cast<const char*>(base) + offset * element;
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  // (not volatile: the order of independent products is the compiler's to choose)
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct DecodeBarriers {
  uint64_t full[kDecodeStages];
  uint64_t empty[kDecodeStages];
};

// Head width 256: two warps share 16 tokens, each accumulating half of the channels (one warp's
// accumulators and query fragments would take 192 registers).
template <int D>
constexpr int kChannelParts = D == 256 ? 2 : 1;
constexpr int kDecodeThreads = (4 + 1) * 32;   // four consumer warps at every width, one producer
template <int D>
constexpr int kDecodeStageBytes = 2 * kTile<D> * D * 2;

// The reference's output stage (cached_attention_ops.cc:120-125): R(R(acc / l) * R(sigmoid(gate))).
__device__ __forceinline__ void store_output(const DecodeArgs& a, int b, int head, int d, float value) {
  if (a.round) value = bf16_round(value);
  if (a.gate) {
    const size_t g = static_cast<size_t>(b) * a.gate_token + static_cast<size_t>(head) * a.gate_head + d;
    const float x = a.gate_is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(a.gate)[g])
                                   : static_cast<const float*>(a.gate)[g];
    float factor = sigmoid(x);
    if (a.round) factor = bf16_round(factor);
    value *= factor;
    if (a.round) value = bf16_round(value);
  }
  const size_t idx = (static_cast<size_t>(b) * a.q_heads + head) * a.head_dim + d;
  if (a.out_is_bf16) static_cast<__nv_bfloat16*>(a.out)[idx] = __float2bfloat16_rn(value);
  else static_cast<float*>(a.out)[idx] = value;
}

// kCluster false: grid (kv_heads, batch, splits), chunks in decreasing index order; partials
//   acc [B, Hq, splits, D], ml [B, Hq, splits, 2] for the merge kernel.
// kCluster true: grid (kv_heads, batch, parts), the parts of a (sequence, KV head) are one cluster and
//   cut the sequence's own length evenly; their partials meet in distributed shared memory and the
//   output leaves from here, so the call is one launch and needs no scratch.
// kThirds: P in three bf16 parts (24 bits) instead of two, see keeps_24_bits.
template <int D, bool kCluster, bool kThirds>
__global__ void __launch_bounds__(kDecodeThreads, 2)
gqa_decode_tc(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
              DecodeArgs a) {
  constexpr int kTile = pluto::kTile<D>, kTokenWarps = pluto::kTokenWarps<D>;
  constexpr int kHalves = D / 64;                 // 64-column (128-byte) swizzled slabs per row
  constexpr int kHalfBytes = kTile * 128;         // one slab of a tile
  constexpr int kTileBytes = kHalves * kHalfBytes;
  constexpr int kStageBytes = 2 * kTileBytes;     // K tile then V tile
  constexpr int kParts = kChannelParts<D>, kWarps = kTokenWarps * kParts;
  static_assert((kWarps + 1) * 32 == kDecodeThreads, "warps");
  constexpr int kOwnBlocks = D / 16 / kParts;     // 16-channel blocks of the accumulator a warp owns
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  DecodeBarriers* bar = reinterpret_cast<DecodeBarriers*>(smem + kDecodeStages * kStageBytes);

  // Launched with programmatic stream serialisation: the set-up of this grid overlaps the end of the
  // one before it, whose results (query, lengths, cache) are read only after the wait.
  if (threadIdx.x == 0) {
    for (int s = 0; s < kDecodeStages; ++s) {
      mbar_init(&bar->full[s], 1);
      mbar_init(&bar->empty[s], kWarps);
    }
    mbar_fence_init();
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  pdl_wait();
  pdl_launch_dependents();   // the merge (or the next call) may be placed as SMs free up

  const int kv_head = blockIdx.x, b = blockIdx.y;
  const int length = bounded_length(a, b, 36);
  int begin, end, split = 0;
  if (kCluster) {
    const int parts = gridDim.z, chunk = ((length + parts - 1) / parts + kTile - 1) / kTile * kTile;
    begin = min(length, static_cast<int>(blockIdx.z) * chunk);
    end = min(length, begin + chunk);
  } else {
    // chunks in decreasing index order, (KV head, sequence) fastest: the four short chunks of every
    // sequence are the last CTAs of the launch
    split = gridDim.z - 1 - blockIdx.z;
    begin = decode_chunk_begin(split, a.split_tokens);
    if (begin >= length) return;  // whole CTA leaves before touching any barrier
    end = min(length, begin + decode_chunk_tokens(split, a.split_tokens));
  }
  const int tiles = (end - begin + kTile - 1) / kTile;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int group = a.q_heads / a.kv_heads;
  __syncthreads();

  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};
  float o[2 * kOwnBlocks][4];
  const int token_warp = warp % kTokenWarps, part = warp / kTokenWarps;

  if (warp == kWarps) {
    // ---------------------------------------------------------------- producer warp
    if (lane == 0) {
      bool ok = true;
      const int rows = a.box_rows;  // tokens per box: divides both the tile and the page size
      for (int it = 0; it < tiles && ok; ++it) {
        const int st = it % kDecodeStages, use = it / kDecodeStages;
        if (use > 0) ok = mbar_wait(&bar->empty[st], (use - 1) & 1, a.status, 30);
        if (!ok) break;
        const int t0 = begin + it * kTile;
        const int boxes = min(kTile, end - t0 + rows - 1) / rows;  // boxes that hold a live token
        mbar_expect_tx(&bar->full[st], static_cast<uint32_t>(boxes) * rows * D * 2 * 2);
        uint8_t* k_tile = smem + st * kStageBytes;
        uint8_t* v_tile = k_tile + kTileBytes;
        for (int bx = 0; bx < boxes; ++bx) {
          const int t = t0 + bx * rows;
          const int page = a.block_table
                               ? a.block_table[static_cast<size_t>(b) * a.max_blocks + t / a.page_size]
                               : b;
          const int in_page = t % a.page_size;
#pragma unroll
          for (int h = 0; h < kHalves; ++h) {
            tma_load_4d(k_tile + h * kHalfBytes + bx * rows * 128, &map_k, h * 64, kv_head, in_page,
                        page, &bar->full[st]);
            tma_load_4d(v_tile + h * kHalfBytes + bx * rows * 128, &map_v, h * 64, kv_head, in_page,
                        page, &bar->full[st]);
          }
        }
      }
      // all copies this thread started must have landed before the CTA may exit
      for (int it = max(0, tiles - kDecodeStages); it < tiles; ++it)
        mbar_wait(&bar->full[it % kDecodeStages], (it / kDecodeStages) & 1, a.status, 31);
    }
  } else {
    // ---------------------------------------------------------------- consumer warps
    // A fragments of Q: rows = query heads of this KV head (rows >= group are zero).
    uint32_t qf[D / 16][4];
    {
      const int r0 = lane / 4;
      const size_t head0 = static_cast<size_t>(b) * a.q_heads + static_cast<size_t>(kv_head) * group;
      const bool pairs = a.q_is_bf16 && (reinterpret_cast<uintptr_t>(a.q) & 3u) == 0;
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {   // rows r0, r0 + 8; columns 0-7, 8-15 of the step
          const int r = r0 + (i & 1) * 8, col = ks * 16 + (i >> 1) * 8 + (lane % 4) * 2;
          uint32_t packed = 0u;
          if (r < group) {
            const size_t at = (head0 + r) * D + col;
            if (pairs) {
              packed = *reinterpret_cast<const uint32_t*>(static_cast<const __nv_bfloat16*>(a.q) + at);
            } else if (a.q_is_bf16) {
              const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(a.q) + at;
              packed = pack_bf16(__bfloat162float(q[0]), __bfloat162float(q[1]));
            } else {
              const float* q = static_cast<const float*>(a.q) + at;
              packed = pack_bf16(q[0], q[1]);
            }
          }
          qf[ks][i] = packed;
        }
      }
    }
#pragma unroll
    for (int nb = 0; nb < 2 * kOwnBlocks; ++nb)
#pragma unroll
      for (int i = 0; i < 4; ++i) o[nb][i] = 0.0f;
    const float scale_log2 = a.scale * 1.4426950408889634f;
    bool ok = true;
    for (int it = 0; it < tiles && ok; ++it) {
      const int st = it % kDecodeStages;
      ok = mbar_wait(&bar->full[st], (it / kDecodeStages) & 1, a.status, 32);
      if (!ok) break;
      const uint32_t k_tile = smem_u32(smem + st * kStageBytes);
      const uint32_t v_tile = k_tile + kTileBytes;
      const int live = end - (begin + it * kTile);  // live tokens in this tile (may exceed kTile)
      if (live < (token_warp + 1) * 16) {
        // Rows past the sequence end hold whatever the page (or an earlier stage) held; their
        // probabilities are zero, but 0 * NaN would poison P V, so this warp clears its own dead
        // V rows (its channels of them) first.  Only the last tile of a sequence takes this path.
        for (int r = max(live, token_warp * 16); r < (token_warp + 1) * 16; ++r)
          for (int c = part * kHalves * 8 / kParts + lane; c < (part + 1) * kHalves * 8 / kParts; c += 32)
            sts_b32x4(v_tile + (c / 8) * kHalfBytes + r * 128 + (c % 8) * 16, 0u, 0u, 0u, 0u);
        fence_proxy_async();
        __syncwarp();
      }
      // ---- S = Q K^T for this warp's 16 tokens: two n-blocks of 8 tokens
      // (two accumulators each, for the even and the odd steps: the chain of dependent products is what
      // a tile waits for)
      float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      float s_odd[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int kp = 0; kp < D / 32; ++kp) {
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          uint32_t kf[4];
          // element (row, col) of a tile sits in slab col/64 at row*128 + ((col%64)/8 ^ row%8)*16
          const int row = token_warp * 16 + nb * 8 + lane % 8;
          const int chunk = (kp * 4 + lane / 8) % 8;
          ldmatrix_x4(kf, k_tile + (kp / 2) * kHalfBytes + row * 128 + ((chunk ^ (row % 8)) * 16));
          mma_bf16(s[nb], qf[2 * kp], kf[0], kf[1]);
          mma_bf16(s_odd[nb], qf[2 * kp + 1], kf[2], kf[3]);
        }
      }
      // ---- online softmax (rows lane/4 and lane/4+8; columns = tokens)
      const int token0 = begin + it * kTile + token_warp * 16 + (lane % 4) * 2;
      float tile_max[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int token = token0 + nb * 8 + (i & 1);
          s[nb][i] = token < end ? (s[nb][i] + s_odd[nb][i]) * scale_log2 : -INFINITY;
          tile_max[i >> 1] = fmaxf(tile_max[i >> 1], s[nb][i]);
        }
      // P enters P V as a bf16 high part and a bf16 remainder, 16 bits, which is free in a bandwidth-bound
      // kernel; with kThirds as a second remainder too, 24 bits, which is not (64 sequences of 32768 tokens,
      // 8 KV heads of 128: 718 us with two, 796 with three).
      uint32_t pf[4], pl[4], pt[4];
      float correction[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        tile_max[r] = fmaxf(tile_max[r], __shfl_xor_sync(0xffffffffu, tile_max[r], 1));
        tile_max[r] = fmaxf(tile_max[r], __shfl_xor_sync(0xffffffffu, tile_max[r], 2));
        const float m_new = fmaxf(m_run[r], tile_max[r]);
        const float m_safe = m_new == -INFINITY ? 0.0f : m_new;
        correction[r] = fast_exp2(m_run[r] - m_safe);
        const float p00 = fast_exp2(s[0][2 * r] - m_safe), p01 = fast_exp2(s[0][2 * r + 1] - m_safe);
        const float p10 = fast_exp2(s[1][2 * r] - m_safe), p11 = fast_exp2(s[1][2 * r + 1] - m_safe);
        float sum = p00 + p01 + p10 + p11;
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        l_run[r] = l_run[r] * correction[r] + sum;
        m_run[r] = m_new;
        pf[r] = pack_bf16(p00, p01);      // a0 / a1: tokens 0-7
        pf[2 + r] = pack_bf16(p10, p11);  // a2 / a3: tokens 8-15
        const float r00 = p00 - bf16_lo(pf[r]), r01 = p01 - bf16_hi(pf[r]);
        const float r10 = p10 - bf16_lo(pf[2 + r]), r11 = p11 - bf16_hi(pf[2 + r]);
        pl[r] = pack_bf16(r00, r01);
        pl[2 + r] = pack_bf16(r10, r11);
        if (kThirds) {
          pt[r] = pack_bf16(r00 - bf16_lo(pl[r]), r01 - bf16_hi(pl[r]));
          pt[2 + r] = pack_bf16(r10 - bf16_lo(pl[2 + r]), r11 - bf16_hi(pl[2 + r]));
        }
      }
      // ---- O = O * correction + P V over this warp's channels; the high-part products of two blocks
      // before their remainders, so that no product waits for the one just issued.  Every tile starts
      // from zero and is added in fp32: the tensor cores truncate when they accumulate, and over the
      // hundreds of tiles of a long sequence that would add up.
#pragma unroll
      for (int np = 0; np < kOwnBlocks; np += 2) {
        uint32_t vf[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int block = part * kOwnBlocks + np + u;
          const int row = token_warp * 16 + ((lane / 8) & 1) * 8 + lane % 8;
          const int chunk = (block * 2 + lane / 16) % 8;
          ldmatrix_x4_trans(vf[u], v_tile + (block / 4) * kHalfBytes + row * 128 + ((chunk ^ (row % 8)) * 16));
        }
        float pv[4][4] = {};
#pragma unroll
        for (int u = 0; u < 4; ++u) mma_bf16(pv[u], pf, vf[u / 2][(u & 1) * 2], vf[u / 2][(u & 1) * 2 + 1]);
#pragma unroll
        for (int u = 0; u < 4; ++u) mma_bf16(pv[u], pl, vf[u / 2][(u & 1) * 2], vf[u / 2][(u & 1) * 2 + 1]);
        if (kThirds) {
#pragma unroll
          for (int u = 0; u < 4; ++u) mma_bf16(pv[u], pt, vf[u / 2][(u & 1) * 2], vf[u / 2][(u & 1) * 2 + 1]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int i = 0; i < 4; ++i) o[2 * np + u][i] = fmaf(o[2 * np + u][i], correction[i >> 1], pv[u][i]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->empty[st]);
    }
  }
  __syncthreads();  // every stage consumed, every copy landed: the ring can be reused as scratch

  // ---- merge the token groups' partial softmax states through shared memory (ld.shared / st.shared
  // by address: `smem` went through alignment arithmetic and is a generic pointer).  Rows are 8 floats
  // longer than the head, so that the pair stores of half a warp (4 rows x 4 pairs) hit all banks once.
  constexpr int kRow = D + 8;
  const uint32_t scratch = smem_u32(smem);                               // fp32 [token groups][16][kRow]
  const uint32_t scratch_ml = scratch + kTokenWarps * 16 * kRow * 4;     // fp32 [token groups][16][2]
  const uint32_t merged = scratch + kDecodeStages * kStageBytes / 2;     // fp32 [16][D], [16][2], [parts][16][2]
  const uint32_t merged_ml = merged + 16 * D * 4, all_ml = merged_ml + 16 * 8;
  static_assert(kTokenWarps * 16 * (kRow + 2) * 4 <= kDecodeStages * kStageBytes / 2 &&
                    16 * (D + 2 + 2 * kMaxClusterParts) * 4 <= kDecodeStages * kStageBytes / 2, "merge scratch");
  if (warp < kWarps) {
    const int r0 = lane / 4;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int r = r0 + half * 8;
      if (r >= group) continue;   // rows without a query head
      const uint32_t row = scratch + ((token_warp * 16 + r) * kRow + part * (D / kParts) + (lane % 4) * 2) * 4;
#pragma unroll
      for (int nb = 0; nb < 2 * kOwnBlocks; ++nb)
        sts_b64(row + nb * 32, f2_pack(o[nb][2 * half], o[nb][2 * half + 1]));
      if (lane % 4 == 0 && part == 0)
        sts_b64(scratch_ml + (token_warp * 16 + r) * 8, f2_pack(m_run[half], l_run[half]));
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < group * D; idx += kDecodeThreads) {
    const int r = idx / D, d = idx % D;
    float m_w[kTokenWarps], m_tot = -INFINITY;
#pragma unroll
    for (int w = 0; w < kTokenWarps; ++w) {
      m_w[w] = lds_f32(scratch_ml + ((w * 16 + r) * 2) * 4);
      m_tot = fmaxf(m_tot, m_w[w]);
    }
    const float m_safe = m_tot == -INFINITY ? 0.0f : m_tot;   // a cluster part without tokens
    float acc = 0.0f, l_tot = 0.0f;
#pragma unroll
    for (int w = 0; w < kTokenWarps; ++w) {
      const float f = fast_exp2(m_w[w] - m_safe);
      acc += lds_f32(scratch + ((w * 16 + r) * kRow + d) * 4) * f;
      l_tot += lds_f32(scratch_ml + ((w * 16 + r) * 2 + 1) * 4) * f;
    }
    if (kCluster) {
      sts_f32(merged + idx * 4, acc);
      if (d == 0) {
        sts_f32(merged_ml + r * 8, m_tot);
        sts_f32(merged_ml + r * 8 + 4, l_tot);
      }
    } else {
      const size_t head = static_cast<size_t>(b) * a.q_heads + static_cast<size_t>(kv_head) * group + r;
      const size_t slot = head * a.splits + split;
      a.partial_acc[slot * D + d] = acc;
      if (d == 0) {
        a.partial_ml[slot * 2] = m_tot;
        a.partial_ml[slot * 2 + 1] = l_tot;
      }
    }
  }
  if (!kCluster) return;

  // ---- the parts' states, in part order; the cluster shares the group's outputs out
  const int parts = gridDim.z;
  cluster_sync();
  for (int i = threadIdx.x; i < parts * group * 2; i += kDecodeThreads) {
    const int z = i / (group * 2), at = i % (group * 2);
    sts_f32(all_ml + (z * 32 + at) * 4, lds_cluster_f32(merged_ml + at * 4, z));
  }
  __syncthreads();
  for (int idx = blockIdx.z * kDecodeThreads + threadIdx.x; idx < group * D; idx += parts * kDecodeThreads) {
    const int r = idx / D, d = idx % D, head = kv_head * group + r;
    float x[kMaxClusterParts], m_tot = -INFINITY;
#pragma unroll
    for (int z = 0; z < kMaxClusterParts; ++z)
      if (z < parts) {
        x[z] = lds_cluster_f32(merged + idx * 4, z);
        m_tot = fmaxf(m_tot, lds_f32(all_ml + (z * 32 + r * 2) * 4));
      }
    float acc = 0.0f, l = 0.0f;
#pragma unroll
    for (int z = 0; z < kMaxClusterParts; ++z)
      if (z < parts) {
        const float m = lds_f32(all_ml + (z * 32 + r * 2) * 4);
        const float w = m == -INFINITY ? 0.0f : fast_exp2(m - m_tot);
        acc = fmaf(x[z], w, acc);
        l = fmaf(lds_f32(all_ml + (z * 32 + r * 2 + 1) * 4), w, l);
      }
    // (a length of zero is a caller error: zeros, not 0 / 0)
    store_output(a, b, head, d, length > 0 ? acc / l : 0.0f);
    if (d == 0 && a.lse)
      a.lse[static_cast<size_t>(b) * a.q_heads + head] = length > 0 ? m_tot * 0.6931471805599453f + logf(l) : -INFINITY;
  }
  cluster_sync();   // the peers' shared memory is read until here
}

// ---------------------------------------------------------------------------------------------
// Exact fp32 kernel with the same split structure: grid (q_heads, batch, splits), one warp per
// token row in flight, each lane owning head_dim/32 (<= 8) channels.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) gqa_decode_generic(DecodeArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int split = gridDim.z - 1 - blockIdx.z, head = blockIdx.x, b = blockIdx.y;
  const int length = bounded_length(a, b, 37);
  const int begin = decode_chunk_begin(split, a.split_tokens);
  if (begin >= length) return;
  const int end = min(length, begin + decode_chunk_tokens(split, a.split_tokens));
  const int D = a.head_dim, kv_head = head / (a.q_heads / a.kv_heads);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const size_t element = a.kv_is_bf16 ? 2 : 4;
  float q[8], acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int d = lane + 32 * i;
    const size_t idx = (static_cast<size_t>(b) * a.q_heads + head) * D + d;
    q[i] = d < D ? (a.q_is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(a.q)[idx])
                                : static_cast<const float*>(a.q)[idx])
                 : 0.0f;
    acc[i] = 0.0f;
  }
  float m = -INFINITY, l = 0.0f;
  for (int t = begin + warp; t < end; t += 4) {
    const char* kr = kv_row(a, false, b, t, kv_head, element);
    const char* vr = kv_row(a, true, b, t, kv_head, element);
    float dot = 0.0f, v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int d = lane + 32 * i;
      float kx = 0.0f;
      v[i] = 0.0f;
      if (d < D) {
        if (a.kv_is_bf16) {
          kx = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(kr)[d]);
          v[i] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(vr)[d]);
        } else {
          kx = reinterpret_cast<const float*>(kr)[d];
          v[i] = reinterpret_cast<const float*>(vr)[d];
        }
      }
      dot = fmaf(kx, q[i], dot);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    const float s = dot * a.scale;
    const float m_new = fmaxf(m, s);
    const float correction = expf(m - m_new), p = expf(s - m_new);
    l = l * correction + p;
    m = m_new;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = fmaf(p, v[i], acc[i] * correction);
  }
  __shared__ float sh_acc[4][256];
  __shared__ float sh_ml[4][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) sh_acc[warp][lane + 32 * i] = acc[i];
  if (lane == 0) { sh_ml[warp][0] = m; sh_ml[warp][1] = l; }
  __syncthreads();
  float m_tot = fmaxf(fmaxf(sh_ml[0][0], sh_ml[1][0]), fmaxf(sh_ml[2][0], sh_ml[3][0]));
  const size_t slot = (static_cast<size_t>(b) * a.q_heads + head) * a.splits + split;
  for (int d = threadIdx.x; d < D; d += 128) {
    float sum = 0.0f;
    for (int w = 0; w < 4; ++w) sum += sh_acc[w][d] * expf(sh_ml[w][0] - m_tot);
    a.partial_acc[slot * D + d] = sum;
  }
  if (threadIdx.x == 0) {
    float l_tot = 0.0f;
    for (int w = 0; w < 4; ++w) l_tot += sh_ml[w][1] * expf(sh_ml[w][0] - m_tot);
    // partial maxima are kept in log2 units so both producers feed one merge kernel
    a.partial_ml[slot * 2] = m_tot * 1.4426950408889634f;
    a.partial_ml[slot * 2 + 1] = l_tot;
  }
}

// Merge of the per-chunk partials in chunk order, then the reference's output stage
// (cached_attention_ops.cc:120-125): out = R(R(acc/l) * R(sigmoid(gate))).  grid (q_heads, batch),
// 128 threads.  The chunks' maxima are reduced in parallel and every chunk's weight
// 2^(m_s - m) is computed once, by one thread, into shared memory; the sums then run over the
// chunks in order (so the result does not depend on the thread count) with the loads of eight
// chunks in flight.
constexpr int kMergeThreads = 128;
constexpr int kMergeSplits = 1024;   // chunk weights held in shared memory per pass

__global__ void __launch_bounds__(kMergeThreads) gqa_decode_merge(DecodeArgs a) {
  pdl_wait();   // the chunk kernel's partials are complete and visible from here on
  pdl_launch_dependents();
  const int head = blockIdx.x, b = blockIdx.y, D = a.head_dim;
  const int length = bounded_length(a, b, 38);
  const int splits = decode_chunk_count(length, a.split_tokens);   // <= a.splits
  if (length <= 0) {
    // nothing to attend to (a caller error: lengths are >= 1): zeros, not 0/0
    for (int d = threadIdx.x; d < D; d += kMergeThreads) {
      const size_t idx = (static_cast<size_t>(b) * a.q_heads + head) * D + d;
      if (a.out_is_bf16) static_cast<__nv_bfloat16*>(a.out)[idx] = __float2bfloat16_rn(0.0f);
      else static_cast<float*>(a.out)[idx] = 0.0f;
    }
    if (threadIdx.x == 0 && a.lse) a.lse[static_cast<size_t>(b) * a.q_heads + head] = -INFINITY;
    return;
  }
  const size_t slot0 = (static_cast<size_t>(b) * a.q_heads + head) * a.splits;
  __shared__ float weight[kMergeSplits];   // 2^(m_s - m_tot)
  __shared__ float scaled_l[kMergeSplits]; // l_s * weight_s
  __shared__ float warp_max[kMergeThreads / 32];
  const float2* ml = reinterpret_cast<const float2*>(a.partial_ml) + slot0;   // (m_s, l_s)

  float m_part = -INFINITY;
  for (int s = threadIdx.x; s < splits; s += kMergeThreads) m_part = fmaxf(m_part, ml[s].x);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m_part = fmaxf(m_part, __shfl_xor_sync(0xffffffffu, m_part, o));
  if (threadIdx.x % 32 == 0) warp_max[threadIdx.x / 32] = m_part;
  __syncthreads();
  float m_tot = warp_max[0];
#pragma unroll
  for (int w = 1; w < kMergeThreads / 32; ++w) m_tot = fmaxf(m_tot, warp_max[w]);

  float l_tot = 0.0f;
  float acc[2] = {0.0f, 0.0f};               // channels threadIdx.x and threadIdx.x + 128
  for (int s0 = 0; s0 < splits; s0 += kMergeSplits) {
    const int count = min(kMergeSplits, splits - s0);
    __syncthreads();                          // the previous pass is done with the arrays
    for (int s = threadIdx.x; s < count; s += kMergeThreads) {
      const float2 v = ml[s0 + s];
      const float w = exp2f(v.x - m_tot);
      weight[s] = w;
      scaled_l[s] = v.y * w;
    }
    __syncthreads();
    for (int s = 0; s < count; ++s) l_tot += scaled_l[s];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int d = threadIdx.x + c * kMergeThreads;
      if (d >= D) continue;
      const float* column = a.partial_acc + (slot0 + s0) * D + d;
      int s = 0;
      for (; s + 8 <= count; s += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = column[static_cast<size_t>(s + u) * D];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc[c] += v[u] * weight[s + u];
      }
      for (; s < count; ++s) acc[c] += column[static_cast<size_t>(s) * D] * weight[s];
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int d = threadIdx.x + c * kMergeThreads;
    if (d < D) store_output(a, b, head, d, acc[c] / l_tot);
  }
  if (threadIdx.x == 0 && a.lse) {
    // natural-log sum-exp of the scaled scores
    a.lse[static_cast<size_t>(b) * a.q_heads + head] = m_tot * 0.6931471805599453f + logf(l_tot);
  }
}

// Two-pass softmax row per (head, sequence) for the inspection hook: row (b, h) of `length`
// entries starts at probs + b*batch_stride + h*head_stride.  grid (q_heads, batch), 256 threads.
__global__ void __launch_bounds__(256) gqa_decode_probs(DecodeArgs a, float* probs,
                                                        size_t batch_stride, size_t head_stride) {
  const int head = blockIdx.x, b = blockIdx.y, D = a.head_dim;
  const int length = a.seq_lens[b];
  const int kv_head = head / (a.q_heads / a.kv_heads);
  const size_t element = a.kv_is_bf16 ? 2 : 4;
  float* row = probs + static_cast<size_t>(b) * batch_stride + static_cast<size_t>(head) * head_stride;
  __shared__ float red[256];
  const size_t q0 = (static_cast<size_t>(b) * a.q_heads + head) * D;
  float local_max = -INFINITY;
  for (int t = threadIdx.x; t < length; t += 256) {
    const char* kr = kv_row(a, false, b, t, kv_head, element);
    float dot = 0.0f;
    for (int d = 0; d < D; ++d) {
      const float kx = a.kv_is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(kr)[d])
                                    : reinterpret_cast<const float*>(kr)[d];
      const float qx = a.q_is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(a.q)[q0 + d])
                                   : static_cast<const float*>(a.q)[q0 + d];
      dot = fmaf(kx, qx, dot);
    }
    row[t] = dot * a.scale;
    local_max = fmaxf(local_max, dot * a.scale);
  }
  red[threadIdx.x] = local_max;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + o]);
    __syncthreads();
  }
  const float m = red[0];
  __syncthreads();
  float local_sum = 0.0f;
  for (int t = threadIdx.x; t < length; t += 256) local_sum += expf(row[t] - m);
  red[threadIdx.x] = local_sum;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  const float inv = 1.0f / red[0];
  for (int t = threadIdx.x; t < length; t += 256) row[t] = expf(row[t] - m) * inv;
}

template <int D>
constexpr size_t decode_smem() {
  return 1024 + kDecodeStages * kDecodeStageBytes<D> + sizeof(DecodeBarriers);
}

// 4-D map of a bf16 page pool: (column, kv head, token in page, page); box = 64 columns x
// box_rows tokens of one kv head, 128-byte swizzle, zero fill outside the pool.
bool make_pool_map(CUtensorMap* map, const void* base, const DecodeArgs& a, int pages) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                              const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Encode encode = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult result;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &result) !=
            cudaSuccess || result != cudaDriverEntryPointSuccess)
      return static_cast<Encode>(nullptr);
    return reinterpret_cast<Encode>(sym);
  }();
  if (encode == nullptr) return false;
  const cuuint64_t dims[4] = {static_cast<cuuint64_t>(a.head_dim), static_cast<cuuint64_t>(a.kv_heads),
                              static_cast<cuuint64_t>(a.page_size), static_cast<cuuint64_t>(pages)};
  const cuuint64_t strides[3] = {static_cast<cuuint64_t>(a.head_dim) * 2, a.token_stride * 2,
                                 a.page_stride * 2};
  const cuuint32_t box[4] = {64, 1, static_cast<cuuint32_t>(a.box_rows), 1};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides,
                box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

}  // namespace

namespace {
// Calls that the tensor-core form took over from the plain kernel keep its precision: P with 24 bits.  They are
// head width 256 and contiguous caches of a length that 16 does not divide; all others have always had 16.
bool keeps_24_bits(const DecodeArgs& a) { return a.head_dim == 256 || (a.block_table == nullptr && a.page_size % 16 != 0); }
}  // namespace

// Of those calls the plain kernel keeps fp32 queries, which the tensor cores would round to bf16, and fp32
// results that nothing rounds: P has 24 bits either way, but a score is a sum that the tensor cores truncate
// (width 256, relative error of the result 2.1e-7 against 1.3e-7 at 64 tokens, 2.7e-7 against 1.9e-7 at 500,
// equal from 4000 on).
bool gqa_decode_uses_tensor_cores(const DecodeArgs& a) {
  if (keeps_24_bits(a) && (!a.q_is_bf16 || (!a.round && !a.out_is_bf16))) return false;
  const int group = a.q_heads / a.kv_heads;
  const int pages = a.block_table ? a.num_pages : a.batch;
  return a.k_bases == nullptr && a.kv_is_bf16 && (a.head_dim == 64 || a.head_dim == 128 || a.head_dim == 256) && group <= 16 &&
         (a.round || a.q_is_bf16) && a.token_stride % 8 == 0 && a.page_stride % 8 == 0 &&
         (a.block_table == nullptr || a.page_size % 16 == 0) && pages > 0 &&
         (reinterpret_cast<uintptr_t>(a.k_base) & 15u) == 0 &&
         (reinterpret_cast<uintptr_t>(a.v_base) & 15u) == 0;
}

namespace {

template <typename... Params>
cudaError_t launch_decode(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                          int cluster_z, const Params&... params) {
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[0].val.programmaticStreamSerializationAllowed = 1;
  attributes[1].id = cudaLaunchAttributeClusterDimension;
  attributes[1].val.clusterDim.x = attributes[1].val.clusterDim.y = 1;
  attributes[1].val.clusterDim.z = static_cast<unsigned>(cluster_z);
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = attributes;
  config.numAttrs = cluster_z > 0 ? 2 : 1;
  return cudaLaunchKernelEx(&config, kernel, params...);
}

template <int D, bool kThirds>
cudaError_t launch_tc(cudaStream_t stream, const CUtensorMap& map_k, const CUtensorMap& map_v, const DecodeArgs& a,
                      int parts) {
  auto kernel = parts > 0 ? gqa_decode_tc<D, true, kThirds> : gqa_decode_tc<D, false, kThirds>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(decode_smem<D>()));
  if (e == cudaSuccess && parts > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  return launch_decode(kernel, dim3(a.kv_heads, a.batch, parts > 0 ? parts : a.splits), kDecodeThreads,
                       decode_smem<D>(), stream, parts, map_k, map_v, a);
}

// Parts per (sequence, KV head) of the one-launch form, 0 for chunks + merge kernel.  A cluster lives in one
// GPC, so only so many are resident at once, two CTAs per SM: 14 of 16 parts, 20 of 12, 33 of 8, 66 of 4, 148
// of 2; one more doubles the time (600 tokens, width 128, us: 14 units in 16 parts 6.3, 15 11.1 in 16 and 6.1
// in 12; 20 in 12 6.3, 22 10.5 in 12 and 6.7 in 8; 33 in 8 7.6, 34 11.7 in 8 and 7.1 in 4; 66 in 4 8.9, 72 14.0
// in 4 and 9.7 in 2; 148 in 2 13.2, 160 21.0 in 2 and 16.6 in 1).  A part keeps at least 32 tokens.  More than 8
// parts are beyond the portable cluster size and opted into.
// Chunks and their merge take over
// - above 256 MB of cache (about 40 us of HBM), where the merge is a few per cent and whole-chip balance
//   counts: 240 units of 4000 tokens (width 256) 143 against 113 us, 64 of 20000 171 / 144, 720 of 8000
//   (width 64) 175 / 138;
// - where the parts are few and long, so that a few CTAs stream what the chip could.  One launch against
//   chunks + merge, us:
//     units       width 64            width 128                    width 256
//       1    16384 10.9 / 10.8   8192  9.3 / 10.4           4000 14.4 / 18.3, 8192 23.1 / 21.4
//            32768 19.2 / 15.6  32768 24.8 / 19.3          32768 75.4 / 38.4
//       2    32768 19.5 / 18.2  16384 15.0 / 14.4, 32768 25.2 / 22.6  8192 23.1 / 20.4, 32768 75.9 / 39.3
//       4    32768 20.0 / 22.1  32768 26.0 / 29.7           4000 14.7 / 18.6, 16384 41.2 / 30.6
//       8    32768 23.1 / 32.0  32768 31.9 / 46.0           4000 17.5 / 20.9, 16384 49.7 / 48.2, 32768 92.9 / 95.1
//      16    32768 41.2 / 50.0  16384 31.4 / 40.4           3000 17.8 / 22.7
//      32    32768 44.8 / 63.2  16384 43.0 / 68.0           8192 52.0 / 75.5
//   A CTA of width 256 (32-token tiles, P in three parts) streams 29 GB/s, the others 45 to 50, so there
//   the line lies at 64 CTAs and 400 tokens a part, else at 32 CTAs and 900 tokens.
int cluster_parts(const DecodeArgs& a) {
  const long long units = static_cast<long long>(a.batch) * a.kv_heads;
  if (units * a.max_length * a.head_dim * 4 > 256LL << 20) return 0;
  int z = units <= 12 ? 16 : units <= 20 ? 12 : units <= 32 ? 8 : units <= 64 ? 4 : units <= 148 ? 2 : 1;
  while (z > 1 && a.max_length < z * 32) z = z == 12 ? 8 : z / 2;
  const bool wide = a.head_dim == 256;
  return units * z <= (wide ? 64 : 32) && a.max_length > z * (wide ? 400 : 900) ? 0 : z;
}

}  // namespace

cudaError_t gqa_decode(cudaStream_t stream, const DecodeArgs& args) {
  DecodeArgs a = args;
  cudaError_t e;
  if (gqa_decode_uses_tensor_cores(a)) {
    // (without a block table a box past the end of its sequence's region reads zeros: any size goes)
    const int tile = a.head_dim == 256 ? kTile<256> : kTile<128>;
    a.box_rows = a.block_table == nullptr || a.page_size % tile == 0 ? tile : 16;
    const int pages = a.block_table ? a.num_pages : a.batch;
    CUtensorMap map_k, map_v;
    if (!make_pool_map(&map_k, a.k_base, a, pages) || !make_pool_map(&map_v, a.v_base, a, pages))
      return cudaErrorInvalidValue;
    const int parts = cluster_parts(a);
    const bool thirds = keeps_24_bits(a);
    auto launch = a.head_dim == 256 ? launch_tc<256, true>
                  : a.head_dim == 128 ? (thirds ? launch_tc<128, true> : launch_tc<128, false>)
                                      : (thirds ? launch_tc<64, true> : launch_tc<64, false>);
    e = launch(stream, map_k, map_v, a, parts);
    if (e != cudaSuccess || parts > 0) return e;
  } else {
    e = launch_decode(gqa_decode_generic, dim3(a.q_heads, a.batch, a.splits), 128, 0, stream, 0, a);
    if (e != cudaSuccess) return e;
  }
  // The merge's CTAs are placed while the chunk kernel's last CTAs still run, and wait for that grid
  // before they read a partial.
  return launch_decode(gqa_decode_merge, dim3(a.q_heads, a.batch), kMergeThreads, 0, stream, 0, a);
}

cudaError_t gqa_decode_probabilities(cudaStream_t stream, const DecodeArgs& a, float* probs,
                                     size_t batch_stride, size_t head_stride) {
  gqa_decode_probs<<<dim3(a.q_heads, a.batch), 256, 0, stream>>>(a, probs, batch_stride, head_stride);
  return cudaGetLastError();
}

}  // namespace pluto
