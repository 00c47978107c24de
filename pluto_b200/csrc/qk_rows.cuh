// The vector that a query or key head becomes (norm, weight, rotation): one warp per row, shared by
// the prepare kernel (qk_prepare.cu) and the single-token step (token_step.cu), so that a token gets
// the same bits from both.
//
// The steps are the reference's, n = R(x * inv * (1 + w)); out = R(R(n * R(cos)) + R(+-n_partner *
// R(sin))).  The sum of squares is taken over blocks of 32 channels, a butterfly inside each (distances
// 16, 8, 4, 2, 1) and the blocks in order, whatever a lane owns; products and sums of the rotation are
// rounded one by one, so no contraction can tell the two kernels apart.
#pragma once

#include "common.cuh"

namespace pluto {

constexpr int kRowOwn = 8;   // channels a lane owns at width 256

// A lane owns kPer consecutive channels of every 32 * kPer; element i of its array is this channel.
template <int kPer>
__device__ __forceinline__ int row_channel(int i, int lane) {
  return (i / kPer) * 32 * kPer + lane * kPer + i % kPer;
}

// Sum of squares of a row whose elements past its width are zero.
template <int kPer>
__device__ __forceinline__ float row_square_sum(const float (&x)[kRowOwn], int lane) {
  static_assert(kPer == 1 || kPer == 4, "channels per access");
  float total = 0.0f;
  if (kPer == 1) {
#pragma unroll
    for (int i = 0; i < kRowOwn; ++i) {
      float s = __fmul_rn(x[i], x[i]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
      total = __fadd_rn(total, s);
    }
    return total;
  }
#pragma unroll
  for (int i = 0; i < kRowOwn; i += 4) {   // 128 channels: four blocks of eight lanes
    float s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s[u] = __fmul_rn(x[i + u], x[i + u]);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s[u] = __fadd_rn(s[u], __shfl_xor_sync(0xffffffffu, s[u], o));
    }
    const float block = __fadd_rn(__fadd_rn(s[0], s[2]), __fadd_rn(s[1], s[3]));
#pragma unroll
    for (int k = 0; k < 4; ++k) total = __fadd_rn(total, __shfl_sync(0xffffffffu, block, 8 * k));
  }
  return total;
}

// One rotated element: n and its partner are normalised, the partner already carries its sign.
__device__ __forceinline__ float rotate(float n, float partner, float cosine, float sine, int round) {
  const float a = __fmul_rn(n, cosine), b = __fmul_rn(partner, sine);
  return round ? bf16_round(__fadd_rn(bf16_round(a), bf16_round(b))) : __fadd_rn(a, b);
}

// cos and sin of a rotary pair at a position.
__device__ __forceinline__ void rotary_angle(int position, int pair, float log_theta, int rotary, int round, float& cosine,
                                             float& sine) {
  const float angle =
      static_cast<float>(position) * expf(static_cast<float>(pair) * (-2.0f * log_theta / static_cast<float>(rotary)));
  cosine = cosf(angle);
  sine = sinf(angle);
  if (round) {
    cosine = bf16_round(cosine);
    sine = bf16_round(sine);
  }
}

}  // namespace pluto
