// FP32-accurate matrix products on the FP16 tensor cores: every operand is the sum of two FP16 values,
//   v * s = v1 + v2,   v1 = fp16(v * s),  v2 = fp16(v * s - v1)      (s a power of two)
// which carries 22 significant bits and more, and a product of two operands is three MMAs (v1 w1, v1 w2, v2 w1; the
// dropped v2 w2 is below 2^-24 of v1 w1). The scale s keeps v * s below 2^14: nothing overflows, and since the absolute
// error of the pair never exceeds 2^-39 of that bound, a bound that is loose by a factor of 2^15 costs no accuracy.
//
// The tensor cores truncate as they accumulate, which over a long K would cost more than FP32 FMAs do. So a partial sum
// covers K = 32 only, its two small products first, and is then added to an FP32 register (round to nearest).
//
// Products are formed transposed, D[channel][edge] = W[channel][k] * X[edge][k]: weights are the M operand, streamed from
// L2, a tile's activations the N operand, resident in shared memory; a thread then owns one channel of 64 edges.
#pragma once
#include <cuda_fp16.h>
#include "tc05.cuh"

namespace sf {

constexpr int SLAB_K = 32;                                    // K of one weight slab = one partial sum
constexpr uint32_t SLAB_BYTES = 2u * 128u * SLAB_K * 2u;      // two planes of [K/8][128][8] FP16

// instruction descriptor: FP16 x FP16 -> FP32, both operands K-major, M x N tile
__host__ __device__ constexpr uint32_t idesc_f16(uint32_t M, uint32_t N) { return (1u << 4) | ((N >> 3) << 17) | ((M >> 4) << 24); }

// exponent e with bound <= 2^e, held in a range whose scales stay far from the ends of FP32
__device__ __forceinline__ int bound_exp(float bound) {
  if (!(bound > 9.0e-13f)) return -40;       // 2^-40
  if (!(bound < 1.1e18f)) return 60;         // 2^60 (and values that are not finite)
  return ilogbf(bound) + 1;
}
__device__ __forceinline__ float scale_for(float bound) { return scalbnf(1.0f, 14 - bound_exp(bound)); }

// both planes of one value, already scaled
__device__ __forceinline__ void split(float v, __half* v1, __half* v2) {
  const __half h = __float2half_rn(v);
  *v1 = h;
  *v2 = __float2half_rn(v - __half2float(h));
}

// The MMAs of one slab of `ksteps` (1 or 2) K-steps into the accumulator at `d`: the small products first.
// a: descriptor of the slab's first plane (rows of 128 channels), b1 / b2: descriptors of the two activation planes at the
// slab's first panel, b_step: descriptor units between K-steps of the activations.
__device__ __forceinline__ void slab_mmas(uint32_t d, uint64_t a, uint32_t ksteps, uint64_t b1, uint64_t b2, uint64_t b_step, uint32_t idesc) {
  const uint64_t a2 = a + ((uint64_t)(ksteps * 16 * 128 * 2) >> 4);   // second plane follows the first
  constexpr uint64_t a_step = (2 * 128 * 16) >> 4;
  tc::mma_bf16(d, a2, b1, idesc, 0u);
  tc::mma_bf16(d, a, b2, idesc, 1u);
  if (ksteps > 1) {
    tc::mma_bf16(d, a2 + a_step, b1 + b_step, idesc, 1u);
    tc::mma_bf16(d, a + a_step, b2 + b_step, idesc, 1u);
  }
  tc::mma_bf16(d, a, b1, idesc, 1u);
  if (ksteps > 1) tc::mma_bf16(d, a + a_step, b1 + b_step, idesc, 1u);
}

}  // namespace sf
