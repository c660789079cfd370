// FP32-accurate matrix products on the FP16 tensor cores: every operand is the sum of two FP16 values,
//   v * s = v1 + v2,   v1 = fp16(v * s),  v2 = fp16(v * s - v1)      (s a power of two)
// which carries 22 significant bits and more, and a product of two operands is three MMAs (v1 w1, v1 w2, v2 w1; the
// dropped v2 w2 is below 2^-24 of v1 w1). The scale s keeps v * s below 2^14: nothing overflows, and since the absolute
// error of the pair never exceeds 2^-39 of that bound, a bound that is loose by a factor of 2^15 costs no accuracy. Bounds and
// scales are a channel's own (split_pack.cuh).
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

// ---- roles of a block --------------------------------------------------------------------------------------
constexpr int WORK_WARPS = 16, WORK_THREADS = WORK_WARPS * 32;
// Two issuing warps take the slabs in turn: a suspending poll of a barrier costs about 220 cycles in the issuing thread even
// when the barrier is ready, and no MMA of that thread is queued meanwhile (one 288-cycle slab per poll: 532 cycles a slab
// measured); with two threads one polls while the other's MMAs run. A slab's accumulator belongs to one thread, so its order
// is fixed.
constexpr int MMA_WARPS = 2, MMA_WARP = WORK_WARPS, PROD_WARP = WORK_WARPS + MMA_WARPS;
constexpr int THREADS = (WORK_WARPS + MMA_WARPS + 1) * 32;
constexpr int SYNC_THREADS = (WORK_WARPS + MMA_WARPS) * 32;   // working and MMA warps meet at barrier 1

// ---- operands and products -----------------------------------------------------------------------------------
constexpr int SLAB_K = 32;                                    // K of one weight slab = one partial sum
constexpr uint32_t SLAB_BYTES = 2u * 128u * SLAB_K * 2u;      // two planes of [K/8][128][8] FP16

// instruction descriptor: FP16 x FP16 -> FP32, both operands K-major, M x N tile
__host__ __device__ constexpr uint32_t idesc_f16(uint32_t M, uint32_t N) { return (1u << 4) | ((N >> 3) << 17) | ((M >> 4) << 24); }

// exponent e with bound <= 2^e, held in a range whose scales stay far from the ends of FP32
__device__ __forceinline__ int bound_exp(float bound) {
  if (!(bound > 9.0e-13f)) return -40;       // 2^-40
  if (!(bound < 1.2e30f)) return 100;        // 2^100 (and values that are not finite)
  return ilogbf(bound) + 1;
}
__device__ __forceinline__ float scale_for(float bound) { return scalbnf(1.0f, 14 - bound_exp(bound)); }

// both planes of one value, already scaled
__device__ __forceinline__ void split(float v, __half* v1, __half* v2) {
  const __half h = __float2half_rn(v);
  *v1 = h;
  *v2 = __float2half_rn(v - __half2float(h));
}

// Shared-memory descriptors of this scheme (tc::smem_desc: no swizzle, 128 bytes between groups of eight rows) differ only in
// their low words, so addresses are advanced in 32 bits and the high word is a constant of the instruction.
constexpr uint32_t DESC_HI = (128u >> 4) | (1u << 14);
__device__ __forceinline__ uint32_t desc_lo(const void* smem, uint32_t lbo_bytes) {
  return ((tc::smem_u32(smem) >> 4) & 0x3FFFu) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
}
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
      :
      : "r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(DESC_HI)
      : "memory");
}

// The MMAs of one slab of `ksteps` (1 or 2) K-steps into the accumulator at `d`: the small products first.
// a: descriptor of the slab's first plane (rows of 128 channels), b1 / b2: descriptors of the two activation planes at the
// slab's first panel, b_step: descriptor units between K-steps of the activations.
__device__ __forceinline__ void slab_mmas(uint32_t d, uint32_t a, uint32_t ksteps, uint32_t b1, uint32_t b2, uint32_t b_step, uint32_t idesc) {
  const uint32_t a2 = a + ksteps * ((16 * 128 * 2) >> 4);   // second plane follows the first
  constexpr uint32_t a_step = (2 * 128 * 16) >> 4;
  mma_f16(d, a2, b1, idesc, 0u);
  mma_f16(d, a, b2, idesc, 1u);
  if (ksteps > 1) {
    mma_f16(d, a2 + a_step, b1 + b_step, idesc, 1u);
    mma_f16(d, a + a_step, b2 + b_step, idesc, 1u);
  }
  mma_f16(d, a, b1, idesc, 1u);
  if (ksteps > 1) mma_f16(d, a + a_step, b1 + b_step, idesc, 1u);
}

// ---- ranges and barriers -----------------------------------------------------------------------------------
__device__ __forceinline__ int work_lower_bound(const int* __restrict__ row_ptr, int lo, int hi, long long target) {
  const long long base = (long long)row_ptr[lo] + lo;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if ((long long)row_ptr[mid] + mid - base < target) lo = mid + 1; else hi = mid;
  }
  return lo;
}

struct BlockRange { int n_begin, n_end; long long e_begin, e_end, ntiles; };

// node-aligned share of segment [lo, hi) for this block, balanced over edges + nodes
__device__ __forceinline__ BlockRange block_range(const int* __restrict__ row_ptr, int lo, int hi, int tile) {
  BlockRange r;
  const long long work = ((long long)row_ptr[hi] - row_ptr[lo]) + (hi - lo);
  long long per = (work + gridDim.x - 1) / gridDim.x;
  if (per < tile) per = tile;
  r.n_begin = blockIdx.x == 0 ? lo : work_lower_bound(row_ptr, lo, hi, per * blockIdx.x);
  r.n_end = blockIdx.x == gridDim.x - 1 ? hi : work_lower_bound(row_ptr, lo, hi, per * (blockIdx.x + 1));
  r.e_begin = r.n_begin < r.n_end ? row_ptr[r.n_begin] : 0;
  r.e_end = r.n_begin < r.n_end ? row_ptr[r.n_end] : 0;
  r.ntiles = (r.e_end - r.e_begin + tile - 1) / tile;
  return r;
}

// barrier 1: working warps + MMA warps; returns the OR of `flag` over its participants
__device__ __forceinline__ int sync_or(int flag) {
  int out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "barrier.cta.red.or.pred p, 1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(out) : "r"(flag), "n"(SYNC_THREADS) : "memory");
  return out;
}
// a bounded wait of a whole warp: every lane leaves with the same answer, since the loads from tensor memory and the barriers
// that follow need all of them (a lane that gave up alone would meet the others at different instructions)
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, tc::mbar_wait(bar, parity)) != 0; }
// barrier 2: working warps only
__device__ __forceinline__ void sync_workers() { asm volatile("barrier.cta.sync 2, %0;" ::"n"(WORK_THREADS) : "memory"); }

}  // namespace sf
