// Weights of the split-precision kernels (split_f16.cuh), packed in streaming order with a scale for every channel.
//
// A hidden channel o is stored as h * 2^(14 - e_o), where 2^e_o bounds |h| over all inputs; the next layer's weights take
// 2^e_o up for their input o and are then scaled per output by their own largest value. So a channel that is far larger or
// smaller than the others costs these no bits (with one scale for a whole layer, a hidden unit of 10^5 beside others of 1,
// or one that its bias keeps off, left the results 8e-5 to 2.4e-4 off, against 1e-7 to 3e-7 of FP32 FMAs), and a thread, which
// owns an output channel, only reads its own scales.
//
// The bounds are those of interval arithmetic: |pre-activation| <= sum |W| bound + |b|. For SiLU, whose negative side is
// at most 0.2785 and falls off exponentially, a unit that a large negative bias keeps off is bounded by what it can reach.
// In the l<=2 layer the bounds are affine in the size `by` of an edge's products, |h_o| <= by p_o + q_o, and have to be
// taken apart into a channel's factor and an edge's: 2^e_o >= p_o + q_o (the size at by = 1), and for the edge the largest
// (by p_o + q_o) / (p_o + q_o) over the channels, which the extremes of q_o / p_o give (edge_size).
#pragma once
#include "common.cuh"
#include "split_f16.cuh"

namespace {

enum SplitBound { SPLIT_LAST, SPLIT_SILU, SPLIT_LINEAR, SPLIT_LEAKY };

struct SplitLayer {
  const float* Wt;                     // [K][N]
  int K, N;
  const float* in_p; const float* in_q; const float* in_scale;   // of the K inputs (null: bounds 1 / 0, scale 2^14)
  const float* bias;
  __half* out;                         // slabs [K chunk of 32][block of 128 outputs][plane][K/8][128][8]
  float* inv;                          // [N]: takes an accumulator back
  float* scale; float* p; float* q;    // [N]: scale 2^(14 - e) and bounds of this layer's results (not SPLIT_LAST)
  float* ratio;                        // with in_q: smallest and largest in_q / in_p
};

// A block packs 32 outputs; a lane is an output, the warps share the inputs. Bound by the latency of two dependent passes over
// the weights (512 x 512: 16 loads per thread in each).
template <SplitBound BOUND>
__global__ void __launch_bounds__(1024) split_layer_kernel(const SplitLayer L) {
  __shared__ float s_p[512], s_q[512], s_fold[512], s_red[3][32][33], s_sw[32], s_ratio[2][32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, o = blockIdx.x * 32 + lane, K = L.K, N = L.N;
  const bool live = o < N;
  float lo = INFINITY, hi = 0.f;
  for (int k = tid; k < K; k += 1024) {
    const float p = L.in_p != nullptr ? L.in_p[k] : 1.f, q = L.in_q != nullptr ? L.in_q[k] : 0.f;
    s_p[k] = p; s_q[k] = q;
    s_fold[k] = L.in_scale != nullptr ? 16384.f / L.in_scale[k] : 1.f;
    if (p > 0.f || q > 0.f) { lo = fminf(lo, q / p); hi = fmaxf(hi, q / p); }
  }
  if (L.ratio != nullptr && blockIdx.x == 0) {
    for (int d = 16; d > 0; d >>= 1) { lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d)); hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d)); }
    if (lane == 0) { s_ratio[0][w] = lo; s_ratio[1][w] = hi; }
  }
  __syncthreads();
  if (L.ratio != nullptr && blockIdx.x == 0 && tid == 0) {
    for (int i = 1; i < 32; i++) { lo = fminf(lo, s_ratio[0][i]); hi = fmaxf(hi, s_ratio[1][i]); }
    L.ratio[0] = lo; L.ratio[1] = hi;
  }
  float sp = 0.f, sq = 0.f, mx = 0.f;
  if (live)
#pragma unroll 4
    for (int k = w; k < K; k += 32) {
      const float a = fabsf(L.Wt[(size_t)k * N + o]);
      sp = fmaf(a, s_p[k], sp); sq = fmaf(a, s_q[k], sq);
      mx = fmaxf(mx, a * s_fold[k]);
    }
  s_red[0][w][lane] = sp; s_red[1][w][lane] = sq; s_red[2][w][lane] = mx;
  __syncthreads();
  if (w == 0) {
    for (int i = 1; i < 32; i++) { sp += s_red[0][i][lane]; sq += s_red[1][i][lane]; mx = fmaxf(mx, s_red[2][i][lane]); }
    sp *= 1.001f; sq *= 1.001f;   // the sums' own rounding
    const float sw = sf::scale_for(mx);
    s_sw[lane] = sw;
    if (live) {
      L.inv[o] = 1.0f / (sw * 16384.f);
      if (BOUND != SPLIT_LAST) {
        const float b = L.bias != nullptr ? L.bias[o] : 0.f;
        if (BOUND == SPLIT_SILU) {
          const float top = sp + b;   // of the pre-activation
          const float above = top > 0.f ? fmaxf(top, 0.2785f) : (top < -1.28f ? -top * expf(top) : 0.2785f);
          sp = fminf(above, sp + fabsf(b)) * 1.001f;
        } else {
          sq += fabsf(b);
          if (L.q != nullptr) L.q[o] = sq;
        }
        L.p[o] = sp;
        L.scale[o] = sf::scale_for(BOUND == SPLIT_SILU ? sp : sp + sq);
      }
    }
  }
  __syncthreads();
  const int kp = (K + 15) / 16 * 16, blocks = (N + 127) / 128;
  const float sw = live ? s_sw[lane] : 0.f;
  for (int kg = w; kg < kp / 8; kg += 32) {
    __align__(16) __half h1[8], h2[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int k = kg * 8 + i;
      sf::split(live && k < K ? L.Wt[(size_t)k * N + o] * s_fold[k] * sw : 0.f, &h1[i], &h2[i]);
    }
    const int ch = kg / 4, kw = min(sf::SLAB_K, kp - ch * sf::SLAB_K);
    __half* slab = L.out + (size_t)ch * sf::SLAB_K * blocks * 256 + (size_t)(o / 128) * kw * 256;
    __half* at = slab + (size_t)(kg % 4) * 1024 + (o % 128) * 8;
    *reinterpret_cast<uint4*>(at) = *reinterpret_cast<const uint4*>(h1);
    *reinterpret_cast<uint4*>(at + (size_t)kw * 128) = *reinterpret_cast<const uint4*>(h2);
  }
}

template <SplitBound BOUND>
int split_layer(const SplitLayer& L, cudaStream_t st) {
  split_layer_kernel<BOUND><<<ld_cdiv(L.N, 128) * 4, 1024, 0, st>>>(L);   // outputs up to whole blocks of 128 are zeros
  LD_LAUNCH_CHECK();
  return LD_OK;
}

}  // namespace
