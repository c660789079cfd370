// PaiNN message step at FP32 accuracy with the distance MLP on the tensor cores: the computation of painn_message.cu
// (Message.forward, archs/meanflow_painn8.py:77-100) with operands split into two FP16 values (split_f16.cuh).
//
// What bounds it: the phases of a tile, which follow one another (matrix products, epilogue, messages, sums), and within the
// products the shared-memory port. The two 4n x 4n layers are 3 x 2 x (4n)^2 flops an edge on the tensor cores; an MMA of
// 128 x 64 x 16 (n = 128) takes 48 cycles, the time to read its 6 KB of operands, not the 32 of the tensor pipe, and the weight
// slabs (2 MB per tile) come in through the same port: 433 cycles a slab of six MMAs measured, 416 by that count. Over the
// launch the tensor pipe is active 29 % of the time.
// n = 128, 8 radial functions, 562 k edges: 3.01 ms, against 22.8 ms on the FMA pipe (painn_message.cu); n = 64, 1024 edges of
// 512 nodes: 55 us against 79. Error against 64 bits in the first case: 4.5e-7, against 7.3e-7.
//
// A block owns a node-aligned, contiguous slice of the CSR and walks it 256 / (n / 32) edges at a time. Roles:
//   * 16 working warps: geometry, radial features -> activation planes in shared memory; per layer each thread adds the
//     partial sums of its channel (64 edges) from tensor memory into registers, then writes bias + SiLU back as the next
//     layer's planes; the last layer goes to shared memory in FP32, is turned into messages (16 edges of a channel per
//     thread) and summed per node in edge order (no atomics; every node written once; the same bits wherever a node's
//     edges fall in a tile).
//   * 2 MMA warps and 1 producer warp (lane 0 of each): six MMAs per 16 KB weight slab; slabs stream through a ring.
// Every wait is bounded: a failed wait is OR-ed into the next block barrier so that all threads leave together, raises
// LD_FLAG_TIMEOUT and leaves NaN in the outputs of the block.
#include "common.cuh"
#include "split_f16.cuh"
#include "split_pack.cuh"
#include "tp_math.h"

namespace {

using namespace sf;

constexpr int SUM_BATCH = 4;                          // nodes whose residuals are in flight together in the per-node sums
constexpr int EPT = 16;                               // edges per thread in the message phase

// MB: blocks of 128 channels; n = 32 MB
template <int MB>
struct Shape {
  static constexpr int N = 128 * MB, n = 32 * MB;
  static constexpr int NE = 256 / MB;                 // edges per tile = N of an MMA
  static constexpr int PANEL = NE * 16 + 16;          // bytes between panels of 8 channels (the 16 spread a warp's stores over the banks)
  static constexpr int PLANE = (N / 8) * PANEL;
  static constexpr int ACT = 2 * PLANE;               // also the FP32 products [N][NE + 1]
  static constexpr int SLOTS = 2 * MB;                // accumulators of NE columns in tensor memory
  // weight slabs in the ring. A warp that waits for a slab has to know that the one before it in the same stage has landed, or
  // the parity it waits for means nothing: with four blocks the stages are even in number, so that both are its own; with
  // fewer, the wait for the accumulators says so.
  static constexpr int STAGES = MB == 4 ? 4 : 5;
  static constexpr int G = WORK_THREADS / n;          // threads per channel in the message phase
  static_assert(N * (NE + 1) * 4 <= ACT, "the products reuse the activation planes");
  static_assert(G * EPT == NE, "the message phase covers the tile");
  static constexpr int GROUPS = WORK_THREADS / N;     // threads per component in the per-node sums
  static constexpr size_t SMEM = (size_t)ACT + STAGES * sf::SLAB_BYTES + 10 * N * 4;
};

struct SplitParams {
  const int* row_ptr; const int* dst; const float* rij;
  int Nt, n_rbf, k0p, radial_kind, seg_nodes;
  float rmax, pi_over_rmax, eps;
  const __half* w[3];      // packed slabs per layer
  const float* b[3];
  const float* scales;     // [3][N] what takes an accumulator back, [2][N] scales of the hidden channels
  const float* actv; const float* x_v; const float* res_a; const float* res_v;
  float* out_a; float* out_v;
  long long* edge_counter;
  int* status;
};

// the two factors of a Gaussian radial feature (radial_feature, kind 1), the envelope once per edge
__device__ __forceinline__ float radial_envelope(float d, float rmax) {
  return 0.5f * (cosf(3.14159265358979323846f * d / rmax) + 1.0f);
}
__device__ __forceinline__ float radial_gaussian(int m, int n, float d, float rmax) {
  const float width = n > 1 ? rmax / (float)(n - 1) : rmax;
  const float u = (d - (float)m * width) / width;
  return expf(-0.5f * u * u);
}

// SiLU with the quotient from the reciprocal instruction (2 ulp; zero below -87.3, where the pair that holds the result resolves
// 2^-79 at best). The exact quotient: 3.29 ms instead of 3.11 (n = 128, 562 k edges), the same distance from 64 bits.
__device__ __forceinline__ float silu_fdiv(float x) { return __fdividef(x, 1.0f + expf(-x)); }

template <int MB>
__global__ void __launch_bounds__(THREADS, 1)
painn_message_split_kernel(const __grid_constant__ SplitParams P) {
  using S = Shape<MB>;
  constexpr int N = S::N, n = S::n, NE = S::NE, SLOTS = S::SLOTS, STAGES = S::STAGES;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar_full[STAGES], bar_empty[STAGES], bar_done[SLOTS], bar_taken[2];
  __shared__ uint32_t tmem_slot;
  __shared__ float s_dir[NE][3];
  __shared__ float s_dist[NE], s_env[NE];
  __shared__ int s_dst[NE], s_src[NE];
  __shared__ int s_rowwin[NE + 1];   // row_ptr[node_lo .. node_lo + NE] of the coming tile
  __shared__ uint32_t s_begin[NE / 32];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* act = smem;                                              // two activation planes
  float* prod = reinterpret_cast<float*>(smem);                           // [N][NE + 1], after the last layer
  unsigned char* ring = smem + S::ACT;
  float* s_bias = reinterpret_cast<float*>(ring + STAGES * sf::SLAB_BYTES);   // [3][N]
  float* s_inv = s_bias + 3 * N;                                          // [3][N]
  float* s_scale = s_inv + 3 * N;                                         // [2][N]
  float* s_carry = s_scale + 2 * N;                                       // [2][N]: sum of the node that goes on, in turn

  for (int i = tid; i < 3 * N; i += THREADS) s_bias[i] = P.b[i / N][i % N];
  for (int i = tid; i < 5 * N; i += THREADS) s_inv[i] = P.scales[i];
  if (tid == 0) {
    for (int s = 0; s < STAGES; s++) { tc::mbar_init(&bar_full[s], 1); tc::mbar_init(&bar_empty[s], 1); }
    for (int s = 0; s < SLOTS; s++) tc::mbar_init(&bar_done[s], 1);      // MMAs of slab q: slot q % SLOTS
    for (int s = 0; s < 2; s++) tc::mbar_init(&bar_taken[s], WORK_WARPS);   // partial sums of a chunk are in registers
    tc::mbar_init_fence();
  }
  if (warp == 0) { tc::tmem_alloc(&tmem_slot, 512); tc::tmem_relinquish(); }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  const int seg_nodes = P.seg_nodes > 0 ? P.seg_nodes : P.Nt;
  int fail = 0;

  if (warp == PROD_WARP) {
    // ===== producer: weight slabs through the ring, independent of the data ====================================
    if (lane == 0) {
      uint32_t loads = 0;
      for (int seg_lo = 0; seg_lo < P.Nt && !fail; seg_lo += seg_nodes) {
        const long long ntiles = block_range(P.row_ptr, seg_lo, min(seg_lo + seg_nodes, P.Nt), NE).ntiles;
        for (long long t = 0; t < ntiles && !fail; t++)
          for (int layer = 0; layer < 3 && !fail; layer++) {
            const int K = layer == 0 ? P.k0p : N;
            const unsigned char* src = reinterpret_cast<const unsigned char*>(P.w[layer]);
            for (int k0 = 0; k0 < K && !fail; k0 += sf::SLAB_K) {
              const uint32_t bytes = 2u * 128u * 2u * (uint32_t)min(sf::SLAB_K, K - k0);
              for (int m = 0; m < MB; m++, loads++, src += bytes) {
                const uint32_t st = loads % STAGES, use = loads / STAGES;
                if (use >= 1 && !tc::mbar_wait(&bar_empty[st], (use - 1) & 1)) { fail = 1; break; }   // MMAs that read it are done
                tc::mbar_expect_tx(&bar_full[st], bytes);
                tc::bulk_g2s(ring + (size_t)st * sf::SLAB_BYTES, src, bytes, &bar_full[st]);
              }
            }
          }
      }
      if (fail) {
        // copies already requested still land in this block's shared memory: give them a bounded chance
        for (uint32_t i = loads > STAGES ? loads - STAGES : 0; i < loads; i++) tc::mbar_wait(&bar_full[i % STAGES], (i / STAGES) & 1);
      }
    }
  } else if (warp >= MMA_WARP) {
    // ===== MMA issue ==============================================================================================
    // the issuing thread runs alone in its warp, so every instruction between two MMAs is exposed: descriptors and ring
    // positions advance by additions, and accumulators are waited for once per chunk of MB slabs
    const uint32_t me = warp - MMA_WARP;
    uint32_t chunks = 0, st = me, full_phase = 0;
    const uint32_t b1 = desc_lo(act, S::PANEL), b2 = desc_lo(act + S::PLANE, S::PANEL);
    const uint32_t a0 = desc_lo(ring, 128 * 16);
    constexpr uint32_t b_step = (2 * S::PANEL) >> 4, st_step = sf::SLAB_BYTES >> 4;
    constexpr uint32_t idesc = sf::idesc_f16(128, NE);
    for (int seg_lo = 0; seg_lo < P.Nt && !fail; seg_lo += seg_nodes) {
      const long long ntiles = block_range(P.row_ptr, seg_lo, min(seg_lo + seg_nodes, P.Nt), NE).ntiles;
      for (long long t = 0; t < ntiles; t++) {
        if (sync_or(fail)) { fail = 1; break; }      // [G] geometry staged
        for (int layer = 0; layer < 3; layer++) {
          if (sync_or(fail)) { fail = 1; break; }    // [X] this layer's activations are written
          if (lane == 0) {
            const int K = layer == 0 ? P.k0p : N;
            uint32_t x1 = b1, x2 = b2;
            for (int k0 = 0; k0 < K && !fail; k0 += sf::SLAB_K, chunks++, x1 += 2 * b_step, x2 += 2 * b_step) {
              const uint32_t ks = K - k0 > 16 ? 2 : 1;
              if (MB == 1 && (chunks & 1) != me) continue;
              // the partial sums that lie in this half of tensor memory have been taken
              if (chunks >= 2 && !tc::mbar_wait(&bar_taken[chunks & 1], ((chunks >> 1) - 1) & 1)) { fail = 1; break; }
              tc::fence_after_sync();
#pragma unroll
              for (int h = 0; h < (MB + 1) / 2; h++) {
                const uint32_t slot = (chunks & 1) * MB + (MB == 1 ? 0 : 2 * h + me);   // slabs are numbered chunk * MB + block
                if (!tc::mbar_wait(&bar_full[st], full_phase)) { fail = 1; break; }
                tc::fence_after_sync();
                sf::slab_mmas(tmem_base + slot * NE, a0 + st * st_step, ks, x1, x2, b_step, idesc);
                tc::mma_commit(&bar_empty[st]);
                tc::mma_commit(&bar_done[slot]);
                st += MMA_WARPS;
                if (st >= STAGES) { st -= STAGES; full_phase ^= 1; }
              }
            }
          }
          fail = __shfl_sync(0xffffffffu, fail, 0);
          if (sync_or(fail)) { fail = 1; break; }    // [A] every partial sum of the layer has been taken
        }
        if (fail) break;
      }
    }
  } else {
    // ===== working warps ============================================================================================
    const int mblk = (warp >> 2) % MB, half = (warp >> 2) / MB, quarter = warp & 3;
    const int o = mblk * 128 + quarter * 32 + lane;   // this thread's channel, and edges [64 half, 64 half + 64)
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + half * 64;
    uint32_t chunks = 0;                              // partial sums taken so far by this thread's channel block
    const int mc = tid % n, mg = tid / n;             // message phase: channel, group of EPT edges
    // per-node sums: row of the products (component sc of channel mc), group
    const int grp = S::GROUPS == 1 ? 0 : tid / N, comp = S::GROUPS == 1 ? tid : tid % N, sc = S::GROUPS == 1 ? mg : comp / n;
    float sum = 0.f;                                  // one group: of node `cur` (more: in s_carry)
    uint32_t tiles = 0;
    long long edges_done = 0;
    // residual of this thread's component, and its result
    auto load = [&](int v) {
      if (sc < 3) return P.res_v != nullptr ? __ldg(P.res_v + ((size_t)v * n + mc) * 3 + sc) : 0.f;
      return P.res_a != nullptr ? __ldg(P.res_a + (size_t)v * n + mc) : 0.f;
    };
    auto store = [&](int v, float val, float r) {
      if (sc < 3) P.out_v[((size_t)v * n + mc) * 3 + sc] = P.res_v != nullptr ? val + r : val;
      else P.out_a[(size_t)v * n + mc] = P.res_a != nullptr ? val + r : val;
    };

    for (int seg_lo = 0; seg_lo < P.Nt && !fail; seg_lo += seg_nodes) {
      const BlockRange br = block_range(P.row_ptr, seg_lo, min(seg_lo + seg_nodes, P.Nt), NE);
      const int n_begin = br.n_begin, n_end = br.n_end;
      int cur = n_begin;          // node that s_carry belongs to
      int node_lo = n_begin;      // source node of the next tile's first edge (or an earlier one)
      sync_workers();             // the previous segment's last readers of s_rowwin are done
      stage_window<NE>(s_rowwin, P.row_ptr, node_lo, max(n_end, n_begin), tid);
      sum = 0.f;
      if (S::GROUPS > 1 && tid < N) s_carry[(tiles & 1) * N + tid] = 0.f;
      sync_workers();

      for (long long e0 = br.e_begin; e0 < br.e_end; e0 += NE) {
        const int cnt = (int)(br.e_end - e0 < NE ? br.e_end - e0 : NE);
        // ---- geometry --------------------------------------------------------------------------------------------
        if (tid < NE) {
          float dx = 0.f, dy = 0.f, dz = 0.f;
          int j = 0, s = -1;
          if (tid < cnt) {
            const long long e = e0 + tid;
            dx = P.rij[e * 3]; dy = P.rij[e * 3 + 1]; dz = P.rij[e * 3 + 2];
            j = P.dst[e];
            s = source_node<NE>(s_rowwin, P.row_ptr, node_lo, n_end, e);
          }
          const float r2 = dx * dx + dy * dy + dz * dz;
          const float inv = 1.0f / sqrtf(P.eps + r2);
          s_dir[tid][0] = dx * inv; s_dir[tid][1] = dy * inv; s_dir[tid][2] = dz * inv;
          const float d = sqrtf(r2);
          s_dist[tid] = d;
          s_env[tid] = P.radial_kind == 1 && d < P.rmax ? radial_envelope(d, P.rmax) : 0.f;
          s_dst[tid] = j;
          s_src[tid] = s;
        }
        if (sync_or(fail)) { fail = 1; break; }                                              // [G]
        // ---- radial features -> planes of the first layer (|feature| <= 1) ----------------------------------------
        for (int i = tid; i < NE * P.k0p; i += WORK_THREADS) {
          const int e = i % NE, k = i / NE;
          float f = 0.f;
          if (e < cnt && k < P.n_rbf)
            f = P.radial_kind == 1 ? radial_gaussian(k, P.n_rbf, s_dist[e], P.rmax) * s_env[e]
                                   : radial_feature(0, k, P.n_rbf, s_dist[e], P.rmax, P.pi_over_rmax);
          __half h1, h2;
          sf::split(f * 16384.f, &h1, &h2);
          unsigned char* at = act + (k >> 3) * S::PANEL + e * 16 + (k & 7) * 2;
          *reinterpret_cast<__half*>(at) = h1;
          *reinterpret_cast<__half*>(at + S::PLANE) = h2;
        }
        tc::fence_async_smem();
        // ---- three layers ------------------------------------------------------------------------------------------
        float acc[64];
        for (int layer = 0; layer < 3; layer++) {
          if (sync_or(fail)) { fail = 1; break; }                                            // [X]
          const int nch = ((layer == 0 ? P.k0p : N) + sf::SLAB_K - 1) / sf::SLAB_K;
#pragma unroll
          for (int i = 0; i < 64; i++) acc[i] = 0.f;
          for (int ch = 0; ch < nch && !fail; ch++, chunks++) {
            const uint32_t slot = (chunks & 1) * MB + mblk;
            if (!warp_wait(&bar_done[slot], (chunks >> 1) & 1)) { fail = 1; break; }
            tc::fence_after_sync();
#pragma unroll
            for (int q = 0; q < 4; q++) {
              float v[16];
              tc::tmem_ld16(taddr + slot * NE + 16 * q, v);
#pragma unroll
              for (int i = 0; i < 16; i++) acc[16 * q + i] += v[i];
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&bar_taken[chunks & 1]);
          }
          if (sync_or(fail)) { fail = 1; break; }                                            // [A] the planes may be overwritten
          const float bias = s_bias[layer * N + o], inv = s_inv[layer * N + o];
          if (layer < 2) {
            const float sx = s_scale[layer * N + o];
            unsigned char* a1 = act + (o >> 3) * S::PANEL + (half * 64) * 16 + (o & 7) * 2;
#pragma unroll
            for (int i = 0; i < 64; i++) {
              __half h1, h2;
              sf::split(silu_fdiv(fmaf(acc[i], inv, bias)) * sx, &h1, &h2);
              *reinterpret_cast<__half*>(a1 + i * 16) = h1;
              *reinterpret_cast<__half*>(a1 + S::PLANE + i * 16) = h2;
            }
            tc::fence_async_smem();
          } else {
            // FP32, over the planes
            float* pr = prod + o * (NE + 1) + half * 64;
#pragma unroll
            for (int i = 0; i < 64; i++) pr[i] = fmaf(acc[i], inv, bias);
          }
        }
        if (fail) break;
        node_lo = s_src[cnt - 1];
        stage_window<NE>(s_rowwin, P.row_ptr, node_lo, n_end, tid);   // for the next tile
        if (S::GROUPS > 1) mark_nodes<NE>(s_begin, s_src, cnt, cur, tid);
        sync_workers();
        // ---- messages of channel mc, edges [EPT mg, EPT mg + EPT), in the place of the products they are made of ------------
        {
          const int r_lo = mg * EPT, r_hi = min(r_lo + EPT, cnt);
          float* pc = prod + mc * (NE + 1);
          for (int eb = r_lo; eb < r_hi; eb += 4) {
            // what four edges take from their neighbours: 28 loads in flight (slots past cnt hold node 0)
            float x[4][3], a[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const size_t j = s_dst[eb + i];
              const float* xp = P.x_v + (j * n + mc) * 3;
              const float* ap = P.actv + j * N + mc;
#pragma unroll
              for (int k = 0; k < 3; k++) x[i][k] = __ldg(xp + k);
#pragma unroll
              for (int k = 0; k < 4; k++) a[i][k] = __ldg(ap + k * n);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const int e = eb + i;
              const float p0 = pc[e] * a[i][0], p1 = pc[n * (NE + 1) + e] * a[i][1], p2 = pc[2 * n * (NE + 1) + e] * a[i][2];
              const float d0 = s_dir[e][0], d1 = s_dir[e][1], d2 = s_dir[e][2];
              pc[e] = x[i][0] * p0 + (x[i][1] * d2 - x[i][2] * d1) * p1 + d0 * p2;
              pc[n * (NE + 1) + e] = x[i][1] * p0 + (x[i][2] * d0 - x[i][0] * d2) * p1 + d1 * p2;
              pc[2 * n * (NE + 1) + e] = x[i][2] * p0 + (x[i][0] * d1 - x[i][1] * d0) * p1 + d2 * p2;
              pc[3 * n * (NE + 1) + e] *= a[i][3];
            }
          }
        }
        sync_workers();
        if constexpr (S::GROUPS == 1)
          node_walk<true>(prod + comp * (NE + 1), s_src, 0, cnt, sum, cur, load, store);
        else
          node_sums<SUM_BATCH, S::GROUPS, NE / S::GROUPS>(prod + comp * (NE + 1), s_src, s_begin, 0, cnt, grp, cur, s_carry + (tiles & 1) * N + comp,
                                                          s_carry + (~tiles & 1) * N + comp, load, store);
        tiles++;
        cur = node_lo;
        sync_workers();   // geometry and planes are rewritten by the next tile
      }
      if (!fail && n_begin < n_end) {
        if (grp == 0) {
          store(cur, S::GROUPS == 1 ? sum : s_carry[(tiles & 1) * N + comp], load(cur));
          empty_nodes<SUM_BATCH>(cur + 1, n_end, load, store);
        }
        edges_done += br.e_end - br.e_begin;
      }
    }
    if (fail && grp == 0) mark_failed(P.row_ptr, P.Nt, seg_nodes, NE, store);
    if (!fail && P.edge_counter != nullptr && tid == 0 && edges_done > 0)
      atomicAdd((unsigned long long*)P.edge_counter, (unsigned long long)edges_done);
  }
  if (fail && lane == 0 && P.status != nullptr) atomicOr(P.status, LD_FLAG_TIMEOUT);
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem_base, 512);
}

template <int MB>
int launch(const SplitParams& P, cudaStream_t st) {
  LD_CUDA_TRY(cudaFuncSetAttribute(painn_message_split_kernel<MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<MB>::SMEM));
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  painn_message_split_kernel<MB><<<sms, THREADS, Shape<MB>::SMEM, st>>>(P);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

}  // namespace

static bool split_form(int n, int n_rbf) { return (n == 32 || n == 64 || n == 128) && n_rbf > 0 && n_rbf <= 4 * n; }

// The packed layers are followed by floats, N = 4n of each: inverse scales of three layers, scales of two hidden ones, their bounds
static long long packed_slabs(int n, int n_rbf) { return 2LL * 4 * n * ((n_rbf + 15) / 16 * 16 + 8 * n); }

// FP16 elements of a packed distance MLP n_rbf -> 4n -> 4n -> 4n (0: these widths have no split form)
extern "C" int ld_painn_split_elems(int n, int n_rbf, long long* elems) {
  if (n <= 0 || n_rbf <= 0) return LD_ERR_SHAPE;
  *elems = split_form(n, n_rbf) ? packed_slabs(n, n_rbf) + 2LL * 7 * 4 * n : 0;
  return LD_OK;
}

// packed: as many FP16 values as ld_painn_split_elems says, 16-byte aligned. Weights [in][out], FP32. scales: not used.
extern "C" int ld_painn_split_pack(const float* W1t, const float* b1, const float* W2t, const float* b2, const float* W3t, int n,
                                   int n_rbf, void* packed, float* scales, void* stream) {
  (void)scales;
  if (!split_form(n, n_rbf)) { ld_set_last_message("painn split pack: n must be 32, 64 or 128, n_rbf at most 4n"); return LD_ERR_UNSUPPORTED; }
  if (b1 == nullptr || b2 == nullptr || ((uintptr_t)packed % 16) != 0) return LD_ERR_SHAPE;
  const int N = 4 * n, k0p = (n_rbf + 15) / 16 * 16;
  cudaStream_t st = (cudaStream_t)stream;
  __half* w = (__half*)packed;
  float* f = (float*)(w + packed_slabs(n, n_rbf));
  float* inv = f; float* scale = f + 3 * N; float* bound = f + 5 * N;
  int rc = split_layer<SPLIT_SILU>(SplitLayer{W1t, n_rbf, N, nullptr, nullptr, nullptr, b1, w, inv, scale, bound, nullptr, nullptr}, st);
  if (rc != LD_OK) return rc;
  w += (size_t)2 * N * k0p;
  rc = split_layer<SPLIT_SILU>(SplitLayer{W2t, N, N, bound, nullptr, scale, b2, w, inv + N, scale + N, bound + N, nullptr, nullptr}, st);
  if (rc != LD_OK) return rc;
  w += (size_t)2 * N * N;
  return split_layer<SPLIT_LAST>(SplitLayer{W3t, N, N, bound + N, nullptr, scale + N, nullptr, w, inv + 2 * N, nullptr, nullptr, nullptr, nullptr}, st);
}

// ld_painn_message_f32 with the distance MLP as packed by ld_painn_split_pack (n = 32, 64 or 128). status_dev receives
// LD_FLAG_TIMEOUT if a bounded wait ran out. scales: not used.
extern "C" int ld_painn_message_f32_split(const int* row_ptr, const int* dst, const float* rij, int Nt, int n, int n_rbf,
                                          int radial_kind, float rmax, float eps, const void* packed, const float* scales,
                                          const float* b1, const float* b2, const float* b3, const float* actv, const float* x_v,
                                          const float* res_a, const float* res_v, float* out_a, float* out_v,
                                          long long* edge_counter, int* status_dev, void* stream) {
  (void)scales;
  if (Nt < 0 || n <= 0 || n_rbf <= 0) return LD_ERR_SHAPE;
  if (!split_form(n, n_rbf)) { ld_set_last_message("painn message (split path): n must be 32, 64 or 128, n_rbf at most 4n"); return LD_ERR_UNSUPPORTED; }
  if (b1 == nullptr || b2 == nullptr || b3 == nullptr) { ld_set_last_message("painn message: biases are required"); return LD_ERR_SHAPE; }
  if (((uintptr_t)packed % 16) != 0) return LD_ERR_SHAPE;
  if (Nt == 0) return LD_OK;
  SplitParams P;
  const int N = 4 * n, k0p = (n_rbf + 15) / 16 * 16;
  P.row_ptr = row_ptr; P.dst = dst; P.rij = rij; P.Nt = Nt; P.n_rbf = n_rbf; P.k0p = k0p; P.radial_kind = radial_kind;
  // blocks walk the node range in segments whose gathered rows (28 n bytes a node) stay in L2
  P.seg_nodes = ld_even_segments(Nt, (40LL << 20) / (28LL * n));
  P.rmax = rmax; P.pi_over_rmax = (float)(3.14159265358979323846 / (double)rmax); P.eps = eps;
  P.w[0] = (const __half*)packed; P.w[1] = P.w[0] + (size_t)2 * N * k0p; P.w[2] = P.w[1] + (size_t)2 * N * N;
  P.b[0] = b1; P.b[1] = b2; P.b[2] = b3; P.actv = actv; P.x_v = x_v; P.res_a = res_a; P.res_v = res_v;
  P.scales = (const float*)(P.w[0] + packed_slabs(n, n_rbf));
  P.out_a = out_a; P.out_v = out_v; P.edge_counter = edge_counter; P.status = status_dev;
  if (n == 128) return launch<4>(P, (cudaStream_t)stream);
  if (n == 64) return launch<2>(P, (cudaStream_t)stream);
  return launch<1>(P, (cudaStream_t)stream);
}
