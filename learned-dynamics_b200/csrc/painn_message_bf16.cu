// PaiNN message step on the tensor cores in BF16 (tolerance 2e-2 relative), widths 32, 64 and 128: the computation of
// painn_message_tc.cu (Message.forward, archs/meanflow_painn8.py:77-100) in the transposed form of painn_message_split.cu,
//   D[channel][edge] = W[channel][k] * X[edge][k].
// Weights are the M operand and stream through a ring of four 16 KB slabs (128 channels x K = 64), a tile of 128 edges is the N
// operand and stays in shared memory. Against edges as the M operand (painn_message_tc.cu: two 32 KB slabs, MMAs that wait for
// them) the ring holds more and smaller slabs, a thread owns one channel, so that an epilogue needs one bias and the messages
// of a channel are formed from coalesced FP32 rows, and the half of the channels that is complete first goes through its
// activation while the other half is multiplied.
// n = 128, 8 radial functions, 2.25 M edges: 3.75 ms, against 4.52 ms (+ 10 us of packing).
//
// A block owns a node-aligned, contiguous slice of the CSR. Roles: 16 working warps, 2 MMA warps (of every pair of channel
// blocks one each), 1 producer warp. Every wait is bounded: a failed wait is OR-ed into the next block barrier so that all
// threads leave together, raises LD_FLAG_TIMEOUT and leaves NaN in the outputs of the block.
#include "common.cuh"
#include "split_f16.cuh"
#include "tp_math.h"

namespace {
using namespace sf;

constexpr int NE = 128, PANEL = NE * 16 + 16;   // edges per tile; bytes between panels of 8 channels
constexpr int KSLAB = 64;                       // K of a weight slab
// weight slabs in the ring, even in number: a warp that waits for a slab has to know that the one before it in the same stage
// has landed, or the parity it waits for means nothing, and with two warps in turn both are then its own
constexpr int RING = 4;

constexpr int SUM_BATCH = 4;                          // nodes whose residuals are in flight together in the per-node sums

template <int MB>
struct Shape {
  static constexpr int N = 128 * MB, n = 32 * MB;
  static constexpr int EW = 32 * MB;                       // edges per thread in the epilogues
  static constexpr int EP = MB == 4 ? 64 : NE;             // edges per pass of the message phase
  static constexpr int G = WORK_THREADS / n, EPT = EP / G; // threads per channel and edges per thread there
  static constexpr int FRONT = (N / 8) * PANEL > N * (EP + 1) * 4 ? (N / 8) * PANEL : N * (EP + 1) * 4;
  static constexpr int GROUPS = WORK_THREADS / N;          // threads per component in the per-node sums
  static constexpr size_t SMEM = (size_t)FRONT + RING * SLAB_BYTES + 2 * N * 4;
};

struct Bf16Params {
  const int* row_ptr; const int* dst; const float* rij;
  int Nt, n_rbf, k0p, radial_kind, seg_nodes;
  float rmax, pi_over_rmax, eps;
  const __nv_bfloat16* w[3];
  const float* b[3];
  const float* actv; const float* x_v; const float* res_a; const float* res_v;
  float* out_a; float* out_v;
  long long* edge_counter;
  int* status;
};

template <int MB>
__global__ void __launch_bounds__(THREADS, 1)
painn_message_bf16_kernel(const __grid_constant__ Bf16Params P) {
  using S = Shape<MB>;
  constexpr int N = S::N, n = S::n, EW = S::EW, EP = S::EP;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar_full[RING], bar_empty[RING], bar_done[MB];
  __shared__ uint32_t tmem_slot;
  __shared__ float s_dir[NE][3];
  __shared__ float s_dist[NE], s_env[NE];
  __shared__ int s_dst[NE], s_src[NE], s_rowwin[NE + 1];
  __shared__ uint32_t s_begin[NE / 32];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* act = smem;                           // activations [N/8 panels][NE][8] BF16
  float* prod = reinterpret_cast<float*>(smem);        // [N][EP + 1], after the last layer
  unsigned char* ring = smem + S::FRONT;
  float* s_carry = reinterpret_cast<float*>(ring + RING * SLAB_BYTES);   // [2][N]: sum of the node that goes on, in turn

  if (tid == 0) {
    for (int s = 0; s < RING; s++) { tc::mbar_init(&bar_full[s], 1); tc::mbar_init(&bar_empty[s], 1); }
    for (int m = 0; m < MB; m++) tc::mbar_init(&bar_done[m], 1);
    tc::mbar_init_fence();
  }
  if (warp == 0) { tc::tmem_alloc(&tmem_slot, N); tc::tmem_relinquish(); }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  const int seg_nodes = P.seg_nodes > 0 ? P.seg_nodes : P.Nt;
  int fail = 0;
  // slabs of a layer, in the order they are streamed: for each pair of channel blocks all K, the two blocks in turn
  constexpr int PAIRS = (MB + 1) / 2, PB = MB == 1 ? 1 : 2;

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
            for (int pr = 0; pr < PAIRS && !fail; pr++)
              for (int k0 = 0; k0 < K && !fail; k0 += KSLAB) {
                const uint32_t bytes = 128u * 2u * (uint32_t)min(KSLAB, K - k0);
                for (int m = 0; m < PB; m++, loads++, src += bytes) {
                  const uint32_t st = loads % RING, use = loads / RING;
                  if (use >= 1 && !tc::mbar_wait(&bar_empty[st], (use - 1) & 1)) { fail = 1; break; }   // MMAs that read it are done
                  tc::mbar_expect_tx(&bar_full[st], bytes);
                  tc::bulk_g2s(ring + (size_t)st * SLAB_BYTES, src, bytes, &bar_full[st]);
                }
              }
          }
      }
      if (fail) {
        // copies already requested still land in this block's shared memory: give them a bounded chance
        for (uint32_t i = loads > RING ? loads - RING : 0; i < loads; i++) tc::mbar_wait(&bar_full[i % RING], (i / RING) & 1);
      }
    }
  } else if (warp >= MMA_WARP) {
    // ===== MMA issue: this warp's block of every pair ==============================================================
    const uint32_t me = warp - MMA_WARP;
    uint32_t st = me, full_phase = 0;
    const uint32_t b0 = desc_lo(act, PANEL), a0 = desc_lo(ring, 128 * 16);
    constexpr uint32_t b_step = (2 * PANEL) >> 4, a_step = (2 * 128 * 16) >> 4, st_step = SLAB_BYTES >> 4;
    constexpr uint32_t idesc = tc::idesc_bf16(128, NE);
    for (int seg_lo = 0; seg_lo < P.Nt && !fail; seg_lo += seg_nodes) {
      const long long ntiles = block_range(P.row_ptr, seg_lo, min(seg_lo + seg_nodes, P.Nt), NE).ntiles;
      for (long long t = 0; t < ntiles && !fail; t++) {
        for (int layer = 0; layer < 3; layer++) {
          if (sync_or(fail)) { fail = 1; break; }    // [X] this layer's activations are written, its accumulators are free
          if (lane == 0 && me < PB) {
            tc::fence_after_sync();
            const int K = layer == 0 ? P.k0p : N;
            for (int pr = 0; pr < PAIRS && !fail; pr++) {
              const uint32_t m = 2 * pr + me, d = tmem_base + m * NE;
              uint32_t x = b0, accumulate = 0u;
              for (int k0 = 0; k0 < K; k0 += KSLAB) {
                if (!tc::mbar_wait(&bar_full[st], full_phase)) { fail = 1; break; }
                tc::fence_after_sync();
                const int ks = min(KSLAB, K - k0) / 16;
                uint32_t a = a0 + st * st_step;
                for (int k = 0; k < ks; k++, a += a_step, x += b_step) {
                  mma_f16(d, a, x, idesc, accumulate);
                  accumulate = 1u;
                }
                tc::mma_commit(&bar_empty[st]);
                st += PB;
                if (st >= RING) { st -= RING; full_phase ^= 1; }
              }
              if (!fail) tc::mma_commit(&bar_done[m]);
            }
          }
          fail = __shfl_sync(0xffffffffu, fail, 0);
          if (sync_or(fail)) { fail = 1; break; }    // [A] every block of the layer is complete
        }
      }
    }
  } else {
    // ===== working warps ============================================================================================
    const int mblk = (warp >> 2) % MB, part = (warp >> 2) / MB, quarter = warp & 3;
    const int o = mblk * 128 + quarter * 32 + lane;   // this thread's channel, and edges [EW part, EW part + EW)
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + mblk * NE + part * EW;
    const float bias1 = P.b[0][o], bias2 = P.b[1][o], bias3 = P.b[2][o];
    const int mc = tid % n, mg = tid / n;             // message phase: channel, group of EPT edges
    // per-node sums: row of the products (component sc of channel mc), group
    const int grp = S::GROUPS == 1 ? 0 : tid / N, comp = S::GROUPS == 1 ? tid : tid % N, sc = S::GROUPS == 1 ? mg : comp / n;
    float sum = 0.f;                                  // one group: of node `cur` (more: in s_carry)
    uint32_t layers = 0;                              // layers completed: phase of bar_done
    uint32_t passes = 0;
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
      if (S::GROUPS > 1 && tid < N) s_carry[(passes & 1) * N + tid] = 0.f;
      sync_workers();

      for (long long e0 = br.e_begin; e0 < br.e_end; e0 += NE) {
        const int cnt = (int)(br.e_end - e0 < NE ? br.e_end - e0 : NE);
        // ---- geometry ----------------------------------------------------------------------------------------------
        if (tid < NE) {
          float dx = 0.f, dy = 0.f, dz = 0.f;
          int j = 0, s = -1;
          if (tid < cnt) {
            const long long e = e0 + tid;
            dx = P.rij[e * 3]; dy = P.rij[e * 3 + 1]; dz = P.rij[e * 3 + 2];
            j = P.dst[e];
            s = source_node<NE>(s_rowwin, P.row_ptr, node_lo, n_end, e);
          }
          const float r2 = dx * dx + dy * dy + dz * dz, inv = rsqrtf(P.eps + r2), d = sqrtf(r2);
          s_dir[tid][0] = dx * inv; s_dir[tid][1] = dy * inv; s_dir[tid][2] = dz * inv;
          s_dist[tid] = d;
          s_env[tid] = d < P.rmax ? 0.5f * (__cosf(P.pi_over_rmax * d) + 1.0f) : 0.f;
          s_dst[tid] = j;
          s_src[tid] = s;
        }
        sync_workers();
        // ---- radial features (rounded to BF16: fast exponentials) ----------------------------------------------------
        {
          const float width = P.n_rbf > 1 ? P.rmax / (float)(P.n_rbf - 1) : P.rmax, inv_w = 1.0f / width;
          for (int i = tid; i < NE * (P.k0p / 2); i += WORK_THREADS) {
            const int e = i % NE, k = (i / NE) * 2;
            const float d = s_dist[e];
            float f[2] = {0.f, 0.f};
#pragma unroll
            for (int q = 0; q < 2; q++)
              if (e < cnt && k + q < P.n_rbf) {
                if (P.radial_kind == 1) {
                  const float u = (d - (float)(k + q) * width) * inv_w;
                  f[q] = __expf(-0.5f * u * u) * s_env[e];
                } else {
                  f[q] = radial_feature(P.radial_kind, k + q, P.n_rbf, d, P.rmax, P.pi_over_rmax);
                }
              }
            *reinterpret_cast<uint32_t*>(act + (k >> 3) * PANEL + e * 16 + (k & 7) * 2) = tc::pack_bf16x2(f[0], f[1]);
          }
        }
        tc::fence_async_smem();
        // ---- two hidden layers ------------------------------------------------------------------------------------------
#pragma unroll 1
        for (int layer = 0; layer < 2; layer++, layers++) {
          tc::fence_before_sync();
          if (sync_or(fail)) { fail = 1; break; }                                            // [X]
          // this block of channels as soon as it is complete; the planes are overwritten when all are
          if (!warp_wait(&bar_done[mblk], layers & 1)) fail = 1;
          tc::fence_after_sync();
          const float bias = layer == 0 ? bias1 : bias2;
          unsigned char* at = act + (o >> 3) * PANEL + (part * EW) * 16 + (o & 7) * 2;
          // the first half of this thread's edges before the planes are free (held in registers), the second half after
          uint32_t h[EW / 4];
#pragma unroll
          for (int q = 0; q < EW / 16; q++) {
            float v[8];
            tc::tmem_ld8(taddr + 8 * q, v);
#pragma unroll
            for (int i = 0; i < 4; i++) h[4 * q + i] = tc::pack_bf16x2(tc::silu_fast(v[2 * i] + bias), tc::silu_fast(v[2 * i + 1] + bias));
          }
          if (sync_or(fail)) { fail = 1; break; }                                            // [A]
#pragma unroll
          for (int i = 0; i < EW / 4; i++) {
            *reinterpret_cast<unsigned short*>(at + (2 * i) * 16) = (unsigned short)h[i];
            *reinterpret_cast<unsigned short*>(at + (2 * i + 1) * 16) = (unsigned short)(h[i] >> 16);
          }
#pragma unroll
          for (int q = 0; q < EW / 32; q++) {
            float v[16];
            tc::tmem_ld16(taddr + EW / 2 + 16 * q, v);
#pragma unroll
            for (int i = 0; i < 8; i++) {
              const uint32_t w = tc::pack_bf16x2(tc::silu_fast(v[2 * i] + bias), tc::silu_fast(v[2 * i + 1] + bias));
              *reinterpret_cast<unsigned short*>(at + (EW / 2 + 16 * q + 2 * i) * 16) = (unsigned short)w;
              *reinterpret_cast<unsigned short*>(at + (EW / 2 + 16 * q + 2 * i + 1) * 16) = (unsigned short)(w >> 16);
            }
          }
          tc::fence_async_smem();
        }
        if (fail) break;
        tc::fence_before_sync();
        if (sync_or(fail)) { fail = 1; break; }                                              // [X]
        if (!warp_wait(&bar_done[mblk], layers & 1)) fail = 1;
        layers++;
        if (sync_or(fail)) { fail = 1; break; }                                              // [A]
        tc::fence_after_sync();
        node_lo = s_src[cnt - 1];
        stage_window<NE>(s_rowwin, P.row_ptr, node_lo, n_end, tid);   // for the next tile
        if (S::GROUPS > 1) mark_nodes<NE>(s_begin, s_src, cnt, cur, tid);
        // ---- EP edges at a time: last layer to shared memory in FP32, messages, per-node sums -----------------------------
        for (int p0 = 0; p0 < cnt; p0 += EP) {
          // columns of the pass that this thread holds (MB = 4: the pass' half of its edges, else all of them)
          constexpr int COLS = MB == 4 ? 64 : EW;
          float* pr = prod + o * (EP + 1) + part * EW;
#pragma unroll
          for (int q = 0; q < COLS / 16; q++) {
            float v[16];
            tc::tmem_ld16(taddr + (MB == 4 ? p0 : 0) + 16 * q, v);
#pragma unroll
            for (int i = 0; i < 16; i++) pr[16 * q + i] = v[i] + bias3;
          }
          sync_workers();
          {
            // messages of channel mc in the place of the products they are made of; 28 loads in flight
            const int r_lo = mg * S::EPT, r_hi = min(r_lo + S::EPT, cnt - p0);
            float* pc = prod + mc * (EP + 1);
            for (int eb = r_lo; eb < r_hi; eb += 4) {
              float x[4][3], a[4][4];
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const size_t j = s_dst[p0 + eb + i];   // slots past cnt hold node 0
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
                const float q0 = pc[e] * a[i][0], q1 = pc[n * (EP + 1) + e] * a[i][1], q2 = pc[2 * n * (EP + 1) + e] * a[i][2];
                const float d0 = s_dir[p0 + e][0], d1 = s_dir[p0 + e][1], d2 = s_dir[p0 + e][2];
                pc[e] = x[i][0] * q0 + (x[i][1] * d2 - x[i][2] * d1) * q1 + d0 * q2;
                pc[n * (EP + 1) + e] = x[i][1] * q0 + (x[i][2] * d0 - x[i][0] * d2) * q1 + d1 * q2;
                pc[2 * n * (EP + 1) + e] = x[i][2] * q0 + (x[i][0] * d1 - x[i][1] * d0) * q1 + d2 * q2;
                pc[3 * n * (EP + 1) + e] *= a[i][3];
              }
            }
          }
          sync_workers();
          const int live = min(EP, cnt - p0);
          if constexpr (S::GROUPS == 1) {
            node_walk<false>(prod + comp * (EP + 1), s_src, p0, live, sum, cur, load, store);
          } else {
            node_sums<SUM_BATCH, S::GROUPS, EP / S::GROUPS>(prod + comp * (EP + 1), s_src, s_begin, p0, live, grp, cur,
                                                            s_carry + (passes & 1) * N + comp, s_carry + (~passes & 1) * N + comp, load, store);
            cur = s_src[p0 + live - 1];
          }
          passes++;
          sync_workers();   // the products (and geometry and planes) are rewritten
        }
      }
      if (!fail && n_begin < n_end) {
        if (grp == 0) {
          store(cur, S::GROUPS == 1 ? sum : s_carry[(passes & 1) * N + comp], load(cur));
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
  if (warp == 0) tc::tmem_dealloc(tmem_base, N);
}

// W [N][K] (element strides sw0, sw1) -> slabs [pair of blocks][K chunk of 64][block of the pair][K/8][128][8], K padded with
// zeros to a multiple of 16
__global__ void slab_pack_kernel(const float* __restrict__ W, long long sw0, long long sw1, int N, int K, __nv_bfloat16* __restrict__ out) {
  const int kp = (K + 15) / 16 * 16;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= kp * N) return;
  const int o = idx % N, k = idx / N, m = o / 128, pb = N == 128 ? 1 : 2;
  const int ch = k / KSLAB, kw = min(KSLAB, kp - ch * KSLAB), kl = k - ch * KSLAB;
  const float v = k < K ? W[(long long)o * sw0 + (long long)k * sw1] : 0.f;
  __nv_bfloat16* pair = out + (size_t)(m / 2) * 2 * kp * 128;
  out = pair + ((size_t)ch * KSLAB * pb + (size_t)(m % 2) * kw) * 128;
  out[(size_t)(kl / 8) * 128 * 8 + (o % 128) * 8 + kl % 8] = __float2bfloat16_rn(v);
}

template <int MB>
int launch(const Bf16Params& P, cudaStream_t st) {
  LD_CUDA_TRY(cudaFuncSetAttribute(painn_message_bf16_kernel<MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<MB>::SMEM));
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  painn_message_bf16_kernel<MB><<<sms, THREADS, Shape<MB>::SMEM, st>>>(P);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

}  // namespace

// N outputs (128, 256 or 512), K inputs: N * (K rounded up to 16) BF16 values, 16-byte aligned
extern "C" int ld_painn_pack_slabs_bf16(const float* W, long long sw0, long long sw1, int N, int K, void* out, void* stream) {
  if (K <= 0 || (N != 128 && N != 256 && N != 512)) { ld_set_last_message("painn slabs: 128, 256 or 512 outputs"); return LD_ERR_UNSUPPORTED; }
  const int kp = (K + 15) / 16 * 16;
  slab_pack_kernel<<<ld_cdiv((long long)kp * N, 256), 256, 0, (cudaStream_t)stream>>>(W, sw0, sw1, N, K, (__nv_bfloat16*)out);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

// ld_painn_message_bf16_tc for n = 32, 64 or 128 with the three weights packed by ld_painn_pack_slabs_bf16; the neighbours'
// features are read in FP32.
extern "C" int ld_painn_message_bf16_slabs(const int* row_ptr, const int* dst, const float* rij, int Nt, int n, int n_rbf, int radial_kind,
                                           float rmax, float eps, const void* w1s, const float* b1, const void* w2s, const float* b2,
                                           const void* w3s, const float* b3, const float* actv, const float* x_v, const float* res_a,
                                           const float* res_v, float* out_a, float* out_v, long long* edge_counter, int* status_dev,
                                           void* stream) {
  if (Nt < 0 || n <= 0 || n_rbf <= 0) return LD_ERR_SHAPE;
  if ((n != 32 && n != 64 && n != 128) || n_rbf > 4 * n) { ld_set_last_message("painn message (slab path): n must be 32, 64 or 128, n_rbf at most 4n"); return LD_ERR_UNSUPPORTED; }
  if (b1 == nullptr || b2 == nullptr || b3 == nullptr) { ld_set_last_message("painn message: biases are required"); return LD_ERR_SHAPE; }
  if ((((uintptr_t)w1s | (uintptr_t)w2s | (uintptr_t)w3s) % 16) != 0) return LD_ERR_SHAPE;
  if (Nt == 0) return LD_OK;
  Bf16Params P;
  P.row_ptr = row_ptr; P.dst = dst; P.rij = rij; P.Nt = Nt; P.n_rbf = n_rbf; P.k0p = (n_rbf + 15) / 16 * 16; P.radial_kind = radial_kind;
  // blocks walk the node range in segments whose gathered rows (28 n bytes a node) stay in L2
  P.seg_nodes = ld_even_segments(Nt, (40LL << 20) / (28LL * n));
  P.rmax = rmax; P.pi_over_rmax = (float)(3.14159265358979323846 / (double)rmax); P.eps = eps;
  P.w[0] = (const __nv_bfloat16*)w1s; P.w[1] = (const __nv_bfloat16*)w2s; P.w[2] = (const __nv_bfloat16*)w3s;
  P.b[0] = b1; P.b[1] = b2; P.b[2] = b3; P.actv = actv; P.x_v = x_v; P.res_a = res_a; P.res_v = res_v;
  P.out_a = out_a; P.out_v = out_v; P.edge_counter = edge_counter; P.status = status_dev;
  if (n == 128) return launch<4>(P, (cudaStream_t)stream);
  if (n == 64) return launch<2>(P, (cudaStream_t)stream);
  return launch<1>(P, (cudaStream_t)stream);
}
