// Scalar output of the l<=2 message layer at FP32 accuracy with the per-edge linear maps on the tensor cores: what
// bee_scalar_kernel of bee_messages.cu computes (Messages.forward of archs/diffuser_atoms15.py:227-253, scalar channel),
// with operands split into two FP16 values (split_f16.cuh).
//
//   y   = the three scalar products of every channel                    K = 3 C
//   psi = Y y ;  h1 = leaky(W1 psi + b1) ;  h2 = leaky(W2 h1 + b2)      widths A, 2 A, 2 A
//   out = psi + Wd psi + W3 h2 + b3, summed per source node, times `scale`
//
// What bounds it: the phases of a tile, which follow one another (the tensor pipe is active 15 % of the time), and within the
// products the shared-memory port (48 cycles per 128 x 64 x 16 MMA, and the weight slabs that arrive through it).
// C = A = 128, 176 k edges: 0.71 ms, against 7.38 ms on the FMA pipe.
//
// A block owns a node-aligned slice of the CSR and walks it 64 edges at a time; roles as in painn_message_split.cu. The
// neighbours' rows are read component-major, [node][13][C], so that a warp's loads are 128 consecutive bytes. The sizes of
// the products are not bounded beforehand: the scale of an edge's operands comes from its largest product, those of the
// later layers from that and from each channel's bounds (split_pack.cuh). Every step of the pipeline is two weight slabs: the
// two blocks of 128 channels of a hidden layer, or two chunks of K of a layer with one block.
#include "common.cuh"
#include "split_f16.cuh"
#include "split_pack.cuh"
#include "bee_edge.cuh"

namespace {
using namespace sf;

constexpr int NE = 64, PANEL = NE * 16 + 16, EPT = 16;
// weight slabs in the ring. A warp that waits for a slab has to know that the one before it in the same stage has landed, or
// the parity it waits for means nothing: five stages back is the other warp's slab, of two or three steps before, and this warp
// has waited for the accumulators of the step two before to be taken.
constexpr int STAGES = 5;

// floats behind the packed weights: per channel what takes an accumulator back (inv_*), the scale of its stored value
// (sc_*), its bound (p_*, q_*); the extremes of q / p of the hidden layers
template <typename T>
struct BeeScales {
  T *inv_y, *inv_3, *inv_d, *sc_psi, *inv_1, *sc_1, *inv_2, *sc_2;   // [A] x 4, [2 A] x 4: read by the edge kernel
  T *ratio_1, *ratio_2;                                              // [2], [2]
  T *p_psi, *p_1, *q_1, *p_2, *q_2;
  __host__ __device__ BeeScales(T* f, int A) {
    inv_y = f; inv_3 = f + A; inv_d = f + 2 * A; sc_psi = f + 3 * A;
    inv_1 = f + 4 * A; sc_1 = f + 6 * A; inv_2 = f + 8 * A; sc_2 = f + 10 * A;
    ratio_1 = f + 12 * A; ratio_2 = ratio_1 + 2;
    p_psi = ratio_1 + 4; p_1 = p_psi + A; q_1 = p_1 + 2 * A; p_2 = q_1 + 2 * A; q_2 = p_2 + 2 * A;
  }
};
constexpr int READ_PER_A = 12, FLOATS_PER_A = 21, FLOATS_EXTRA = 4;

// C product channels, A scalar channels
template <int C, int A>
struct BeeShape {
  static constexpr int HB = 2 * A / 128;                 // blocks of 128 channels of a hidden layer
  static constexpr int YPLANE = (3 * C / 8) * PANEL, HPLANE = (2 * A / 8) * PANEL, PPLANE = (A / 8) * PANEL;
  static constexpr int FRONT = YPLANE > HPLANE ? 2 * YPLANE : 2 * HPLANE;   // products, then hidden layers
  static constexpr size_t SMEM = (size_t)FRONT + 2 * PPLANE + STAGES * SLAB_BYTES + (READ_PER_A + 2) * A * 4;
  // slabs (K = 32 each) of the four matrix products, in the order they are streamed
  static constexpr int SY = 3 * C / 32, S1 = A / 32 * HB, S2 = 2 * A / 32 * HB, S3 = 2 * A / 32, SD = A / 32;
  static constexpr int SLABS = SY + S1 + S2 + S3 + SD;
  static_assert(A * (NE + 1) * 4 <= FRONT, "the edges' results take the place of the planes");
  static_assert(SY % 2 == 0 && S1 % 2 == 0 && S2 % 2 == 0 && S3 % 2 == 0 && SD % 2 == 0, "a step is two slabs");
};

struct BeeSplitParams {
  const int* row_ptr; const int* dst; const float* rij;
  int Nt, seg_nodes;
  float r0, scale;
  const float* rows;                       // [Nt][13][C]
  const float* enc_w; const float* enc_b; const float* jacobi;
  const __half* w;                         // packed slabs of Y, W1, W2, W3, Wd
  const float* scales;                     // BeeScales
  const float* b1; const float* b2; const float* b3;
  float* out_a;
  int* status;
};

__device__ __forceinline__ float leaky(float v) { return v > 0.f ? v : 0.1f * v; }

// of one edge: scale of its products, and the powers of two above the sizes of the products and the hidden layers (and one
// over them); a channel's scale stands beside them
struct EdgeScales { float y, up_y, down_y, up_1, down_1, up_2, down_2; };

// above (by p + q) / (p + q) for every q / p in [lo, hi]: falls with q / p when by >= 1, else rises
__device__ __forceinline__ float edge_size(float by, float lo, float hi) {
  const float r = by >= 1.f ? lo : hi;
  return isinf(r) ? 1.f : (by + r) / (1.f + r) * 1.001f;
}

template <int C, int A>
__global__ void __launch_bounds__(THREADS, 1)
bee_scalar_split_kernel(const __grid_constant__ BeeSplitParams P) {
  using S = BeeShape<C, A>;
  constexpr int HB = S::HB;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar_full[STAGES], bar_empty[STAGES], bar_done[4], bar_taken[2];
  __shared__ uint32_t tmem_slot;
  __shared__ EdgeGeom s_geom[NE];
  __shared__ EdgeScales s_sc[NE];
  __shared__ unsigned s_max[NE];
  __shared__ int s_dst[NE], s_src[NE], s_rowwin[NE + 1];
  __shared__ uint32_t s_begin[NE / 32];
  __shared__ float s_jac[72];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* front = smem;                       // planes of the products, later of the hidden layers
  float* vals = reinterpret_cast<float*>(smem);      // [A][NE + 1], after the last layer
  unsigned char* psi_pl = smem + S::FRONT;           // planes of psi
  unsigned char* ring = psi_pl + 2 * S::PPLANE;
  float* s_scales = reinterpret_cast<float*>(ring + STAGES * SLAB_BYTES);
  const BeeScales<const float> chan(s_scales, A);
  float* s_carry = s_scales + READ_PER_A * A;   // [2][A]: sum of the node that goes on, in turn

  if (tid < 8) ld_poly8_to_chebyshev(P.jacobi + tid * 9, s_jac + tid * 9);   // Chebyshev form of the radial polynomials
  for (int i = tid; i < READ_PER_A * A; i += THREADS) s_scales[i] = P.scales[i];
  if (tid == 0) {
    for (int s = 0; s < STAGES; s++) { tc::mbar_init(&bar_full[s], 1); tc::mbar_init(&bar_empty[s], 1); }
    for (int s = 0; s < 4; s++) tc::mbar_init(&bar_done[s], 1);            // MMAs of slab q: accumulator q % 4
    for (int s = 0; s < 2; s++) tc::mbar_init(&bar_taken[s], WORK_WARPS);  // partial sums of a step are in registers
    tc::mbar_init_fence();
  }
  if (warp == 0) { tc::tmem_alloc(&tmem_slot, 256); tc::tmem_relinquish(); }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  const int seg_nodes = P.seg_nodes > 0 ? P.seg_nodes : P.Nt;
  int fail = 0;

  if (warp == PROD_WARP) {
    // ===== producer: weight slabs through the ring =============================================================
    if (lane == 0) {
      uint32_t loads = 0;
      for (int seg_lo = 0; seg_lo < P.Nt && !fail; seg_lo += seg_nodes) {
        const long long ntiles = block_range(P.row_ptr, seg_lo, min(seg_lo + seg_nodes, P.Nt), NE).ntiles;
        for (long long t = 0; t < ntiles && !fail; t++) {
          const unsigned char* src = reinterpret_cast<const unsigned char*>(P.w);
          for (int q = 0; q < S::SLABS; q++, loads++, src += SLAB_BYTES) {
            const uint32_t st = loads % STAGES, use = loads / STAGES;
            if (use >= 1 && !tc::mbar_wait(&bar_empty[st], (use - 1) & 1)) { fail = 1; break; }   // MMAs that read it are done
            tc::mbar_expect_tx(&bar_full[st], SLAB_BYTES);
            tc::bulk_g2s(ring + (size_t)st * SLAB_BYTES, src, SLAB_BYTES, &bar_full[st]);
          }
        }
      }
      if (fail) {
        // copies already requested still land in this block's shared memory: give them a bounded chance
        for (uint32_t i = loads > STAGES ? loads - STAGES : 0; i < loads; i++) tc::mbar_wait(&bar_full[i % STAGES], (i / STAGES) & 1);
      }
    }
  } else if (warp >= MMA_WARP) {
    // ===== MMA issue: of every step, slab `me` ====================================================================
    const uint32_t me = warp - MMA_WARP;
    uint32_t steps = 0, st = me, full_phase = 0;
    const uint32_t a0 = desc_lo(ring, 128 * 16);
    constexpr uint32_t b_step = (2 * PANEL) >> 4, b_chunk = 2 * b_step, st_step = SLAB_BYTES >> 4;
    constexpr uint32_t idesc = idesc_f16(128, NE);
    // nslabs slabs whose activations start at x (planes `plane` bytes apart); blocks: 2 when a step is two channel blocks
    auto product = [&](const unsigned char* x, int plane, int nslabs, int blocks) {
      if (lane != 0) return;
      uint32_t x1 = desc_lo(x, PANEL), x2 = desc_lo(x + plane, PANEL);
      if (blocks == 1) { x1 += me * b_chunk; x2 += me * b_chunk; }
      const uint32_t advance = blocks == 1 ? 2 * b_chunk : b_chunk;
      for (int q = 0; q < nslabs && !fail; q += 2, steps++, x1 += advance, x2 += advance) {
        if (steps >= 2 && !tc::mbar_wait(&bar_taken[steps & 1], ((steps >> 1) - 1) & 1)) { fail = 1; break; }
        tc::fence_after_sync();
        if (!tc::mbar_wait(&bar_full[st], full_phase)) { fail = 1; break; }
        tc::fence_after_sync();
        const uint32_t slot = (steps & 1) * 2 + me;
        slab_mmas(tmem_base + slot * NE, a0 + st * st_step, 2, x1, x2, b_step, idesc);
        tc::mma_commit(&bar_empty[st]);
        tc::mma_commit(&bar_done[slot]);
        st += MMA_WARPS;
        if (st >= STAGES) { st -= STAGES; full_phase ^= 1; }
      }
    };
    for (int seg_lo = 0; seg_lo < P.Nt && !fail; seg_lo += seg_nodes) {
      const long long ntiles = block_range(P.row_ptr, seg_lo, min(seg_lo + seg_nodes, P.Nt), NE).ntiles;
      for (long long t = 0; t < ntiles && !fail; t++) {
        for (int layer = 0; layer < 4; layer++) {
          if (sync_or(fail)) { fail = 1; break; }    // [X] this layer's activations are written
          if (layer == 0) product(front, S::YPLANE, S::SY, 1);
          else if (layer == 1) product(psi_pl, S::PPLANE, S::S1, HB);
          else if (layer == 2) product(front, S::HPLANE, S::S2, HB);
          else { product(front, S::HPLANE, S::S3, 1); product(psi_pl, S::PPLANE, S::SD, 1); }
          fail = __shfl_sync(0xffffffffu, fail, 0);
          if (sync_or(fail)) { fail = 1; break; }    // [A] every partial sum of the layer has been taken
        }
      }
    }
  } else {
    // ===== working warps ============================================================================================
    const int quarter = warp & 3, grp = warp >> 2;
    const uint32_t tlane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    // layers with one channel block: channel o1, edges [16 grp, 16 grp + 16); hidden layers: channel oh, EH edges from eh
    const int o1 = quarter * 32 + lane, e1 = grp * EPT;
    constexpr int EH = HB == 2 ? 32 : 16;
    const int hblk = HB == 2 ? (grp & 1) : 0, oh = hblk * 128 + quarter * 32 + lane, eh = HB == 2 ? (grp >> 1) * 32 : grp * 16;
    const bool live = o1 < A;                         // A = 64: the upper half of the block is padding
    const float b1 = P.b1[oh], b2 = P.b2[oh], b3 = live ? P.b3[o1] : 0.f;
    // product phase: channel pc, EPP edges from pe
    constexpr int PG = WORK_THREADS / C, EPP = NE / PG;
    const int pc = tid % C, pe = (tid / C) * EPP;
    float w8[8];
#pragma unroll
    for (int m = 0; m < 8; m++) w8[m] = P.enc_w[pc * 8 + m];
    const float wb = P.enc_b[pc];
    uint32_t steps = 0, tiles = 0;
    constexpr int GROUPS = WORK_THREADS / A;          // per-node sums: threads per channel
    const int comp = tid % A, sgrp = tid / A;
    auto load = [](int) { return 0.f; };
    auto store = [&](int v, float val, float) { P.out_a[(size_t)v * A + comp] = val * P.scale; };

    // adds the partial sums of `nslabs` slabs with one channel block to acc (16 edges)
    auto take1 = [&](int nslabs, float* acc) {
      for (int q = 0; q < nslabs && !fail; q += 2, steps++) {
        const uint32_t slot = (steps & 1) * 2, ph = (steps >> 1) & 1;
        if (!warp_wait(&bar_done[slot], ph) || !warp_wait(&bar_done[slot + 1], ph)) { fail = 1; break; }
        tc::fence_after_sync();
        float v[32];
        tc::tmem_ld16x2(tlane + slot * NE + e1, tlane + (slot + 1) * NE + e1, v);
#pragma unroll
        for (int i = 0; i < EPT; i++) acc[i] += v[i] + v[16 + i];
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bar_taken[steps & 1]);
      }
    };
    // the same for a hidden layer
    auto take_hidden = [&](int nslabs, float* acc) {
      if constexpr (HB == 1) {
        take1(nslabs, acc);
      } else {
      for (int q = 0; q < nslabs && !fail; q += 2, steps++) {
        const uint32_t slot = (steps & 1) * 2 + hblk;
        if (!warp_wait(&bar_done[slot], (steps >> 1) & 1)) { fail = 1; break; }
        tc::fence_after_sync();
        float v[32];
        tc::tmem_ld32(tlane + slot * NE + eh, v);
#pragma unroll
        for (int i = 0; i < EH; i++) acc[i] += v[i];
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bar_taken[steps & 1]);
      }
      }
    };
    auto put = [&](unsigned char* planes, int plane, int k, int e, float v) {
      __half v1, v2;
      split(v, &v1, &v2);
      unsigned char* at = planes + (k >> 3) * PANEL + e * 16 + (k & 7) * 2;
      *reinterpret_cast<__half*>(at) = v1;
      *reinterpret_cast<__half*>(at + plane) = v2;
    };

    for (int seg_lo = 0; seg_lo < P.Nt && !fail; seg_lo += seg_nodes) {
      const BlockRange br = block_range(P.row_ptr, seg_lo, min(seg_lo + seg_nodes, P.Nt), NE);
      const int n_begin = br.n_begin, n_end = br.n_end;
      int cur = n_begin;          // node that s_carry belongs to
      int node_lo = n_begin;      // source node of the next tile's first edge (or an earlier one)
      sync_workers();             // the previous segment's last readers of s_rowwin are done
      stage_window<NE>(s_rowwin, P.row_ptr, node_lo, max(n_end, n_begin), tid);
      if (tid < A) s_carry[(tiles & 1) * A + tid] = 0.f;
      sync_workers();

      for (long long e0 = br.e_begin; e0 < br.e_end; e0 += NE) {
        const int cnt = (int)(br.e_end - e0 < NE ? br.e_end - e0 : NE);
        // ---- geometry ----------------------------------------------------------------------------------------------
        if (tid < NE) {
          int j = 0, s = -1;
          if (tid < cnt) {
            const long long e = e0 + tid;
            edge_geometry(P.rij, e, P.r0, s_jac, &s_geom[tid]);
            j = P.dst[e];
            s = source_node<NE>(s_rowwin, P.row_ptr, node_lo, n_end, e);
          }
          s_dst[tid] = j;
          s_src[tid] = s;
          s_max[tid] = 0u;
        }
        sync_workers();
        // ---- products of channel pc with EPP edges, and the largest of every edge ------------------------------------
        float y[EPP][3];
#pragma unroll
        for (int i = 0; i < EPP; i++) {
          const int e = pe + i;
          float y0 = 0.f, y1 = 0.f, y2 = 0.f;
          if (e < cnt) {
            const float* f = P.rows + (size_t)s_dst[e] * 13 * C + pc;
            float l[13];
#pragma unroll
            for (int k = 0; k < 13; k++) l[k] = __ldg(f + k * C);
            const float4* gp = reinterpret_cast<const float4*>(&s_geom[e]);
            const float4 g0 = gp[0], g1 = gp[1], gr = gp[2];
            float pa = wb;
            pa = fmaf(g0.x, w8[0], pa); pa = fmaf(g0.y, w8[1], pa); pa = fmaf(g0.z, w8[2], pa); pa = fmaf(g0.w, w8[3], pa);
            pa = fmaf(g1.x, w8[4], pa); pa = fmaf(g1.y, w8[5], pa); pa = fmaf(g1.z, w8[6], pa); pa = fmaf(g1.w, w8[7], pa);
            const float rh[3] = {gr.x, gr.y, gr.z};
            y0 = l[0] * pa;
            y1 = (l[1] * rh[0] + l[2] * rh[1] + l[3] * rh[2]) * pa;
#pragma unroll
            for (int x = 0; x < 3; x++)
              y2 = fmaf(l[4 + 3 * x] * rh[0] + l[5 + 3 * x] * rh[1] + l[6 + 3 * x] * rh[2], rh[x], y2);
            y2 *= pa;
          }
          y[i][0] = y0; y[i][1] = y1; y[i][2] = y2;
          // sizes as bit patterns: ordered like the numbers, with infinities and NaN above them
          unsigned m = max(max(__float_as_uint(y0) & 0x7fffffffu, __float_as_uint(y1) & 0x7fffffffu), __float_as_uint(y2) & 0x7fffffffu);
          m = __reduce_max_sync(0xffffffffu, m);
          if (lane == 0) atomicMax(&s_max[e], m);
        }
        sync_workers();
        if (tid < NE) {
          const float by = __uint_as_float(s_max[tid]);
          const BeeScales<const float> all(P.scales, A);
          EdgeScales c;
          c.y = scale_for(by);
          c.down_y = c.y * (1.f / 16384.f); c.up_y = 1.0f / c.down_y;
          c.down_1 = scale_for(edge_size(by, all.ratio_1[0], all.ratio_1[1])) * (1.f / 16384.f); c.up_1 = 1.0f / c.down_1;
          c.down_2 = scale_for(edge_size(by, all.ratio_2[0], all.ratio_2[1])) * (1.f / 16384.f); c.up_2 = 1.0f / c.down_2;
          s_sc[tid] = c;
        }
        sync_workers();
#pragma unroll
        for (int i = 0; i < EPP; i++) {
          const float sc = s_sc[pe + i].y;
#pragma unroll
          for (int k = 0; k < 3; k++) put(front, S::YPLANE, k * C + pc, pe + i, y[i][k] * sc);
        }
        tc::fence_async_smem();
        if (sync_or(fail)) { fail = 1; break; }                                              // [X0]
        // ---- psi = Y y -----------------------------------------------------------------------------------------------
        float psi[EPT];
#pragma unroll
        for (int i = 0; i < EPT; i++) psi[i] = 0.f;
        take1(S::SY, psi);
        if (sync_or(fail)) { fail = 1; break; }                                              // [A0]
        const float inv_y = live ? chan.inv_y[o1] : 0.f, sc_psi = live ? chan.sc_psi[o1] : 0.f;
#pragma unroll
        for (int i = 0; i < EPT; i++) {
          psi[i] *= inv_y;
          if (live) put(psi_pl, S::PPLANE, o1, e1 + i, psi[i] * sc_psi);
          psi[i] *= s_sc[e1 + i].up_y;
        }
        tc::fence_async_smem();
        if (sync_or(fail)) { fail = 1; break; }                                              // [X1]
        // ---- two hidden layers ------------------------------------------------------------------------------------------
        float acc[EH];
#pragma unroll
        for (int layer = 1; layer < 3; layer++) {
#pragma unroll
          for (int i = 0; i < EH; i++) acc[i] = 0.f;
          take_hidden(layer == 1 ? S::S1 : S::S2, acc);
          if (sync_or(fail)) { fail = 1; break; }                                            // [A1], [A2]
          const float inv = layer == 1 ? chan.inv_1[oh] : chan.inv_2[oh], sc = layer == 1 ? chan.sc_1[oh] : chan.sc_2[oh];
#pragma unroll
          for (int i = 0; i < EH; i++) {
            const EdgeScales& c = s_sc[eh + i];
            const float h = layer == 1 ? leaky(fmaf(acc[i], c.up_y * inv, b1)) * (c.down_1 * sc) : leaky(fmaf(acc[i], c.up_1 * inv, b2)) * (c.down_2 * sc);
            put(front, S::HPLANE, oh, eh + i, h);
          }
          tc::fence_async_smem();
          if (sync_or(fail)) { fail = 1; break; }                                            // [X2], [X3]
        }
        if (fail) break;
        // ---- out = psi + Wd psi + W3 h2 + b3 --------------------------------------------------------------------------
        float o3[EPT], od[EPT];
#pragma unroll
        for (int i = 0; i < EPT; i++) o3[i] = od[i] = 0.f;
        take1(S::S3, o3);
        take1(S::SD, od);
        if (sync_or(fail)) { fail = 1; break; }                                              // [A3]
        // ---- per-node sums ------------------------------------------------------------------------------------------------
        node_lo = s_src[cnt - 1];
        if (live) {
          const float inv_3 = chan.inv_3[o1], inv_d = chan.inv_d[o1];
#pragma unroll
          for (int i = 0; i < EPT; i++)
            vals[o1 * (NE + 1) + e1 + i] = psi[i] + (fmaf(o3[i], s_sc[e1 + i].up_2 * inv_3, b3) + od[i] * (s_sc[e1 + i].up_y * inv_d));
        }
        stage_window<NE>(s_rowwin, P.row_ptr, node_lo, n_end, tid);   // for the next tile
        mark_nodes<NE>(s_begin, s_src, cnt, cur, tid);
        sync_workers();
        node_sums<1, GROUPS, NE / GROUPS>(vals + comp * (NE + 1), s_src, s_begin, 0, cnt, sgrp, cur, s_carry + (tiles & 1) * A + comp,
                                       s_carry + (~tiles & 1) * A + comp, load, store);
        tiles++;
        cur = node_lo;
        sync_workers();   // geometry and planes are rewritten by the next tile
      }
      if (!fail && n_begin < n_end && sgrp == 0) {
        store(cur, s_carry[(tiles & 1) * A + comp], 0.f);
        empty_nodes<1>(cur + 1, n_end, load, store);
      }
    }
    if (fail && sgrp == 0) mark_failed(P.row_ptr, P.Nt, seg_nodes, NE, store);
  }
  if (fail && lane == 0 && P.status != nullptr) atomicOr(P.status, LD_FLAG_TIMEOUT);
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem_base, 256);
}

// l0 [rows][C], l1 [rows][C][3], l2 [rows][C][9] -> [rows][13][C]
__global__ void __launch_bounds__(256) bee_rows13_kernel(const float* __restrict__ l0, const float* __restrict__ l1, const float* __restrict__ l2,
                                                         long long n, int C, float* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;   // (row, channel)
  if (i >= n) return;
  const long long row = i / C;
  float* o = out + row * 13 * C + (i - row * C);
  o[0] = l0[i];
#pragma unroll
  for (int k = 0; k < 3; k++) o[(size_t)(1 + k) * C] = l1[i * 3 + k];
#pragma unroll
  for (int k = 0; k < 9; k++) o[(size_t)(4 + k) * C] = l2[i * 9 + k];
}

template <int C, int A>
int launch(const BeeSplitParams& P, cudaStream_t st) {
  LD_CUDA_TRY(cudaFuncSetAttribute(bee_scalar_split_kernel<C, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BeeShape<C, A>::SMEM));
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  bee_scalar_split_kernel<C, A><<<sms, THREADS, BeeShape<C, A>::SMEM, st>>>(P);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

bool split_form(int C, int A) { return (C == 64 || C == 128) && (A == 64 || A == 128); }

}  // namespace

static long long packed_slabs(int chan, int dim_a) {
  const long long hb = 2 * dim_a / 128;
  return (3 * chan / 32 + (dim_a / 32 + 2 * dim_a / 32) * hb + 3 * dim_a / 32) * (long long)(SLAB_BYTES / 2);
}

// FP16 elements of the packed weights of a layer with `chan` product and dim_a scalar channels (0: no split form)
extern "C" int ld_bee_split_elems(int chan, int dim_a, long long* elems) {
  if (chan <= 0 || dim_a <= 0) return LD_ERR_SHAPE;
  *elems = split_form(chan, dim_a) ? packed_slabs(chan, dim_a) + 2LL * (FLOATS_PER_A * dim_a + FLOATS_EXTRA) : 0;
  return LD_OK;
}

// packed: as many FP16 values as ld_bee_split_elems says, 16-byte aligned. Weights [in][out], FP32. scales: not used.
extern "C" int ld_bee_split_pack(const float* Yt, const float* W1t, const float* b1, const float* W2t, const float* b2, const float* W3t,
                                 const float* Wdt, int chan, int dim_a, void* packed, float* scales, void* stream) {
  (void)scales;
  if (!split_form(chan, dim_a)) { ld_set_last_message("bee split pack: chan and dim_a must be 64 or 128"); return LD_ERR_UNSUPPORTED; }
  if (((uintptr_t)packed % 16) != 0) return LD_ERR_SHAPE;
  cudaStream_t st = (cudaStream_t)stream;
  const int A = dim_a, hb = 2 * A / 128;
  __half* wy = (__half*)packed;
  const BeeScales<float> c((float*)(wy + packed_slabs(chan, A)), A);
  __half* w1 = wy + (size_t)(3 * chan / 32) * (SLAB_BYTES / 2);
  __half* w2 = w1 + (size_t)(A / 32 * hb) * (SLAB_BYTES / 2);
  __half* w3 = w2 + (size_t)(2 * A / 32 * hb) * (SLAB_BYTES / 2);
  __half* wd = w3 + (size_t)(2 * A / 32) * (SLAB_BYTES / 2);
  int rc = split_layer<SPLIT_LINEAR>(SplitLayer{Yt, 3 * chan, A, nullptr, nullptr, nullptr, nullptr, wy, c.inv_y, c.sc_psi, c.p_psi, nullptr, nullptr}, st);
  if (rc == LD_OK) rc = split_layer<SPLIT_LEAKY>(SplitLayer{W1t, A, 2 * A, c.p_psi, nullptr, c.sc_psi, b1, w1, c.inv_1, c.sc_1, c.p_1, c.q_1, nullptr}, st);
  if (rc == LD_OK) rc = split_layer<SPLIT_LEAKY>(SplitLayer{W2t, 2 * A, 2 * A, c.p_1, c.q_1, c.sc_1, b2, w2, c.inv_2, c.sc_2, c.p_2, c.q_2, c.ratio_1}, st);
  if (rc == LD_OK) rc = split_layer<SPLIT_LAST>(SplitLayer{W3t, 2 * A, A, c.p_2, c.q_2, c.sc_2, nullptr, w3, c.inv_3, nullptr, nullptr, nullptr, c.ratio_2}, st);
  if (rc == LD_OK) rc = split_layer<SPLIT_LAST>(SplitLayer{Wdt, A, A, c.p_psi, nullptr, c.sc_psi, nullptr, wd, c.inv_d, nullptr, nullptr, nullptr, nullptr}, st);
  return rc;
}

// rows13 [rows][13][chan] = (l0 | l1 | l2 component-major): the neighbour rows of the two FP32 edge kernels
extern "C" int ld_bee_rows13_f32(const float* l0, const float* l1, const float* l2, long long rows, int chan, float* rows13, void* stream) {
  if (rows < 0 || chan <= 0) return LD_ERR_SHAPE;
  const long long n = rows * chan;
  if (n == 0) return LD_OK;
  bee_rows13_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(l0, l1, l2, n, chan, rows13);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

// ld_bee_messages_scalar_f32 on neighbour rows from ld_bee_rows13_f32 and weights from ld_bee_split_pack. status_dev
// receives LD_FLAG_TIMEOUT if a bounded wait ran out. scales: not used.
extern "C" int ld_bee_messages_scalar_f32_split(const int* row_ptr, const int* dst, const float* rij, int Nt, int chan, int dim_a, float r0,
                                                const float* rows13, const float* enc_w, const float* enc_b, const float* jacobi,
                                                const void* packed, const float* scales, const float* b1, const float* b2,
                                                const float* b3, float scale, float* out_a, int* status_dev, void* stream) {
  (void)scales;
  if (Nt < 0 || chan <= 0 || dim_a <= 0 || !(r0 > 0.f)) return LD_ERR_SHAPE;
  if (!split_form(chan, dim_a)) { ld_set_last_message("bee messages (split path): chan and dim_a must be 64 or 128"); return LD_ERR_UNSUPPORTED; }
  if (b1 == nullptr || b2 == nullptr || b3 == nullptr || ((uintptr_t)packed % 16) != 0) return LD_ERR_SHAPE;
  if (Nt == 0) return LD_OK;
  BeeSplitParams P;
  P.row_ptr = row_ptr; P.dst = dst; P.rij = rij; P.Nt = Nt;
  P.seg_nodes = ld_even_segments(Nt, (40LL << 20) / (52LL * chan));   // the gathered rows of a segment stay in L2
  P.r0 = r0; P.scale = scale; P.rows = rows13; P.enc_w = enc_w; P.enc_b = enc_b; P.jacobi = jacobi;
  P.w = (const __half*)packed; P.scales = (const float*)(P.w + packed_slabs(chan, dim_a)); P.b1 = b1; P.b2 = b2; P.b3 = b3; P.out_a = out_a; P.status = status_dev;
  cudaStream_t st = (cudaStream_t)stream;
  if (chan == 128) return dim_a == 128 ? launch<128, 128>(P, st) : launch<128, 64>(P, st);
  return dim_a == 128 ? launch<64, 128>(P, st) : launch<64, 64>(P, st);
}
