// Scalar output of the l<=2 message layer at FP32 accuracy with the per-edge linear maps on the tensor cores: what
// bee_scalar_kernel of bee_messages.cu computes (Messages.forward of archs/diffuser_atoms15.py:227-253, scalar channel),
// with operands split into two FP16 values (split_f16.cuh).
//
//   y   = the three scalar products of every channel                    K = 3 C
//   psi = Y y ;  h1 = leaky(W1 psi + b1) ;  h2 = leaky(W2 h1 + b2)      widths A, 2 A, 2 A
//   out = psi + Wd psi + W3 h2 + b3, summed per source node, times `scale`
//
// What bounds it: the shared-memory port under the MMAs (48 cycles per 128 x 64 x 16 MMA plus the weight slabs that arrive
// through it) and the phases of a tile that follow one another. C = A = 128, 219 k edges: 0.68 ms, against 7.39 ms on
// the FMA pipe.
//
// A block owns a node-aligned slice of the CSR and walks it 64 edges at a time; roles as in painn_message_split.cu. The
// neighbours' rows are read component-major, [node][13][C], so that a warp's loads are 128 consecutive bytes. The sizes of
// the products are not bounded beforehand: the scale of an edge's operands comes from its largest product, those of the
// later layers from that and from row sums of the weights. Every step of the pipeline is two weight slabs: the two blocks
// of 128 channels of a hidden layer, or two chunks of K of a layer with one block.
#include "common.cuh"
#include "split_f16.cuh"
#include "bee_edge.cuh"

namespace {
using namespace sf;

constexpr int NE = 64, PANEL = NE * 16 + 16, EPT = 16;
// scales[10] = swY, sw1, sw2, sw3, swd, max row sums of |Y|, |W1|, max |b1|, max row sum of |W2|, max |b2|

// C product channels, A scalar channels
template <int C, int A>
struct BeeShape {
  static constexpr int HB = 2 * A / 128;                 // blocks of 128 channels of a hidden layer
  static constexpr int YPLANE = (3 * C / 8) * PANEL, HPLANE = (2 * A / 8) * PANEL, PPLANE = (A / 8) * PANEL;
  static constexpr int FRONT = YPLANE > HPLANE ? 2 * YPLANE : 2 * HPLANE;   // products, then hidden layers
  static constexpr size_t SMEM = (size_t)FRONT + 2 * PPLANE + STAGES * SLAB_BYTES;
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
  const float* scales;                     // [10]
  const float* b1; const float* b2; const float* b3;
  float* out_a;
  int* status;
};

__device__ __forceinline__ float leaky(float v) { return v > 0.f ? v : 0.1f * v; }

// scales of one edge: operand scales and the inverse products that take an accumulator back
struct EdgeScales { float y, inv_y, psi, inv_1, inv_d, h1, inv_2, h2, inv_3; };

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
  __shared__ float s_jac[72];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* front = smem;                       // planes of the products, later of the hidden layers
  float* vals = reinterpret_cast<float*>(smem);      // [A][NE + 1], after the last layer
  unsigned char* psi_pl = smem + S::FRONT;           // planes of psi
  unsigned char* ring = psi_pl + 2 * S::PPLANE;

  if (tid < 8) ld_poly8_to_chebyshev(P.jacobi + tid * 9, s_jac + tid * 9);   // Chebyshev form of the radial polynomials
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
    uint32_t steps = 0;

    // adds the partial sums of `nslabs` slabs with one channel block to acc (16 edges)
    auto take1 = [&](int nslabs, float* acc) {
      for (int q = 0; q < nslabs && !fail; q += 2, steps++) {
        const uint32_t slot = (steps & 1) * 2, ph = (steps >> 1) & 1;
        if (!tc::mbar_wait(&bar_done[slot], ph) || !tc::mbar_wait(&bar_done[slot + 1], ph)) { fail = 1; break; }
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
        if (!tc::mbar_wait(&bar_done[slot], (steps >> 1) & 1)) { fail = 1; break; }
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
      float carry = 0.f;          // thread tid < A: sum of channel tid of node `cur`
      int cur = n_begin;
      int node_lo = n_begin;      // source node of the next tile's first edge (or an earlier one)
      sync_workers();             // the previous segment's last readers of s_rowwin are done
      for (int i = tid; i <= NE; i += WORK_THREADS) s_rowwin[i] = P.row_ptr[min(node_lo + i, n_end > n_begin ? n_end : n_begin)];
      sync_workers();
      // output of node `from`, zeros for the nodes (from, next)
      auto flush_until = [&](int from, int next, float val) {
        if (tid < A)
          for (int v = from; v < next; v++) P.out_a[(size_t)v * A + tid] = v == from ? val * P.scale : 0.f;
      };

      for (long long e0 = br.e_begin; e0 < br.e_end; e0 += NE) {
        const int cnt = (int)(br.e_end - e0 < NE ? br.e_end - e0 : NE);
        // ---- geometry ----------------------------------------------------------------------------------------------
        if (tid < NE) {
          int j = 0, s = -1;
          if (tid < cnt) {
            const long long e = e0 + tid;
            edge_geometry(P.rij, e, P.r0, s_jac, &s_geom[tid]);
            j = P.dst[e];
            int lo, hi;   // source node: largest v with row_ptr[v] <= e, in the staged window first
            if ((long long)s_rowwin[NE] > e) {
              lo = 0; hi = NE;
              while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if ((long long)s_rowwin[mid] > e) hi = mid; else lo = mid; }
              s = node_lo + lo;
            } else {
              lo = node_lo + NE; hi = n_end;
              while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if ((long long)P.row_ptr[mid] > e) hi = mid; else lo = mid; }
              s = lo;
            }
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
          const float by = __uint_as_float(s_max[tid]), bp = P.scales[5] * by, bh1 = fmaf(P.scales[6], bp, P.scales[7]) * 1.001f,
                      bh2 = fmaf(P.scales[8], bh1, P.scales[9]) * 1.001f;   // (row sums already carry their rounding)
          EdgeScales c;
          c.y = scale_for(by); c.psi = scale_for(bp); c.h1 = scale_for(bh1); c.h2 = scale_for(bh2);
          c.inv_y = 1.0f / (c.y * P.scales[0]);
          c.inv_1 = 1.0f / (c.psi * P.scales[1]); c.inv_d = 1.0f / (c.psi * P.scales[4]);
          c.inv_2 = 1.0f / (c.h1 * P.scales[2]); c.inv_3 = 1.0f / (c.h2 * P.scales[3]);
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
        fail = __any_sync(0xffffffffu, fail);
        if (sync_or(fail)) { fail = 1; break; }                                              // [A0]
#pragma unroll
        for (int i = 0; i < EPT; i++) {
          psi[i] *= s_sc[e1 + i].inv_y;
          if (live) put(psi_pl, S::PPLANE, o1, e1 + i, psi[i] * s_sc[e1 + i].psi);
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
          fail = __any_sync(0xffffffffu, fail);
          if (sync_or(fail)) { fail = 1; break; }                                            // [A1], [A2]
#pragma unroll
          for (int i = 0; i < EH; i++) {
            const EdgeScales& c = s_sc[eh + i];
            const float h = layer == 1 ? leaky(fmaf(acc[i], c.inv_1, b1)) * c.h1 : leaky(fmaf(acc[i], c.inv_2, b2)) * c.h2;
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
        fail = __any_sync(0xffffffffu, fail);
        if (sync_or(fail)) { fail = 1; break; }                                              // [A3]
        // ---- per-node sums, thread = channel: one edge after the other, so that a node's sum does not depend on where its
        // edges fall in a tile or a block -----------------------------------------------------------------------------
        node_lo = s_src[cnt - 1];
        if (live) {
#pragma unroll
          for (int i = 0; i < EPT; i++)
            vals[o1 * (NE + 1) + e1 + i] = psi[i] + (fmaf(o3[i], s_sc[e1 + i].inv_3, b3) + od[i] * s_sc[e1 + i].inv_d);
        }
        for (int i = tid; i <= NE; i += WORK_THREADS) s_rowwin[i] = P.row_ptr[min(node_lo + i, n_end)];   // for the next tile
        sync_workers();
        if (tid < A) {
          const float* m = vals + tid * (NE + 1);
          int c_node = cur;
          for (int eb = 0; eb < cnt; eb += 8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = m[eb + i];
            const int last = min(eb + 8, cnt) - 1;
            if (s_src[last] == c_node && last == eb + 7) {
#pragma unroll
              for (int i = 0; i < 8; i++) carry += v[i];
            } else {
#pragma unroll
              for (int i = 0; i < 8; i++)
                if (eb + i < cnt) {
                  const int s = s_src[eb + i];
                  if (s != c_node) { flush_until(c_node, s, carry); carry = 0.f; c_node = s; }
                  carry += v[i];
                }
            }
          }
        }
        cur = node_lo;
        sync_workers();   // geometry and planes are rewritten by the next tile
      }
      if (!fail && n_begin < n_end) flush_until(cur, n_end, carry);
    }
  }
  if (fail && lane == 0 && P.status != nullptr) atomicOr(P.status, LD_FLAG_TIMEOUT);
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem_base, 256);
}

// Wt: [in][out]. One block per matrix (Y, W1, W2, W3, Wd): its scale, and for the first three the largest row sum (over the
// inputs) and the largest bias.
__global__ void __launch_bounds__(256) bee_split_scales_kernel(const float* Yt, const float* W1t, const float* b1, const float* W2t,
                                                               const float* b2, const float* W3t, const float* Wdt, int C, int A, float* scales) {
  __shared__ float s_sum[256], s_max[256], s_b[256];
  const int which = blockIdx.x, o = threadIdx.x;
  const float* W = which == 0 ? Yt : which == 1 ? W1t : which == 2 ? W2t : which == 3 ? W3t : Wdt;
  const int K = which == 0 ? 3 * C : (which == 1 || which == 4) ? A : 2 * A, N = (which == 1 || which == 2) ? 2 * A : A;
  const float* b = which == 1 ? b1 : which == 2 ? b2 : nullptr;
  float sum = 0.f, mx = 0.f;
  if (o < N)
    for (int k = 0; k < K; k++) { const float a = fabsf(W[(size_t)k * N + o]); sum += a; mx = fmaxf(mx, a); }
  s_sum[o] = sum * 1.001f; s_max[o] = mx; s_b[o] = o < N && b != nullptr ? fabsf(b[o]) : 0.f;
  __syncthreads();
  for (int d = 128; d > 0; d >>= 1) {
    if (o < d) { s_sum[o] = fmaxf(s_sum[o], s_sum[o + d]); s_max[o] = fmaxf(s_max[o], s_max[o + d]); s_b[o] = fmaxf(s_b[o], s_b[o + d]); }
    __syncthreads();
  }
  if (o == 0) {
    scales[which] = scale_for(s_max[0]);
    if (which == 0) scales[5] = s_sum[0];
    if (which == 1) { scales[6] = s_sum[0]; scales[7] = s_b[0]; }
    if (which == 2) { scales[8] = s_sum[0]; scales[9] = s_b[0]; }
  }
}

// Wt [K][N] -> slabs [K chunk of 32][block of 128 outputs][plane][4][128][8]; outputs from N on are zeros
__global__ void bee_split_pack_kernel(const float* __restrict__ Wt, int K, int N, const float* __restrict__ scale, __half* __restrict__ out) {
  const int Np = (N + 127) / 128 * 128;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= K * Np) return;
  const int o = idx % Np, k = idx / Np;
  const float v = o < N ? Wt[(size_t)k * N + o] * scale[0] : 0.f;
  __half* slab = out + ((size_t)(k / SLAB_K) * (Np / 128) + o / 128) * (SLAB_BYTES / 2);
  __half* at = slab + (size_t)((k % SLAB_K) / 8) * 128 * 8 + (o % 128) * 8 + k % 8;
  split(v, at, at + SLAB_K * 128);
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

// FP16 elements of the packed weights of a layer with `chan` product and dim_a scalar channels (0: no split form)
extern "C" int ld_bee_split_elems(int chan, int dim_a, long long* elems) {
  if (chan <= 0 || dim_a <= 0) return LD_ERR_SHAPE;
  const long long hb = 2 * dim_a / 128;
  *elems = split_form(chan, dim_a) ? (3 * chan / 32 + (dim_a / 32 + 2 * dim_a / 32) * hb + 3 * dim_a / 32) * (long long)(SLAB_BYTES / 2) : 0;
  return LD_OK;
}

// packed: as many FP16 values as ld_bee_split_elems says, 16-byte aligned; scales: ten floats. Weights [in][out], FP32.
extern "C" int ld_bee_split_pack(const float* Yt, const float* W1t, const float* b1, const float* W2t, const float* b2, const float* W3t,
                                 const float* Wdt, int chan, int dim_a, void* packed, float* scales, void* stream) {
  if (!split_form(chan, dim_a)) { ld_set_last_message("bee split pack: chan and dim_a must be 64 or 128"); return LD_ERR_UNSUPPORTED; }
  cudaStream_t st = (cudaStream_t)stream;
  bee_split_scales_kernel<<<5, 256, 0, st>>>(Yt, W1t, b1, W2t, b2, W3t, Wdt, chan, dim_a, scales);
  LD_LAUNCH_CHECK();
  const float* W[5] = {Yt, W1t, W2t, W3t, Wdt};
  const int K[5] = {3 * chan, dim_a, 2 * dim_a, 2 * dim_a, dim_a}, N[5] = {dim_a, 2 * dim_a, 2 * dim_a, dim_a, dim_a};
  __half* out = (__half*)packed;
  for (int l = 0; l < 5; l++) {
    const int Np = (N[l] + 127) / 128 * 128;
    bee_split_pack_kernel<<<ld_cdiv((long long)K[l] * Np, 256), 256, 0, st>>>(W[l], K[l], N[l], scales + l, out);
    LD_LAUNCH_CHECK();
    out += (size_t)K[l] / SLAB_K * (Np / 128) * (SLAB_BYTES / 2);
  }
  return LD_OK;
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
// receives LD_FLAG_TIMEOUT if a bounded wait ran out.
extern "C" int ld_bee_messages_scalar_f32_split(const int* row_ptr, const int* dst, const float* rij, int Nt, int chan, int dim_a, float r0,
                                                const float* rows13, const float* enc_w, const float* enc_b, const float* jacobi,
                                                const void* packed, const float* scales, const float* b1, const float* b2,
                                                const float* b3, float scale, float* out_a, int* status_dev, void* stream) {
  if (Nt < 0 || chan <= 0 || dim_a <= 0 || !(r0 > 0.f)) return LD_ERR_SHAPE;
  if (!split_form(chan, dim_a)) { ld_set_last_message("bee messages (split path): chan and dim_a must be 64 or 128"); return LD_ERR_UNSUPPORTED; }
  if (b1 == nullptr || b2 == nullptr || b3 == nullptr || ((uintptr_t)packed % 16) != 0) return LD_ERR_SHAPE;
  if (Nt == 0) return LD_OK;
  BeeSplitParams P;
  P.row_ptr = row_ptr; P.dst = dst; P.rij = rij; P.Nt = Nt;
  P.seg_nodes = ld_even_segments(Nt, (40LL << 20) / (52LL * chan));   // the gathered rows of a segment stay in L2
  P.r0 = r0; P.scale = scale; P.rows = rows13; P.enc_w = enc_w; P.enc_b = enc_b; P.jacobi = jacobi;
  P.w = (const __half*)packed; P.scales = scales; P.b1 = b1; P.b2 = b2; P.b3 = b3; P.out_a = out_a; P.status = status_dev;
  cudaStream_t st = (cudaStream_t)stream;
  if (chan == 128) return dim_a == 128 ? launch<128, 128>(P, st) : launch<128, 64>(P, st);
  return dim_a == 128 ? launch<64, 128>(P, st) : launch<64, 64>(P, st);
}
