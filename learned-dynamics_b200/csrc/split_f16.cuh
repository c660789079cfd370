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


// ---- edges and their source nodes ------------------------------------------------------------------------------
// row_ptr[node .. node + NE] of the coming tile, whose first edge belongs to `node` or a later one
template <int NE>
__device__ __forceinline__ void stage_window(int* s_rowwin, const int* __restrict__ row_ptr, int node, int n_end, int tid) {
  for (int i = tid; i <= NE; i += WORK_THREADS) s_rowwin[i] = row_ptr[min(node + i, n_end)];
}
// source node of edge e: the largest v with row_ptr[v] <= e, in the staged window first
template <int NE>
__device__ __forceinline__ int source_node(const int* s_rowwin, const int* __restrict__ row_ptr, int node, int n_end, long long e) {
  if ((long long)s_rowwin[NE] > e) {
    int lo = 0, hi = NE;
    while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if ((long long)s_rowwin[mid] > e) hi = mid; else lo = mid; }
    return node + lo;
  }
  int lo = node + NE, hi = n_end;   // row_ptr[lo] <= e < row_ptr[hi]
  while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if ((long long)row_ptr[mid] > e) hi = mid; else lo = mid; }
  return lo;
}

// Sums over a tile's edges per source node, one edge after the other, so that a node's sum has the same bits wherever its
// edges fall in a tile or a block. A thread adds one component (m: its values, in edge order); `load` fetches what is added to a
// node's sum when it is written, `store` writes it. Bound by latency when nodes have few edges, so loads of several nodes are
// put in flight together.
//   node_walk: a thread per component walks all edges, its sum stays in a register.
//   node_sums: GROUPS threads per component share the tile, each with the nodes that begin in its SPAN edges; nodes are found
//   from a bit per edge (mark_nodes), and the sum of the node whose edges may go on in the next tile is carried over in shared
//   memory.
// Measured with a walk for every width and with groups (65536 nodes, BF16): n = 32, one edge a node 180 -> 104 us, with
// residuals 340 -> 110; n = 64, four edges a node 453 -> 360 and 628 -> 373.

// bit e: edge e begins another node than edge e - 1 (edge 0: than `cur`). Threads [0, NE).
template <int NE>
__device__ __forceinline__ void mark_nodes(uint32_t* s_begin, const int* s_src, int cnt, int cur, int tid) {
  if (tid >= NE) return;
  const uint32_t b = __ballot_sync(0xffffffffu, tid < cnt && s_src[tid] != (tid == 0 ? cur : s_src[tid - 1]));
  if ((tid & 31) == 0) s_begin[tid >> 5] = b;
}

// rows [from, to) without edges
template <int BATCH, class Load, class Store>
__device__ __forceinline__ void empty_nodes(int from, int to, const Load& load, const Store& store) {
  for (int v = from; v < to; v += BATCH) {
    float r[BATCH];
#pragma unroll
    for (int q = 0; q < BATCH; q++) r[q] = v + q < to ? load(v + q) : 0.f;
#pragma unroll
    for (int q = 0; q < BATCH; q++)
      if (v + q < to) store(v + q, 0.f, r[q]);
  }
}

// edges [p0, p0 + live) of the tile, m[0] belongs to edge p0 (whole eighths are read); sum, cur: of the node that goes on.
// AHEAD: what eight edges' nodes load is put in flight before the first is written. The FP32 kernel gains by it (n = 128, one
// edge a node, 65536 nodes: 933 -> 747 us with residuals, 776 -> 720 without), the BF16 kernel pays more for the registers on
// dense graphs (3.53 -> 3.69 ms at 256 edges a node) than it gains.
template <bool AHEAD, class Load, class Store>
__device__ __forceinline__ void node_walk(const float* m, const int* s_src, int p0, int live, float& sum, int& cur, const Load& load,
                                          const Store& store) {
  for (int eb = 0; eb < live; eb += 8) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = m[eb + i];
    const int last = min(eb + 8, live) - 1;
    if (s_src[p0 + last] == cur && last == eb + 7) {   // one node's
#pragma unroll
      for (int i = 0; i < 8; i++) sum += v[i];
      continue;
    }
    float r[8];   // for the node that ends before edge i
    if (AHEAD) {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int before = i == 0 ? cur : s_src[p0 + min(eb + i - 1, last)];
        r[i] = s_src[p0 + min(eb + i, last)] != before ? load(before) : 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (eb + i < live) {
        const int s = s_src[p0 + eb + i];
        if (s != cur) {
          if (AHEAD) { store(cur, sum, r[i]); sum = 0.f; cur++; }
          for (; cur < s; cur++, sum = 0.f) store(cur, sum, load(cur));
        }
        sum += v[i];
      }
  }
}

// a + m[0] + m[1] + ..., the loads ahead of the additions
template <int COUNT>
__device__ __forceinline__ float add_run(const float* m, float a) {
  float v[COUNT];
#pragma unroll
  for (int i = 0; i < COUNT; i++) v[i] = m[i];
#pragma unroll
  for (int i = 0; i < COUNT; i++) a += v[i];
  return a;
}

// as above; cur: the node that carry_in belongs to
template <int BATCH, int GROUPS, int SPAN, class Load, class Store>
__device__ __forceinline__ void node_sums(const float* m, const int* s_src, const uint32_t* s_begin, int p0, int live, int grp, int cur,
                                          const float* carry_in, float* carry_out, const Load& load, const Store& store) {
  // the edges that begin a node, one after the other; then `live`
  int word = (p0 + grp * SPAN) >> 5;
  const int words = (p0 + live + 31) >> 5;
  uint32_t bits = word < words ? s_begin[word] & (0xffffffffu << ((p0 + grp * SPAN) & 31)) : 0u;
  auto next = [&]() {
    while (bits == 0u) {
      if (++word >= words) return live;
      bits = s_begin[word];
    }
    const int e = word * 32 + __ffs(bits) - 1 - p0;
    bits &= bits - 1u;
    return e;
  };
  const int stop = min(live, (grp + 1) * SPAN);   // nodes that begin at or after it are the next group's
  int e = 0, end, node = cur;
  float first = 0.f;
  if (grp == 0) {
    first = *carry_in;
    end = next();   // (0: `cur` has no edge here)
  } else {
    e = next();
    if (e >= stop) return;
    node = s_src[p0 + e];
    end = next();
  }
  for (bool more = true; more;) {
    int nd[BATCH], lo[BATCH], hi[BATCH];
    float r[BATCH], v0[BATCH];   // residual and first edge of each
#pragma unroll
    for (int q = 0; q < BATCH; q++) {
      hi[q] = -1;
      r[q] = 0.f;
      if (more) {
        nd[q] = node; lo[q] = e; hi[q] = end;
        v0[q] = m[min(e, live - 1)];
        if (end < live) r[q] = load(node);
        e = end;
        more = e < stop;
        if (more) { node = s_src[p0 + e]; end = next(); }
      }
    }
#pragma unroll
    for (int q = 0; q < BATCH; q++) {
      if (hi[q] < 0) continue;
      float a = first;
      first = 0.f;
      int k = lo[q];
      if (k < hi[q]) { a += v0[q]; k++; }
      for (; k + 8 <= hi[q]; k += 8) a = add_run<8>(m + k, a);
      if (k + 4 <= hi[q]) { a = add_run<4>(m + k, a); k += 4; }
      if (k + 2 <= hi[q]) { a = add_run<2>(m + k, a); k += 2; }
      if (k < hi[q]) a += m[k];
      if (hi[q] < live) {
        store(nd[q], a, r[q]);
        empty_nodes<BATCH>(nd[q] + 1, s_src[p0 + hi[q]], load, store);
      } else {
        *carry_out = a;
      }
    }
  }
}

// After a wait that ran out: NaN for every node of this block, so that the outputs themselves show that they are incomplete
// (callers that do not read the status word would take what was in the buffer for results).
template <class Store>
__device__ __forceinline__ void mark_failed(const int* __restrict__ row_ptr, int Nt, int seg_nodes, int tile, const Store& store) {
  for (int seg_lo = 0; seg_lo < Nt; seg_lo += seg_nodes) {
    const BlockRange br = block_range(row_ptr, seg_lo, min(seg_lo + seg_nodes, Nt), tile);
    for (int v = br.n_begin; v < br.n_end; v++) store(v, __int_as_float(0x7fc00000), 0.f);
  }
}

}  // namespace sf
