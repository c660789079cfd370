// Channel mixing for rank-0/1/2 Cartesian tensors, FP32 SIMT path:
//   y[r, o, s] = sum_i W[o, i] * x[r, i, s],   s in [0, 3^inds)
// Replaces tensorLinearKern / tensorLinearBackwardKern of the reference
// (extensions/tensor_ops/tensor_ops_kern.cu:6-71; autograd glue tensor_ops.cpp:31-170).
// The reference gives one warp to each (output channel, row); here a block computes a tile of outputs x
// (rows * 3^inds) columns from shared memory. W may be strided (the backward pass uses it transposed); x and y are
// contiguous. This path keeps full FP32 products and accumulation (1e-5 parity); the tensor-core
// path for large row counts lives in gemm_tc.cu.
//
// What bounds both kernels: the reads of x (S floats per channel) for narrow outputs, the FMA pipe for wide ones, and in
// between the instructions around the FMAs, which the layouts keep few. x is staged exactly as it lies in memory (per row,
// KC channels of S consecutive components; no transposition for any S) by asynchronous copies of the widest words that its
// alignment allows, with a running (row, word) position instead of a division per word.
// Measured on the edges of 4 x 128 beads (36 k rows, 128 channels), before (one 64-output tile for every width, 4 x 4 or
// 4 x 9 elements per thread, single buffered) and now: 128 -> 32, S = 9: 146 -> 108 us; 32 -> 128, S = 9: 146 -> 112 us;
// 128 -> 64, S = 3: 91 -> 66 us; dW of 128 -> 32, S = 9: 746 -> 72 us; dW of 128 -> 64, S = 3: 242 -> 41 us.
#include "common.cuh"

namespace {

constexpr int TL_THREADS = 256;
constexpr int TL_STAGES = 3;   // two steps of loads in flight behind the one that is multiplied (two stages: 2 to 4 % slower)

__device__ __forceinline__ void tl_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void tl_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

template <int VEC>
__device__ __forceinline__ void tl_cp(float* smem, const float* gmem, bool ok) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = ok ? 4 * VEC : 0;   // 0: the word is zero-filled and gmem is not read
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(gmem), "n"(4 * VEC), "r"(n));
}

// ROWS rows of W floats (in memory ld floats apart) into shared rows PITCH floats apart, VEC floats at a time. Rows from
// `live_rows` and floats from `live` on (a multiple of VEC) are zeros.
template <int VEC, int ROWS, int W, int PITCH>
__device__ __forceinline__ void tl_rows(float* smem, const float* __restrict__ g, long long ld, int live_rows, int live) {
  constexpr int WPR = W / VEC, DR = TL_THREADS / WPR, DW = TL_THREADS % WPR;
  static_assert(W % VEC == 0 && PITCH % VEC == 0, "rows hold whole words");
  int rl = threadIdx.x / WPR, w = threadIdx.x % WPR;
#pragma unroll 4
  for (int it = 0; it < (ROWS * WPR + TL_THREADS - 1) / TL_THREADS; it++) {
    if (rl < ROWS) {
      const bool ok = rl < live_rows && w * VEC < live;
      tl_cp<VEC>(smem + rl * PITCH + w * VEC, ok ? g + rl * ld + w * VEC : g, ok);
    }
    rl += DR; w += DW;
    if (w >= WPR) { w -= WPR; rl++; }
  }
}

// A thread owns OU outputs x NR rows with all their S components. Two channels of a row are 2 S consecutive floats, read
// as S 8-byte words; the pitch is 2 modulo 4, so that the words of the 16 rows of a half warp fall into different banks.
// TY groups of threads share the outputs, TX = 256 / TY the rows.
template <int S, int TY, int OU, int NR>
struct TlTile {
  static constexpr int KC = S == 3 ? 16 : 8, PITCH = KC * S + 2;
  static constexpr int TX = TL_THREADS / TY, TO = TY * OU, TR = TX * NR;
  static constexpr int WP = TO + 4;   // weight rows stay 16-byte aligned
  static constexpr int XF = (TR * PITCH + 3) / 4 * 4;
  static constexpr int STAGE = XF + KC * WP;
  static constexpr size_t BYTES = TL_STAGES * sizeof(float) * STAGE;
};

// W[o, i] at w[0] + o * sw0 + i * sw1; a stack of three matrices (PARTS = 3) has `part` outputs in each of w[0], w[1], w[2]
struct TlWeights { const float* w[3]; long long sw0, sw1; int part; };

template <int S, int TY, int OU, int NR, int VEC, int PARTS>
__global__ void __launch_bounds__(TL_THREADS, 2)
tensor_linear_kernel(const TlWeights W, const float* __restrict__ x, float* __restrict__ y, long long rows, int I, int O) {
  using T = TlTile<S, TY, OU, NR>;
  constexpr int KC = T::KC, PITCH = T::PITCH, TX = T::TX, TO = T::TO, TR = T::TR, WP = T::WP;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const long long r0 = (long long)blockIdx.x * TR;
  const int o0 = blockIdx.y * TO;
  const int rcnt = (int)(rows - r0 < TR ? rows - r0 : TR);
  float acc[OU][NR * S];
#pragma unroll
  for (int u = 0; u < OU; u++)
#pragma unroll
    for (int j = 0; j < NR * S; j++) acc[u][j] = 0.f;

  auto stage = [&](int buf, int i0) {
    float* xs = smem + buf * T::STAGE;
    float* ws = xs + T::XF;
    tl_rows<VEC, TR, KC * S, PITCH>(xs, x + (r0 * I + i0) * S, (long long)I * S, rcnt, min(KC, I - i0) * S);
    for (int idx = tid; idx < KC * TO; idx += TL_THREADS) {
      // lanes run along whichever index of W is the contiguous one
      const int kc = W.sw1 == 1 ? idx % KC : idx / TO, o = W.sw1 == 1 ? idx / KC : idx % TO;
      const bool ok = i0 + kc < I && o0 + o < O;
      const float* w = W.w[0];
      int row = o0 + o;
      if (PARTS == 3) {
        if (row >= 2 * W.part) { w = W.w[2]; row -= 2 * W.part; }
        else if (row >= W.part) { w = W.w[1]; row -= W.part; }
      }
      tl_cp<1>(ws + kc * WP + o, ok ? w + row * W.sw0 + (i0 + kc) * W.sw1 : w, ok);
    }
    tl_commit();
  };

  const int steps = (I + KC - 1) / KC;
#pragma unroll
  for (int k = 0; k < TL_STAGES - 1; k++) { if (k < steps) stage(k, k * KC); else tl_commit(); }
  for (int k = 0; k < steps; k++) {
    tl_wait<TL_STAGES - 2>();   // this thread's part of step k has arrived (groups without copies keep the count)
    __syncthreads();            // everybody's has, and everybody is done with step k - 1, whose buffer is staged next
    if (k + TL_STAGES - 1 < steps) stage((k + TL_STAGES - 1) % TL_STAGES, (k + TL_STAGES - 1) * KC); else tl_commit();
    const float* xs = smem + (k % TL_STAGES) * T::STAGE + tx * PITCH;
    const float* ws = smem + (k % TL_STAGES) * T::STAGE + T::XF + ty * OU;
#pragma unroll 2
    for (int kc = 0; kc < KC; kc += 2) {
      float b[NR][2 * S];   // two channels of each row
#pragma unroll
      for (int n = 0; n < NR; n++)
#pragma unroll
        for (int q = 0; q < S; q++) {
          const float2 v = *reinterpret_cast<const float2*>(xs + n * TX * PITCH + kc * S + 2 * q);
          b[n][2 * q] = v.x; b[n][2 * q + 1] = v.y;
        }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        float a[OU];
        if (OU % 4 == 0) {
#pragma unroll
          for (int u = 0; u < OU; u += 4) {
            const float4 v = *reinterpret_cast<const float4*>(ws + (kc + h) * WP + u);
            a[u] = v.x; a[u + 1] = v.y; a[u + 2] = v.z; a[u + 3] = v.w;
          }
        } else {
#pragma unroll
          for (int u = 0; u < OU; u++) a[u] = ws[(kc + h) * WP + u];
        }
#pragma unroll
        for (int u = 0; u < OU; u++)
#pragma unroll
          for (int n = 0; n < NR; n++)
#pragma unroll
            for (int s = 0; s < S; s++) acc[u][n * S + s] = fmaf(a[u], b[n][h * S + s], acc[u][n * S + s]);
      }
    }
  }
  const int oc = o0 + ty * OU;
  if (OU % 4 == 0 && O % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0) {
#pragma unroll
    for (int n = 0; n < NR; n++) {
      const int rl = tx + TX * n;
      if (rl >= rcnt || oc >= O) continue;
      float* yr = y + ((r0 + rl) * O + oc) * S;   // OU * S consecutive floats, fewer at the end of the outputs
#pragma unroll
      for (int q = 0; q < OU * S / 4; q++) {
        float4 v;
        v.x = acc[(4 * q) / S][n * S + (4 * q) % S];         v.y = acc[(4 * q + 1) / S][n * S + (4 * q + 1) % S];
        v.z = acc[(4 * q + 2) / S][n * S + (4 * q + 2) % S]; v.w = acc[(4 * q + 3) / S][n * S + (4 * q + 3) % S];
        if (OU == 4 || oc + OU <= O || 4 * q < (O - oc) * S) reinterpret_cast<float4*>(yr)[q] = v;
      }
    }
    return;
  }
  if (OU % 4 != 0) {   // the small tiles
#pragma unroll
    for (int n = 0; n < NR; n++) {
      const int rl = tx + TX * n;
      if (rl >= rcnt) continue;
      float* yr = y + ((r0 + rl) * O + oc) * S;
#pragma unroll
      for (int u = 0; u < OU; u++)
#pragma unroll
        for (int s = 0; s < S; s++)
          if (oc + u < O) yr[u * S + s] = acc[u][n * S + s];
    }
    return;
  }
  // rows that 16-byte words do not fit: through shared memory, some rows at a time, so that a warp stores consecutive
  // floats (stored lane by lane, every 4-byte store of a warp went to 32 sectors; 16384 rows, S = 9, 33 -> 47: 67 -> 41 us)
  const int live = min(TO, O - o0) * S, pitch = live | 1;       // (odd: no bank conflicts)
  const int rp = min(rcnt, (int)(T::BYTES / 4) / pitch);        // rows per pass
  tl_wait<0>();
#pragma unroll 1
  for (int p0 = 0; p0 < rcnt; p0 += rp) {
    __syncthreads();   // the stages, or the rows of the pass before, have been read
#pragma unroll
    for (int n = 0; n < NR; n++) {
      const int rl = tx + TX * n - p0;
      if (rl < 0 || rl >= rp) continue;
      float* at = smem + rl * pitch + ty * OU * S;
#pragma unroll
      for (int u = 0; u < OU; u++)
        if (oc + u < O) {
#pragma unroll
          for (int s = 0; s < S; s++) at[u * S + s] = acc[u][n * S + s];
        }
    }
    __syncthreads();
    const int rows_here = min(rp, rcnt - p0);
    float* yp = y + ((r0 + p0) * O + o0) * S;
    if (O <= TO && live < 32) {   // short rows that follow one another
      for (int f = tid; f < rows_here * live; f += TL_THREADS) {
        const int rl = f / live;
        yp[f] = smem[rl * pitch + f - rl * live];
      }
    } else {
      for (int rl = tid >> 5; rl < rows_here; rl += TL_THREADS / 32)
        for (int i = tid & 31; i < live; i += 32) yp[(long long)rl * O * S + i] = smem[rl * pitch + i];
    }
  }
}

// dW[o, i] = sum_{r, s} dy[r, o, s] * x[r, i, s]. A block computes a TO x TI tile of dW over one slice of rows. Rows are
// staged as they lie in memory; an operand of (channel, s) is read at stride S between lanes (odd: no bank conflicts).
// A thread owns 8 x 8 elements of the tile, so that 64 FMAs stand against 16 shared loads; the KG groups of threads that a
// small tile leaves take the rows of a step in turn and are summed in fixed order at the end.
// nsplit > 1: partial[z][o][i] written, summed afterwards in fixed order (no atomics).
template <int S, int TO, int TI>
struct DwTile {
  static constexpr int TY = TO / 8, TX = TI / 8, G = TY * TX, KG = TL_THREADS / G;
  static constexpr int RMIN = S == 9 ? 4 : (S == 3 ? 8 : 32);
  static constexpr int RK = RMIN > KG ? RMIN : KG;   // rows per step
  static constexpr int AF = RK * TO * S, BF = RK * TI * S;
  static constexpr size_t STAGE = TL_STAGES * sizeof(float) * (AF + BF), RED = sizeof(float) * 64 * G;
  static constexpr size_t BYTES = STAGE > RED ? STAGE : RED;
};

template <int S, int TO, int TI, int VEC>
__global__ void __launch_bounds__(TL_THREADS, 2)
tensor_linear_dw_kernel(const float* __restrict__ dy, const float* __restrict__ x, float* __restrict__ out,
                        long long rows, int I, int O, long long rows_per_split) {
  using T = DwTile<S, TO, TI>;
  constexpr int RK = T::RK, TY = T::TY, TX = T::TX, G = T::G, KG = T::KG;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, grp = tid / G, t = tid % G, tx = t % TX, ty = t / TX;
  const int o0 = blockIdx.y * TO, i0 = blockIdx.x * TI;
  const long long rbeg = (long long)blockIdx.z * rows_per_split;
  const long long rend = (rbeg + rows_per_split < rows) ? rbeg + rows_per_split : rows;
  const int olive = min(TO, O - o0) * S, ilive = min(TI, I - i0) * S;
  float acc[8][8];
#pragma unroll
  for (int u = 0; u < 8; u++)
#pragma unroll
    for (int v = 0; v < 8; v++) acc[u][v] = 0.f;

  auto stage = [&](int buf, long long r) {
    float* as = smem + buf * (T::AF + T::BF);
    const int live = (int)(rend - r < RK ? rend - r : RK);
    tl_rows<VEC, RK, TO * S, TO * S>(as, dy + (r * O + o0) * S, (long long)O * S, live, olive);
    tl_rows<VEC, RK, TI * S, TI * S>(as + T::AF, x + (r * I + i0) * S, (long long)I * S, live, ilive);
    tl_commit();
  };

#pragma unroll
  for (int q = 0; q < TL_STAGES - 1; q++) { if (rbeg + q * RK < rend) stage(q, rbeg + q * RK); else tl_commit(); }
  int k = 0, kn = TL_STAGES - 1;   // buffers of this step and of the one that is staged beside it
  for (long long r = rbeg; r < rend; r += RK) {
    tl_wait<TL_STAGES - 2>();
    __syncthreads();
    if (r + (TL_STAGES - 1) * RK < rend) stage(kn, r + (TL_STAGES - 1) * RK); else tl_commit();
    const float* as = smem + k * (T::AF + T::BF) + ty * S;
    const float* bs = smem + k * (T::AF + T::BF) + T::AF + tx * S;
#pragma unroll 1
    for (int rl = grp; rl < RK; rl += KG) {
      const float* ap = as + rl * (TO * S);
      const float* bp = bs + rl * (TI * S);
#pragma unroll
      for (int s = 0; s < S; s++) {
        float a[8], b[8];
#pragma unroll
        for (int u = 0; u < 8; u++) a[u] = ap[u * TY * S + s];
#pragma unroll
        for (int v = 0; v < 8; v++) b[v] = bp[v * TX * S + s];
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
          for (int v = 0; v < 8; v++) acc[u][v] = fmaf(a[u], b[v], acc[u][v]);
      }
    }
    k = k + 1 < TL_STAGES ? k + 1 : 0;
    kn = kn + 1 < TL_STAGES ? kn + 1 : 0;
  }
  tl_wait<0>();
  __syncthreads();   // the stages hold partial sums from here on
  for (int g = 1; g < KG; g++) {
    if (grp == g) {
#pragma unroll
      for (int u = 0; u < 8; u++)
#pragma unroll
        for (int v = 0; v < 8; v++) smem[(u * 8 + v) * G + t] = acc[u][v];
    }
    __syncthreads();
    if (grp == 0) {
#pragma unroll
      for (int u = 0; u < 8; u++)
#pragma unroll
        for (int v = 0; v < 8; v++) acc[u][v] += smem[(u * 8 + v) * G + t];
    }
    __syncthreads();
  }
  if (grp != 0) return;
  float* dst = out + (size_t)blockIdx.z * O * I;
#pragma unroll
  for (int u = 0; u < 8; u++)
#pragma unroll
    for (int v = 0; v < 8; v++) {
      const int o = o0 + ty + TY * u, i = i0 + tx + TX * v;
      if (o < O && i < I) dst[(size_t)o * I + i] = acc[u][v];
    }
}

// out[i] = sum over z of partial[z][i]: 32 elements per block, eight threads per element take every eighth slice
__global__ void __launch_bounds__(256) sum_partials_kernel(const float* __restrict__ partial, int nsplit, size_t n, float* __restrict__ out) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const size_t i = (size_t)blockIdx.x * 32 + lane;
  float a = 0.f;
  if (i < n)
    for (int z = w; z < nsplit; z += 8) a += partial[(size_t)z * n + i];
  red[w][lane] = a;
  __syncthreads();
  if (w == 0 && i < n) {
#pragma unroll
    for (int q = 1; q < 8; q++) a += red[q][lane];
    out[i] = a;
  }
}

int dw_to(int O) { return O <= 32 ? 32 : 64; }
int dw_ti(int I) { return I <= 32 ? 32 : (I <= 64 ? 64 : 128); }

// slices of the rows: two blocks per SM over all tiles, but at least 64 columns' worth of rows in a slice
int dw_splits(int inds, long long rows, int I, int O) {
  const long long tiles = (long long)ld_cdiv(I, dw_ti(I)) * ld_cdiv(O, dw_to(O));
  const int s = inds == 0 ? 1 : (inds == 1 ? 3 : 9);
  long long want = (148 * 2 + tiles - 1) / tiles;
  const long long maxs = (rows * s + 127) / 128;
  if (want > maxs) want = maxs;
  if (want < 1) want = 1;
  return (int)want;
}

template <int S, int TY, int OU, int NR, int VEC, int PARTS>
int tl_run(const TlWeights& W, const float* x, float* y, long long rows, int I, int O, cudaStream_t st) {
  using T = TlTile<S, TY, OU, NR>;
  if (T::BYTES > 48 * 1024)
    LD_CUDA_TRY(cudaFuncSetAttribute(tensor_linear_kernel<S, TY, OU, NR, VEC, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::BYTES));
  const dim3 g((unsigned)((rows + T::TR - 1) / T::TR), ld_cdiv(O, T::TO));
  tensor_linear_kernel<S, TY, OU, NR, VEC, PARTS><<<g, TL_THREADS, T::BYTES, st>>>(W, x, y, rows, I, O);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

template <int S, int TY, int OU, int NR, int PARTS>
int tl_launch(const TlWeights& W, const float* x, float* y, long long rows, int I, int O, cudaStream_t st) {
  // 8-byte copies need even rows of x on an 8-byte boundary
  if (I % 2 == 0 && ((uintptr_t)x & 7) == 0) return tl_run<S, TY, OU, NR, 2, PARTS>(W, x, y, rows, I, O, st);
  return tl_run<S, TY, OU, NR, 1, PARTS>(W, x, y, rows, I, O, st);
}

// Which tile: 8 outputs x 6 to 9 columns per thread, as many outputs per block as there are (32, 64 or 128) and the rest of
// the threads along the rows, so that x is read once. Where that leaves SMs without a block, tiles of 64 outputs and half the
// accumulators per thread, and where those do as well, tiles of 32 outputs and a quarter of the columns (twice the shared loads
// per FMA, but up to sixteen times the blocks). 128 -> 128 channels: 2048 rows, S = 9, 50 us in small tiles, 32 in the middle
// ones; 16384 rows, S = 1, 49 and 36.
template <int S, int NR, int NR_MID, int NR_SMALL, int PARTS = 1>
int tl_pick(const TlWeights& W, const float* x, float* y, long long rows, int I, int O, cudaStream_t st) {
  const int tr = O <= 32 ? TlTile<S, 4, 8, NR>::TR : (O <= 64 ? TlTile<S, 8, 8, NR>::TR : TlTile<S, 16, 8, NR>::TR);
  const long long blocks = (rows + tr - 1) / tr * (O <= 128 ? 1 : ld_cdiv(O, 128));
  if (blocks >= 148) {
    if (O <= 32) return tl_launch<S, 4, 8, NR, PARTS>(W, x, y, rows, I, O, st);
    if (O <= 64) return tl_launch<S, 8, 8, NR, PARTS>(W, x, y, rows, I, O, st);
    return tl_launch<S, 16, 8, NR, PARTS>(W, x, y, rows, I, O, st);
  }
  constexpr int TR_MID = TlTile<S, 16, 4, NR_MID>::TR;
  if (O > 32 && (rows + TR_MID - 1) / TR_MID * ld_cdiv(O, 64) >= 148) return tl_launch<S, 16, 4, NR_MID, PARTS>(W, x, y, rows, I, O, st);
  return tl_launch<S, 16, 2, NR_SMALL, PARTS>(W, x, y, rows, I, O, st);
}

template <int S, int TO, int TI, int VEC>
int dw_run(const float* dy, const float* x, float* out, long long rows, int I, int O, int ns, cudaStream_t st) {
  using T = DwTile<S, TO, TI>;
  if (T::BYTES > 48 * 1024)
    LD_CUDA_TRY(cudaFuncSetAttribute(tensor_linear_dw_kernel<S, TO, TI, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::BYTES));
  const long long per = (rows + ns - 1) / ns;
  tensor_linear_dw_kernel<S, TO, TI, VEC><<<dim3(ld_cdiv(I, TI), ld_cdiv(O, TO), ns), TL_THREADS, T::BYTES, st>>>(dy, x, out, rows, I, O, per);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

template <int S, int TO, int TI>
int dw_launch(const float* dy, const float* x, float* out, long long rows, int I, int O, int ns, cudaStream_t st) {
  // 16-byte copies need rows of whole 16-byte words on a 16-byte boundary
  if (O % 4 == 0 && I % 4 == 0 && (((uintptr_t)dy | (uintptr_t)x) & 15) == 0) return dw_run<S, TO, TI, 4>(dy, x, out, rows, I, O, ns, st);
  return dw_run<S, TO, TI, 1>(dy, x, out, rows, I, O, ns, st);
}

template <int S>
int dw_pick(const float* dy, const float* x, float* out, long long rows, int I, int O, int ns, cudaStream_t st) {
  const int to = dw_to(O), ti = dw_ti(I);
  if (to == 32) {
    if (ti == 32) return dw_launch<S, 32, 32>(dy, x, out, rows, I, O, ns, st);
    if (ti == 64) return dw_launch<S, 32, 64>(dy, x, out, rows, I, O, ns, st);
    return dw_launch<S, 32, 128>(dy, x, out, rows, I, O, ns, st);
  }
  if (ti == 32) return dw_launch<S, 64, 32>(dy, x, out, rows, I, O, ns, st);
  if (ti == 64) return dw_launch<S, 64, 64>(dy, x, out, rows, I, O, ns, st);
  return dw_launch<S, 64, 128>(dy, x, out, rows, I, O, ns, st);
}

}  // namespace

// inds in {0,1,2}. W[o,i] at W + o*sw0 + i*sw1 (element strides). x:[rows, I, 3^inds], y:[rows, O, 3^inds].
extern "C" int ld_tensor_linear(int inds, const float* W, long long sw0, long long sw1, const float* x, float* y,
                                long long rows, int dim_in, int dim_out, void* stream) {
  if (inds < 0 || inds > 2) { ld_set_last_message("tensor_linear supports up to 2 tensor indices"); return LD_ERR_UNSUPPORTED; }
  if (rows < 0 || dim_in < 0 || dim_out < 0) return LD_ERR_SHAPE;
  if (rows == 0 || dim_out == 0) return LD_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const TlWeights Ws{{W, W, W}, sw0, sw1, dim_out};
  if (inds == 0) return tl_pick<1, 8, 4, 2>(Ws, x, y, rows, dim_in, dim_out, st);
  if (inds == 1) return tl_pick<3, 2, 2, 1>(Ws, x, y, rows, dim_in, dim_out, st);
  return tl_pick<9, 1, 1, 1>(Ws, x, y, rows, dim_in, dim_out, st);
}

// The three channel mixings of PaiNN's Update in one launch, the weights read where they lie: y [rows][3n][3] = (W_l x | W_r x |
// W_v x) for x_v [rows][n][3] and contiguous [n][n] weights.
extern "C" int ld_painn_update_mix(const float* W_l, const float* W_r, const float* W_v, const float* x_v, long long rows, int n, float* y,
                                   void* stream) {
  if (rows < 0 || n <= 0 || n > 0x7fffffff / 3) return LD_ERR_SHAPE;
  if (rows == 0) return LD_OK;
  return tl_pick<3, 2, 2, 1, 3>(TlWeights{{W_l, W_r, W_v}, n, 1, n}, x_v, y, rows, n, 3 * n, (cudaStream_t)stream);
}

extern "C" int ld_tensor_linear_dw_workspace(int inds, long long rows, int dim_in, int dim_out, size_t* bytes) {
  if (inds < 0 || inds > 2 || rows < 0) return LD_ERR_SHAPE;
  int ns = dim_in > 0 && dim_out > 0 ? dw_splits(inds, rows, dim_in, dim_out) : 1;
  *bytes = ns > 1 ? (size_t)ns * dim_in * dim_out * 4 : 0;
  return LD_OK;
}

// dW[o,i] (contiguous [dim_out, dim_in]) = sum_{r,s} dy[r,o,s] x[r,i,s]
extern "C" int ld_tensor_linear_dw(int inds, const float* dy, const float* x, float* dW, long long rows, int dim_in,
                                   int dim_out, void* workspace, size_t workspace_bytes, void* stream) {
  if (inds < 0 || inds > 2) return LD_ERR_UNSUPPORTED;
  if (rows < 0 || dim_in < 0 || dim_out < 0) return LD_ERR_SHAPE;
  if (dim_in == 0 || dim_out == 0) return LD_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (rows == 0) { LD_CUDA_TRY(cudaMemsetAsync(dW, 0, (size_t)dim_in * dim_out * 4, st)); return LD_OK; }
  const int ns = dw_splits(inds, rows, dim_in, dim_out);
  const size_t need = ns > 1 ? (size_t)ns * dim_in * dim_out * 4 : 0;
  if (need > workspace_bytes || (need > 0 && workspace == nullptr)) return LD_ERR_WORKSPACE;
  float* out = ns > 1 ? (float*)workspace : dW;
  int rc;
  if (inds == 0) rc = dw_pick<1>(dy, x, out, rows, dim_in, dim_out, ns, st);
  else if (inds == 1) rc = dw_pick<3>(dy, x, out, rows, dim_in, dim_out, ns, st);
  else rc = dw_pick<9>(dy, x, out, rows, dim_in, dim_out, ns, st);
  if (rc != LD_OK) return rc;
  if (ns > 1) {
    const size_t n = (size_t)dim_in * dim_out;
    sum_partials_kernel<<<(unsigned)((n + 31) / 32), 256, 0, st>>>((const float*)workspace, ns, n, dW);
    LD_LAUNCH_CHECK();
  }
  return LD_OK;
}
