// The node-level parts of the PaiNN block, FP32: the three-layer MLPs on rows (archs/meanflow_painn8.py:38-51) and the
// pointwise halves of Update (:53-75).
#include "common.cuh"
#include "mlp_tile.cuh"

namespace {

constexpr int MR_THREADS = 512;

struct MlpRows {
  const float* W[3];   // [in][out]
  const float* b[3];
  const float* Wd;     // optional direct term [k0][n3]
  int k0, n1, n2, n3;
};

// One block: R rows through all three layers, activations in shared memory as [k][R]. Weights are read straight from L2, each
// once per block, by 16-byte loads: a thread has four columns of all R rows and every KG-th k (KG = 512 / (N / 4) groups of
// threads, so that a narrow layer still has 512 loads in flight), and the groups' sums are added up in shared memory.
// Bound by the loads of the weights at few rows (64 -> 256 -> 256 -> 256 on 512 rows: 11.7 us; a tile of 32 rows per block, 16
// blocks, took 68) and by the FMA pipe at many (2048 rows, 128 -> 512 -> 512 -> 512: 83 us against 206).
template <int R, bool ALIGNED = true>
__device__ __forceinline__ void mr_accumulate(const float* __restrict__ in, int K, const float* __restrict__ W, int N, int g, int KG, int c4,
                                              float (&acc)[4][R]) {
#pragma unroll 4
  for (int k = g; k < K; k += KG) {
    const float* wp = W + (size_t)k * N + c4;
    const float4 w = ALIGNED ? __ldg(reinterpret_cast<const float4*>(wp)) : make_float4(__ldg(wp), __ldg(wp + 1), __ldg(wp + 2), __ldg(wp + 3));
#pragma unroll
    for (int r = 0; r < R; r += 4) {
      const float4 h = *reinterpret_cast<const float4*>(in + k * R + r);
      const float hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        acc[0][r + q] = fmaf(w.x, hv[q], acc[0][r + q]); acc[1][r + q] = fmaf(w.y, hv[q], acc[1][r + q]);
        acc[2][r + q] = fmaf(w.z, hv[q], acc[2][r + q]); acc[3][r + q] = fmaf(w.w, hv[q], acc[3][r + q]);
      }
    }
  }
}

template <int R>
__global__ void __launch_bounds__(MR_THREADS, 1)
mlp3_rows_kernel(const float* __restrict__ x, long long rows, MlpRows m, int act, float* __restrict__ out) {
  extern __shared__ __align__(16) float smem[];
  float* xs = smem;                          // [k0][R]
  float* h1 = xs + (size_t)m.k0 * R;         // [n1][R]
  float* h2 = h1 + (size_t)m.n1 * R;         // [n2][R]
  float* part = h2 + (size_t)m.n2 * R;       // [KG][R][N]
  const int tid = threadIdx.x;
  const long long r0 = (long long)blockIdx.x * R;
  const int live = (int)(rows - r0 < R ? rows - r0 : R);
  for (int i = tid; i < R * m.k0; i += MR_THREADS) {
    const int r = i / m.k0, k = i - r * m.k0;
    xs[k * R + r] = r < live ? x[(r0 + r) * m.k0 + k] : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int layer = 0; layer < 3; layer++) {
    const float* in = layer == 0 ? xs : (layer == 1 ? h1 : h2);
    const int K = layer == 0 ? m.k0 : (layer == 1 ? m.n1 : m.n2), N = layer == 0 ? m.n1 : (layer == 1 ? m.n2 : m.n3);
    const int CT = N >> 2, KG = MR_THREADS / CT, g = tid / CT, c4 = (tid - g * CT) * 4;
    if (g < KG) {
      float acc[4][R];
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int r = 0; r < R; r++) acc[j][r] = 0.f;
      mr_accumulate<R>(in, K, m.W[layer], N, g, KG, c4, acc);
      if (layer == 2 && m.Wd != nullptr) {
        if ((reinterpret_cast<uintptr_t>(m.Wd) & 15) == 0) mr_accumulate<R>(xs, m.k0, m.Wd, N, g, KG, c4, acc);
        else mr_accumulate<R, false>(xs, m.k0, m.Wd, N, g, KG, c4, acc);
      }
#pragma unroll
      for (int r = 0; r < R; r++)
        *reinterpret_cast<float4*>(part + ((size_t)g * R + r) * N + c4) = make_float4(acc[0][r], acc[1][r], acc[2][r], acc[3][r]);
    }
    __syncthreads();
    float* h = layer == 0 ? h1 : h2;
    for (int i = tid; i < R * N; i += MR_THREADS) {
      const int r = i / N, c = i - r * N;
      float v = m.b[layer] != nullptr ? m.b[layer][c] : 0.f;
      float a = 0.f;
      for (int q = 0; q < KG; q++) a += part[((size_t)q * R + r) * N + c];
      v = a + v;
      if (layer < 2) h[c * R + r] = mt_act(v, act);
      else if (r < live) out[(r0 + r) * N + c] = v;
    }
    __syncthreads();
  }
}

int check_widths(const MlpRows& m) {
  const int dims[3] = {m.n1, m.n2, m.n3};
  for (int i = 0; i < 3; i++) {
    if (dims[i] <= 0 || dims[i] % 8 != 0) { ld_set_last_message("mlp: layer widths must be positive multiples of 8"); return LD_ERR_UNSUPPORTED; }
    if (dims[i] > 512) { ld_set_last_message("mlp (FP32 path): widths above 512 are not supported"); return LD_ERR_UNSUPPORTED; }
  }
  if (m.k0 <= 0 || m.k0 > 512) { ld_set_last_message("mlp (FP32 path): widths above 512 are not supported"); return LD_ERR_UNSUPPORTED; }
  if ((((uintptr_t)m.W[0] | (uintptr_t)m.W[1] | (uintptr_t)m.W[2]) % 16) != 0) {
    ld_set_last_message("mlp: packed weights must be 16-byte aligned");
    return LD_ERR_SHAPE;
  }
  return LD_OK;
}

template <int R>
int mr_launch(const float* x, long long rows, const MlpRows& m, int act, float* out, cudaStream_t st) {
  const size_t smem = sizeof(float) * R * ((size_t)m.k0 + m.n1 + m.n2 + 4 * MR_THREADS);
  LD_CUDA_TRY(cudaFuncSetAttribute(mlp3_rows_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  mlp3_rows_kernel<R><<<(unsigned)((rows + R - 1) / R), MR_THREADS, smem, st>>>(x, rows, m, act, out);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

// y [rows][3n][3]: the three channel mixings of x_v, stacked (left, right, value)
__global__ void __launch_bounds__(256) update_front_kernel(const float* __restrict__ y, const float* __restrict__ x_a, long long total, int n,
                                                           float* __restrict__ inner, float* __restrict__ cat) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const long long row = i / n;
  const int c = (int)(i - row * n);
  const float* l = y + (row * 3 * n + c) * 3;
  const float* r = l + (size_t)n * 3;
  const float r0 = r[0], r1 = r[1], r2 = r[2];
  inner[i] = l[0] * r0 + l[1] * r1 + l[2] * r2;
  cat[row * 2 * n + c] = x_a[i];
  cat[row * 2 * n + n + c] = sqrtf(r0 * r0 + r1 * r1 + r2 * r2);
}

__global__ void __launch_bounds__(256) update_back_kernel(const float* __restrict__ y, const float* __restrict__ m, const float* __restrict__ inner,
                                                          const float* __restrict__ x_a, const float* __restrict__ x_v, long long total, int n,
                                                          float* __restrict__ scaled, float* __restrict__ base, float* __restrict__ out_v) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const long long row = i / n;
  const int c = (int)(i - row * n);
  const float* v = y + (row * 3 * n + 2 * n + c) * 3;
  const float* mr = m + row * 3 * n + c;
  const float s = mr[0], v0 = v[0] * s, v1 = v[1] * s, v2 = v[2] * s;
  const float d = sqrtf(1.f + (v0 * v0 + v1 * v1 + v2 * v2));
  out_v[i * 3] = x_v[i * 3] + v0 / d; out_v[i * 3 + 1] = x_v[i * 3 + 1] + v1 / d; out_v[i * 3 + 2] = x_v[i * 3 + 2] + v2 / d;
  scaled[i] = inner[i] * mr[n];
  base[i] = x_a[i] + mr[2 * n];
}

}  // namespace

// Three dense layers on `rows` rows. Weights are passed transposed ("packed"): Wkt is [in][out]
// contiguous, i.e. nn.Linear.weight.t().contiguous(). act: 0 none, 1 SiLU, 2 LeakyReLU(0.1),
// applied after layers 1 and 2. Wdt (optional, [k0][n3], of any alignment) adds a direct linear term x*Wd.
extern "C" int ld_mlp3_rows(const float* x, long long rows, int k0, const float* W1t, const float* b1, int n1,
                            const float* W2t, const float* b2, int n2, const float* W3t, const float* b3, int n3, int act,
                            const float* Wdt, float* out, void* stream) {
  if (rows < 0) return LD_ERR_SHAPE;
  const MlpRows m{{W1t, W2t, W3t}, {b1, b2, b3}, Wdt, k0, n1, n2, n3};
  const int rc = check_widths(m);
  if (rc != LD_OK) return rc;
  if (rows == 0) return LD_OK;
  cudaStream_t st = (cudaStream_t)stream;
  // few rows: more blocks; many: more FMAs per weight that is loaded
  if (rows <= 4 * 148) return mr_launch<4>(x, rows, m, act, out, st);
  if (rows <= 8 * 148) return mr_launch<8>(x, rows, m, act, out, st);
  return mr_launch<16>(x, rows, m, act, out, st);
}

// The pointwise halves of PaiNN's Update on rows of n channels. y [rows][3n][3] holds the three channel mixings of x_v
// (lin_l, lin_r, lin_v). Front: inner [rows][n] = l . r, cat [rows][2n] = (x_a | |r|), the input of the update's MLP.
extern "C" int ld_painn_update_front(const float* y, const float* x_a, long long rows, int n, float* inner, float* cat, void* stream) {
  if (rows < 0 || n <= 0) return LD_ERR_SHAPE;
  const long long total = rows * n;
  if (total == 0) return LD_OK;
  update_front_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(y, x_a, total, n, inner, cat);
  LD_LAUNCH_CHECK();
  return LD_OK;
}

// Back, with m [rows][3n] = the MLP's output: out_v = x_v + u / sqrt(1 + |u|^2) for u = v * m[:n], scaled = inner * m[n:2n] (what the
// group norm is taken of), base = x_a + m[2n:] (what it is added to).
extern "C" int ld_painn_update_back(const float* y, const float* m, const float* inner, const float* x_a, const float* x_v, long long rows, int n,
                                    float* scaled, float* base, float* out_v, void* stream) {
  if (rows < 0 || n <= 0) return LD_ERR_SHAPE;
  const long long total = rows * n;
  if (total == 0) return LD_OK;
  update_back_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(y, m, inner, x_a, x_v, total, n, scaled, base, out_v);
  LD_LAUNCH_CHECK();
  return LD_OK;
}
