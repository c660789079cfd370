// Geometry of an edge in the FP32 kernels of the l<=2 message layer.
#pragma once
#include <cuda_runtime.h>
#include "tp_math.h"

namespace {

// per-edge geometry shared by all channels: rhat[3] and the eight radial features
struct __align__(16) EdgeGeom { float enc[8]; float rhat[3]; float pad; };   // 48 bytes: three 16-byte shared-memory loads

__device__ __forceinline__ void edge_geometry(const float* __restrict__ rij, long long e, float r0,
                                              const float* __restrict__ jac, EdgeGeom* g) {
  const float x = rij[e * 3], y = rij[e * 3 + 1], z = rij[e * 3 + 2];
  const float d = sqrtf(x * x + y * y + z * z);
  const float zz = d / r0;
  const float env = fmaxf(1.f - zz, 0.f);
  ld_radial_cheb8(zz, env, jac, g->enc);
  const float s = 7.f / r0;
  const float ux = x * s, uy = y * s, uz = z * s;
  const float inv = 1.0f / sqrtf(1.f + ux * ux + uy * uy + uz * uz);
  g->rhat[0] = ux * inv; g->rhat[1] = uy * inv; g->rhat[2] = uz * inv;
}

}  // namespace
