// Device harness of the arithmetic that stands for divisions: the ray setup's
// shear terms (ordinarylight_b200/csrc/olc_trace.cuh) and byte texels
// (olc_textures.cuh), beside the divisions themselves.
#include <cuda_runtime.h>

#include <cstdint>

#include "olc_common.cuh"
#include "olc_trace.cuh"
#include "olc_textures.cuh"

namespace {

__global__ void k_shear(uint32_t n, const float* d, float* got, float* want) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float3 v = make_float3(d[3 * i], d[3 * i + 1], d[3 * i + 2]);
  TraceRay r;
  setup_ray(r, make_float3(0.0f, 0.0f, 0.0f), v);
  const float c[3] = {v.x, v.y, v.z};
  const float z = c[r.kp >> 4];
  got[3 * i] = r.sx;
  got[3 * i + 1] = r.sy;
  got[3 * i + 2] = r.sz;
  want[3 * i] = __fdiv_rn(c[r.kp & 3], z);
  want[3 * i + 1] = __fdiv_rn(c[(r.kp >> 2) & 3], z);
  want[3 * i + 2] = __fdiv_rn(1.0f, z);
}

__global__ void k_bytes(float* got, float* want) {
  got[threadIdx.x] = olc::unorm8(threadIdx.x);
  want[threadIdx.x] = __fdiv_rn((float)threadIdx.x, 255.0f);
}

}  // namespace

// Device arrays: d [n * 3], got and want [n * 3].
extern "C" __attribute__((visibility("default"))) int shear_terms(uint32_t n, const float* d, float* got, float* want) {
  k_shear<<<(n + 255) / 256, 256>>>(n, d, got, want);
  return (int)cudaDeviceSynchronize();
}

// Device arrays: got and want [256].
extern "C" __attribute__((visibility("default"))) int byte_texels(float* got, float* want) {
  k_bytes<<<1, 256>>>(got, want);
  return (int)cudaDeviceSynchronize();
}
