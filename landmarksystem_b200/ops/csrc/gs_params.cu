// Per-Gaussian parameter passes around the rasteriser: activations (exp of the log-scales, unit quaternions, sigmoid of the
// opacity logits) with their backward, and the densification statistics of a step.
//
// Each replaces a chain of tensor operations (activations 7 forward and 16 backward launches; statistics 11 launches that
// gather by a boolean mask and wait for its count on the host).  All are bound by memory: 32 B in and 32 B out per Gaussian
// forward, 96 B backward.  IEEE arithmetic: the activated values feed the projection.
#include "common.cuh"

namespace lmb {

constexpr int kParamThreads = 256;
constexpr float kNormEps = 1e-12f;       // floor of the quaternion norm

// scaling rows are elementwise, so a thread takes elements i, i + N, i + 2N of them and row i of the others
__global__ void __launch_bounds__(kParamThreads)
gs_activate_kernel(long long N, const float* __restrict__ scaling, const float4* __restrict__ rotation,
                   const float* __restrict__ opacity, float* __restrict__ scales, float4* __restrict__ quats,
                   float* __restrict__ alphas) {
  const long long i = (long long)blockIdx.x * kParamThreads + threadIdx.x;
  if (i >= N) return;
#pragma unroll
  for (int k = 0; k < 3; ++k) scales[k * N + i] = expf(scaling[k * N + i]);
  const float4 q = rotation[i];
  const float n = sqrtf(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
  const float d = n < kNormEps ? kNormEps : n;
  quats[i] = make_float4(q.x / d, q.y / d, q.z / d, q.w / d);
  alphas[i] = 1.f / (1.f + expf(-opacity[i]));
}

// d/dx exp = exp; d/dq (q / |q|) = (g - u (u.g)) / |q|, without the second term where the floor holds; s (1 - s)
__global__ void __launch_bounds__(kParamThreads)
gs_activate_bwd_kernel(long long N, const float* __restrict__ scales, const float4* __restrict__ rotation,
                       const float* __restrict__ alphas, const float* __restrict__ d_scales, const float4* __restrict__ d_quats,
                       const float* __restrict__ d_alphas, float* __restrict__ d_scaling, float4* __restrict__ d_rotation,
                       float* __restrict__ d_opacity) {
  const long long i = (long long)blockIdx.x * kParamThreads + threadIdx.x;
  if (i >= N) return;
#pragma unroll
  for (int k = 0; k < 3; ++k) d_scaling[k * N + i] = d_scales[k * N + i] * scales[k * N + i];
  const float4 q = rotation[i], g = d_quats[i];
  const float n = sqrtf(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
  const bool floored = n < kNormEps;
  const float inv = 1.f / (floored ? kNormEps : n);
  const float4 u = make_float4(q.x * inv, q.y * inv, q.z * inv, q.w * inv);
  const float dot = floored ? 0.f : u.x * g.x + u.y * g.y + u.z * g.z + u.w * g.w;
  d_rotation[i] = make_float4((g.x - u.x * dot) * inv, (g.y - u.y * dot) * inv, (g.z - u.z * dot) * inv, (g.w - u.w * dot) * inv);
  d_opacity[i] = d_alphas[i] * (alphas[i] * (1.f - alphas[i]));
}

__global__ void __launch_bounds__(kParamThreads)
gs_view_stats_kernel(long long N, const unsigned char* __restrict__ visible, const int* __restrict__ radii,
                     const float* __restrict__ d_means2D, float* __restrict__ max_radii, float* __restrict__ grad_accum,
                     float* __restrict__ denom) {
  const long long i = (long long)blockIdx.x * kParamThreads + threadIdx.x;
  if (i >= N || !visible[i]) return;
  const float r = (float)radii[i], m = max_radii[i];
  max_radii[i] = m < r ? r : m;
  const float gx = d_means2D[3 * i], gy = d_means2D[3 * i + 1];
  grad_accum[i] += sqrtf(gx * gx + gy * gy);
  denom[i] += 1.f;
}

}  // namespace lmb

using namespace lmb;

// scaling, scales: [N, 3]; rotation, quats: [N, 4], 16-byte aligned; opacity, alphas: [N, 1]
LMB_API int lmb_gs_activate(long long N, const float* scaling, const float* rotation, const float* opacity, float* scales,
                            float* quats, float* alphas, cudaStream_t stream) {
  if (N <= 0) return 0;
  gs_activate_kernel<<<ceil_div(N, kParamThreads), kParamThreads, 0, stream>>>(N, scaling, (const float4*)rotation, opacity, scales,
                                                                              (float4*)quats, alphas);
  LMB_LAUNCH_CHECK();
  return 0;
}

LMB_API int lmb_gs_activate_bwd(long long N, const float* scales, const float* rotation, const float* alphas, const float* d_scales,
                                const float* d_quats, const float* d_alphas, float* d_scaling, float* d_rotation, float* d_opacity,
                                cudaStream_t stream) {
  if (N <= 0) return 0;
  gs_activate_bwd_kernel<<<ceil_div(N, kParamThreads), kParamThreads, 0, stream>>>(N, scales, (const float4*)rotation, alphas, d_scales,
      (const float4*)d_quats, d_alphas, d_scaling, (float4*)d_rotation, d_opacity);
  LMB_LAUNCH_CHECK();
  return 0;
}

// visible: [N] bytes; d_means2D: [N, 3]; max_radii, grad_accum, denom: [N], updated where visible
LMB_API int lmb_gs_view_stats(long long N, const unsigned char* visible, const int* radii, const float* d_means2D, float* max_radii,
                              float* grad_accum, float* denom, cudaStream_t stream) {
  if (N <= 0) return 0;
  gs_view_stats_kernel<<<ceil_div(N, kParamThreads), kParamThreads, 0, stream>>>(N, visible, radii, d_means2D, max_radii, grad_accum,
                                                                                denom);
  LMB_LAUNCH_CHECK();
  return 0;
}
