// Proposal networks of Nerfacto: scene contraction, hash-grid lookup, two-layer perceptron and truncated exponential in one
// kernel, forward and backward (the reference: landmark/nerf_components/ray_samplers/proposal_network_sampler.py, with
// tiny-cuda-nn networks).  All fp32, as the tensor operations they replace.
//
// A proposal level evaluates 256 + 96 samples per ray.  As tensor operations that was 40 launches per network, each moving
// 4 - 40 bytes per sample through memory (4.2 M samples at 16 k rays: contraction 20 passes over [N, 3], features and hidden
// layer written and read, two fp32 GEMMs of width 16); here a sample is 12 B in and 4 B out, features and hidden units stay in
// registers, and the kernel is bound by its 40 gathers per sample from an L2-resident
// table.  16384-ray Nerfacto step, per step: forward 1.8 ms of tensor operations -> 0.26 ms, backward (every other step there)
// 0.41 ms; the step 7309 -> 6133 us.  Spacing and middles as kernels:
// 5300 -> 4757 us (250 -> 195 launches).
#include "hashgrid.cuh"

namespace lmb {

constexpr int kPropThreads = 256;
constexpr int kPropHidden = 16;
constexpr int kPropMaxLevels = 8;

struct UnitMap {
  const float* box;    // device, {low corner, high corner}, or null: position -> [0, 1], or [-1, 1] before a contraction
  int contract;        // L-infinity contraction onto the cube of half-width 2, then to [0, 1]
};

// Coordinate in the unit cube, zeroed outside of it.
__device__ __forceinline__ bool unit_position(const UnitMap& u, const float* __restrict__ p, float* x) {
#pragma unroll
  for (int d = 0; d < 3; ++d) x[d] = u.box ? (p[d] - __ldg(u.box + d)) / (__ldg(u.box + 3 + d) - __ldg(u.box + d)) : p[d];
  if (u.contract) {
    if (u.box) {
#pragma unroll
      for (int d = 0; d < 3; ++d) x[d] = x[d] * 2.f - 1.f;
    }
    const float mag = fmaxf(fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fabsf(x[2])), 1e-9f);
    const float k = 2.f - 1.f / mag;
#pragma unroll
    for (int d = 0; d < 3; ++d) x[d] = ((mag <= 1.f ? x[d] : k * (x[d] / mag)) + 2.f) / 4.f;
  }
  const bool inside = x[0] > 0.f && x[0] < 1.f && x[1] > 0.f && x[1] < 1.f && x[2] > 0.f && x[2] < 1.f;
#pragma unroll
  for (int d = 0; d < 3; ++d) x[d] *= inside ? 1.f : 0.f;
  return inside;
}

__global__ void __launch_bounds__(kPropThreads)
unit_position_kernel(long long n, const float* __restrict__ pos, UnitMap u, float* __restrict__ out, unsigned char* __restrict__ inside) {
  const long long i = (long long)blockIdx.x * kPropThreads + threadIdx.x;
  if (i >= n) return;
  float x[3];
  inside[i] = unit_position(u, pos + 3 * i, x);
#pragma unroll
  for (int d = 0; d < 3; ++d) out[3 * i + d] = x[d];
}

// Spacing coordinate s in [0, 1] -> distance: x = s far + (1 - s) near, then 2 x below one half and 1 / (2 - 2 x) above.  Every
// product and sum is rounded by itself, as the tensor operations do (nine launches per set of bins).
__global__ void __launch_bounds__(kPropThreads)
spacing_kernel(long long n, const float* __restrict__ s, float near, float far, float* __restrict__ out) {
  const long long i = (long long)blockIdx.x * kPropThreads + threadIdx.x;
  if (i >= n) return;
  const float x = __fadd_rn(__fmul_rn(s[i], far), __fmul_rn(__fsub_rn(1.f, s[i]), near));
  out[i] = x < 0.5f ? 2.f * x : __fdiv_rn(1.f, __fsub_rn(2.f, 2.f * x));
}

// Middle of interval k of ray r as a point; rows of starts and ends are `stride` apart
__global__ void __launch_bounds__(kPropThreads)
midpoints_kernel(long long n, int S, const float* __restrict__ o, const float* __restrict__ d, const float* __restrict__ starts,
                 const float* __restrict__ ends, long long stride, float* __restrict__ out) {
  const long long i = (long long)blockIdx.x * kPropThreads + threadIdx.x;
  if (i >= n) return;
  const long long r = div_index(i, S), k = i - r * S;
  const float mid = 0.5f * __fadd_rn(starts[r * stride + k], ends[r * stride + k]);
#pragma unroll
  for (int c = 0; c < 3; ++c) out[3 * i + c] = __fadd_rn(o[3 * r + c], __fmul_rn(d[3 * r + c], mid));
}

// features of kL levels (two per level) at x
template <int kL>
__device__ __forceinline__ void lookup(const HashMeta& m, const float* __restrict__ table, const float* x, float* f) {
#pragma unroll
  for (int l = 0; l < kL; ++l) {
    f[2 * l] = f[2 * l + 1] = 0.f;
    if (l >= m.n_levels) continue;
    const LevelIndex index((uint32_t)m.res[l], (uint32_t)(m.offset[l + 1] - m.offset[l]));
    const float2* tab = reinterpret_cast<const float2*>(table) + m.offset[l];
    float w[3];
    uint32_t p0[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float p = x[d] * m.scale[l] + 0.5f;
      const float fl = floorf(p);
      w[d] = p - fl;
      p0[d] = (uint32_t)max((int)fl, 0);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint32_t ix = min(p0[0] + (c & 1), index.res - 1), iy = min(p0[1] + ((c >> 1) & 1), index.res - 1),
                     iz = min(p0[2] + ((c >> 2) & 1), index.res - 1);
      const float wt = ((c & 1) ? w[0] : 1.f - w[0]) * ((c & 2) ? w[1] : 1.f - w[1]) * ((c & 4) ? w[2] : 1.f - w[2]);
      const float2 e = __ldg(tab + index(ix, iy, iz));
      f[2 * l] += wt * e.x; f[2 * l + 1] += wt * e.y;
    }
  }
}

// first-layer rows padded to 2 kL columns (zeros behind the real ones), then the second layer
template <int kL>
struct PropWeights { float w1[kPropHidden][2 * kL]; float w2[kPropHidden]; };

template <int kL>
__device__ __forceinline__ void load_weights(PropWeights<kL>& s, const float* __restrict__ w1, const float* __restrict__ w2, int n_feat) {
  for (int i = threadIdx.x; i < kPropHidden * 2 * kL; i += kPropThreads) {
    const int j = i / (2 * kL), k = i % (2 * kL);
    s.w1[j][k] = k < n_feat ? w1[j * n_feat + k] : 0.f;
  }
  if (threadIdx.x < kPropHidden) s.w2[threadIdx.x] = w2[threadIdx.x];
  __syncthreads();
}

// hidden units after relu (a unit that is not a number stays one), and the output
template <int kL>
__device__ __forceinline__ float perceptron(const PropWeights<kL>& s, const float* f, float* h) {
  float raw = 0.f;
#pragma unroll
  for (int j = 0; j < kPropHidden; ++j) {
    float a = 0.f;
#pragma unroll
    for (int k = 0; k < 2 * kL; ++k) a += f[k] * s.w1[j][k];
    h[j] = a < 0.f ? 0.f : a;
    raw += h[j] * s.w2[j];
  }
  return raw;
}

template <int kL>
__global__ void __launch_bounds__(kPropThreads)
prop_density_kernel(long long n, const float* __restrict__ pos, UnitMap u, HashMeta m, const float* __restrict__ table,
                    const float* __restrict__ w1, const float* __restrict__ w2, float* __restrict__ density) {
  __shared__ __align__(16) PropWeights<kL> s;
  load_weights(s, w1, w2, 2 * m.n_levels);
  const long long i = (long long)blockIdx.x * kPropThreads + threadIdx.x;
  if (i >= n) return;
  float x[3], f[2 * kL], h[kPropHidden];
  const bool inside = unit_position(u, pos + 3 * i, x);
  lookup<kL>(m, table, x, f);
  density[i] = expf(perceptron<kL>(s, f, h)) * (inside ? 1.f : 0.f);
}

// Gradients of the features (for the table's own backward kernel) and of the weights.  A thread recomputes its sample; the
// weight gradients, a product over samples, go through shared memory: 8 groups of 4 x kL outputs, 32 slices of 8 samples per
// round, summed in registers across the rounds of a persistent block.
template <int kL>
__global__ void __launch_bounds__(kPropThreads, 2)
prop_density_bwd_kernel(long long n, const float* __restrict__ pos, UnitMap u, HashMeta m, const float* __restrict__ table,
                        const float* __restrict__ w1, const float* __restrict__ w2, const float* __restrict__ d_density,
                        float* __restrict__ unit, float* __restrict__ d_feat, float* __restrict__ d_w1, float* __restrict__ d_w2) {
  __shared__ __align__(16) PropWeights<kL> s;
  __shared__ float s_dh[kPropThreads][kPropHidden + 1], s_f[kPropThreads][2 * kL + 1];
  const int n_feat = 2 * m.n_levels, t = threadIdx.x;
  load_weights(s, w1, w2, n_feat);
  const int j0 = (t & 3) * 4, k0 = (t >> 2 & 1) * kL, slice = t >> 3;
  float g1[4][kL], g2[kPropHidden];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < kL; ++k) g1[j][k] = 0.f;
#pragma unroll
  for (int j = 0; j < kPropHidden; ++j) g2[j] = 0.f;
  for (long long base = (long long)blockIdx.x * kPropThreads; base < n; base += (long long)gridDim.x * kPropThreads) {
    const long long i = base + t;
    float f[2 * kL], h[kPropHidden], draw = 0.f;
#pragma unroll
    for (int k = 0; k < 2 * kL; ++k) f[k] = 0.f;
#pragma unroll
    for (int j = 0; j < kPropHidden; ++j) h[j] = 0.f;
    if (i < n) {
      float x[3];
      const bool inside = unit_position(u, pos + 3 * i, x);
#pragma unroll
      for (int d = 0; d < 3; ++d) unit[3 * i + d] = x[d];
      lookup<kL>(m, table, x, f);
      const float raw = perceptron<kL>(s, f, h);
      draw = d_density[i] * (inside ? 1.f : 0.f) * expf(fminf(fmaxf(raw, -15.f), 15.f));
    }
    asm volatile("" ::: "memory");                    // read the weights again rather than keep all of them in registers
    float df[2 * kL];
#pragma unroll
    for (int k = 0; k < 2 * kL; ++k) { df[k] = 0.f; s_f[t][k] = f[k]; }
#pragma unroll
    for (int j = 0; j < kPropHidden; ++j) {
      g2[j] += draw * h[j];
      const float dh = h[j] > 0.f ? draw * s.w2[j] : 0.f;
      s_dh[t][j] = dh;
#pragma unroll
      for (int k = 0; k < 2 * kL; ++k) df[k] += dh * s.w1[j][k];
    }
    if (i < n) {
#pragma unroll
      for (int k = 0; k < 2 * kL; ++k)
        if (k < n_feat) d_feat[i * n_feat + k] = df[k];
    }
    __syncthreads();
#pragma unroll 1
    for (int r = 0; r < kPropThreads / 32; ++r) {
      const int q = r * 32 + slice;
      float a[4], b[kL];
#pragma unroll
      for (int j = 0; j < 4; ++j) a[j] = s_dh[q][j0 + j];
#pragma unroll
      for (int k = 0; k < kL; ++k) b[k] = s_f[q][k0 + k];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int k = 0; k < kL; ++k) g1[j][k] += a[j] * b[k];
    }
    __syncthreads();
  }
  // lanes of a warp that hold the same outputs (every 8th) sum first
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < kL; ++k) {
      float v = g1[j][k];
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      if ((t & 31) < 8 && k0 + k < n_feat) atomicAdd(d_w1 + (j0 + j) * n_feat + k0 + k, v);
    }
#pragma unroll
  for (int j = 0; j < kPropHidden; ++j) {
    float v = g2[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((t & 31) == 0) atomicAdd(d_w2 + j, v);
  }
}

}  // namespace lmb

using namespace lmb;

// pos: [n, 3]; box: device [2, 3] or null; out: [n, 3]; inside: [n] bytes
LMB_API int lmb_unit_position(long long n, const float* pos, const float* box, int contract, float* out, unsigned char* inside, cudaStream_t stream) {
  if (n <= 0) return 0;
  unit_position_kernel<<<ceil_div(n, kPropThreads), kPropThreads, 0, stream>>>(n, pos, UnitMap{box, contract}, out, inside);
  LMB_LAUNCH_CHECK();
  return 0;
}

// near, far: spacing coordinates of the range's ends
LMB_API int lmb_spacing_to_euclid(long long n, const float* s, float near, float far, float* out, cudaStream_t stream) {
  if (n <= 0) return 0;
  spacing_kernel<<<ceil_div(n, kPropThreads), kPropThreads, 0, stream>>>(n, s, near, far, out);
  LMB_LAUNCH_CHECK();
  return 0;
}

// o, d: [R, 3]; starts, ends: [R, S] with rows `stride` floats apart; out: [R, S, 3]
LMB_API int lmb_midpoints(long long R, int S, const float* o, const float* d, const float* starts, const float* ends, long long stride,
                          float* out, cudaStream_t stream) {
  if (R <= 0 || S <= 0) return 0;
  midpoints_kernel<<<ceil_div(R * S, kPropThreads), kPropThreads, 0, stream>>>(R * S, S, o, d, starts, ends, stride, out);
  LMB_LAUNCH_CHECK();
  return 0;
}

// table: fp32, two features per entry, on 8 bytes; w1: [16, 2 n_levels]; w2: [16]; density: [n]
LMB_API int lmb_prop_density(long long n, const float* pos, const float* box, int contract, const HashMeta* meta, const float* table,
                             const float* w1, const float* w2, float* density, cudaStream_t stream) {
  if (meta->n_features != 2 || meta->n_levels < 1 || meta->n_levels > kPropMaxLevels) return (int)cudaErrorInvalidValue;
  if (n <= 0) return 0;
  const auto kernel = meta->n_levels <= 5 ? prop_density_kernel<5> : prop_density_kernel<kPropMaxLevels>;
  kernel<<<ceil_div(n, kPropThreads), kPropThreads, 0, stream>>>(n, pos, UnitMap{box, contract}, *meta, table, w1, w2, density);
  LMB_LAUNCH_CHECK();
  return 0;
}

// unit: [n, 3] and d_feat: [n, 2 n_levels], written, for lmb_hashgrid_bwd; d_w1, d_w2: added to
LMB_API int lmb_prop_density_bwd(long long n, const float* pos, const float* box, int contract, const HashMeta* meta, const float* table,
                                 const float* w1, const float* w2, const float* d_density, float* unit, float* d_feat, float* d_w1,
                                 float* d_w2, cudaStream_t stream) {
  if (meta->n_features != 2 || meta->n_levels < 1 || meta->n_levels > kPropMaxLevels) return (int)cudaErrorInvalidValue;
  if (n <= 0) return 0;
  const auto kernel = meta->n_levels <= 5 ? prop_density_bwd_kernel<5> : prop_density_bwd_kernel<kPropMaxLevels>;
  const int blocks = ceil_div(n, kPropThreads);
  kernel<<<blocks < 148 * 4 ? blocks : 148 * 4, kPropThreads, 0, stream>>>(n, pos, UnitMap{box, contract}, *meta, table, w1, w2, d_density, unit, d_feat,
                                                                          d_w1, d_w2);
  LMB_LAUNCH_CHECK();
  return 0;
}
