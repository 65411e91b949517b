// Marched samples as rows: a ray's samples are consecutive rows of compact arrays, offsets[r] .. offsets[r + 1].
//
//  * row_index_kernel      counts -> flat slot (ray * S + s) of every row, in order
//  * rows_composite_*      weights, colour and depth of the rays straight from the rows, forward and backward
//
// The padded [R, S] form of the same math scattered densities and colours into cleared arrays, evaluated weights and
// composite over all slots and gathered the gradients back: 1.3 ms of an 18.5 ms Instant-NGP step of 131072 rays, and a
// dozen launches per rendered chunk.  Rows are summed in the order in which the padded kernels (composite.cu) sum a compacted ray, so the
// results are the same bits.  One warp per ray; bound by memory (4 + 12 B a row in, the same out in the backward).
#include "common.cuh"

namespace lmb {

constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ float excl_prod(float v, float& total) {
  float x = v;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const float y = __shfl_up_sync(kAll, x, d);
    if (lane >= d) x *= y;
  }
  total = __shfl_sync(kAll, x, 31);
  const float e = __shfl_up_sync(kAll, x, 1);
  return lane == 0 ? 1.f : e;
}
__device__ __forceinline__ float incl_sum(float v, float& total) {
  float x = v;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const float y = __shfl_up_sync(kAll, x, d);
    if (lane >= d) x += y;
  }
  total = __shfl_sync(kAll, x, 31);
  return x;
}
__device__ __forceinline__ float all_sum(float v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(kAll, v, d);
  return v;
}

__global__ void __launch_bounds__(256)
row_index_kernel(int R, int S, const int* __restrict__ offsets, long long* __restrict__ idx) {
  const int ray = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (ray >= R) return;
  const int first = offsets[ray], n = offsets[ray + 1] - first;
  for (int s = threadIdx.x & 31; s < n; s += 32) idx[(long long)first + s] = (long long)ray * S + s;
}

// alpha of row s of a ray
__device__ __forceinline__ float row_alpha(float sigma, float t0, float t1) { return 1.f - __expf(-sigma * (t1 - t0)); }

__global__ void __launch_bounds__(256)
rows_composite_kernel(int R, int S, const int* __restrict__ offsets, const float* __restrict__ sigma, const float* __restrict__ rgb,
                      const float* __restrict__ ts, const float* __restrict__ te, float bg, float* __restrict__ out_rgb,
                      float* __restrict__ out_depth) {
  const int ray = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (ray >= R) return;
  const long long first = offsets[ray], slot = (long long)ray * S;
  const int n = offsets[ray + 1] - (int)first;
  float carry = 1.f, r = 0.f, g = 0.f, b = 0.f, depth = 0.f, acc = 0.f;
  for (int s0 = 0; s0 < n; s0 += 32) {
    const int s = s0 + lane;
    float a = 0.f, t0 = 0.f, t1 = 0.f;
    if (s < n) { t0 = ts[slot + s]; t1 = te[slot + s]; a = row_alpha(sigma[first + s], t0, t1); }
    float total;
    const float T = carry * excl_prod(s < n ? 1.f - a + 1e-10f : 1.f, total);
    carry *= total;
    const float w = a * T;
    if (s < n && w != 0.f) {
      const float* c = rgb + (first + s) * 3;
      r += w * c[0]; g += w * c[1]; b += w * c[2];
      depth += w * (0.5f * (t0 + t1));
      acc += w;
    }
  }
  r = all_sum(r); g = all_sum(g); b = all_sum(b); depth = all_sum(depth); acc = all_sum(acc);
  if (lane == 0) {
    const float rest = bg * (1.f - acc);
    out_rgb[3LL * ray] = r + rest; out_rgb[3LL * ray + 1] = g + rest; out_rgb[3LL * ray + 2] = b + rest;
    out_depth[ray] = depth;
  }
}

// Gradients of the rows from that of the rays' colours (depth carries none).  The weight's gradient of a row is
// d . (c - bg); with its sum over the ray known, the second pass needs only running sums.
__global__ void __launch_bounds__(256)
rows_composite_bwd_kernel(int R, int S, const int* __restrict__ offsets, const float* __restrict__ sigma, const float* __restrict__ rgb,
                          const float* __restrict__ ts, const float* __restrict__ te, float bg, const float* __restrict__ d_out,
                          float* __restrict__ d_sigma, float* __restrict__ d_rgb) {
  const int ray = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (ray >= R) return;
  const long long first = offsets[ray], slot = (long long)ray * S;
  const int n = offsets[ray + 1] - (int)first;
  const float d0 = d_out[3LL * ray], d1 = d_out[3LL * ray + 1], d2 = d_out[3LL * ray + 2];
  float carry = 1.f, sum = 0.f;
  for (int s0 = 0; s0 < n; s0 += 32) {
    const int s = s0 + lane;
    float a = 0.f, dw = 0.f;
    if (s < n) {
      const float* c = rgb + (first + s) * 3;
      a = row_alpha(sigma[first + s], ts[slot + s], te[slot + s]);
      dw = d0 * (c[0] - bg) + d1 * (c[1] - bg) + d2 * (c[2] - bg);
    }
    float total;
    const float T = carry * excl_prod(s < n ? 1.f - a + 1e-10f : 1.f, total);
    sum += all_sum(dw * a * T);
    carry *= total;
  }
  carry = 1.f;
  float prefix = 0.f;
  for (int s0 = 0; s0 < n; s0 += 32) {
    const int s = s0 + lane;
    float a = 0.f, dw = 0.f, d = 0.f;
    if (s < n) {
      const float* c = rgb + (first + s) * 3;
      const float t0 = ts[slot + s], t1 = te[slot + s];
      d = t1 - t0;
      a = row_alpha(sigma[first + s], t0, t1);
      dw = d0 * (c[0] - bg) + d1 * (c[1] - bg) + d2 * (c[2] - bg);
    }
    const float t = 1.f - a + 1e-10f;
    float total, step;
    const float T = carry * excl_prod(s < n ? t : 1.f, total);
    const float incl = prefix + incl_sum(dw * a * T, step);
    if (s < n) {
      const float w = a * T, dalpha = dw * T - (sum - incl) / t;
      d_sigma[first + s] = dalpha * d * (1.f - a);
      float* o = d_rgb + (first + s) * 3;
      o[0] = w * d0; o[1] = w * d1; o[2] = w * d2;
    }
    carry *= total;
    prefix += step;
  }
}

}  // namespace lmb

using namespace lmb;

// offsets: int32 [R + 1]; idx: int64 [offsets[R]]
LMB_API int lmb_row_index(int R, int S, const int* offsets, long long* idx, cudaStream_t stream) {
  if (R <= 0) return 0;
  row_index_kernel<<<ceil_div((long long)R * 32, 256), 256, 0, stream>>>(R, S, offsets, idx);
  LMB_LAUNCH_CHECK();
  return 0;
}

// sigma: [M]; rgb: [M, 3]; ts, te: [R, S], the first offsets[r + 1] - offsets[r] slots of ray r are its rows
LMB_API int lmb_rows_composite(int R, int S, const int* offsets, const float* sigma, const float* rgb, const float* ts, const float* te,
                               float bg, float* out_rgb, float* out_depth, cudaStream_t stream) {
  if (R <= 0) return 0;
  rows_composite_kernel<<<ceil_div((long long)R * 32, 256), 256, 0, stream>>>(R, S, offsets, sigma, rgb, ts, te, bg, out_rgb, out_depth);
  LMB_LAUNCH_CHECK();
  return 0;
}

LMB_API int lmb_rows_composite_bwd(int R, int S, const int* offsets, const float* sigma, const float* rgb, const float* ts,
                                   const float* te, float bg, const float* d_out, float* d_sigma, float* d_rgb, cudaStream_t stream) {
  if (R <= 0) return 0;
  rows_composite_bwd_kernel<<<ceil_div((long long)R * 32, 256), 256, 0, stream>>>(R, S, offsets, sigma, rgb, ts, te, bg, d_out, d_sigma,
                                                                                 d_rgb);
  LMB_LAUNCH_CHECK();
  return 0;
}
