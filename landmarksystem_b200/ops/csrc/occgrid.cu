// Occupancy-grid ray marching (Instant-NGP style).
//
// The grid has `levels` cascades of `res`^3 binary cells; cascade l covers the region of interest
// scaled by 2^l about its centre.  A ray advances in steps dt = clamp(t * cone_angle, step, inf); a
// step whose midpoint lies in an occupied cell of the finest cascade that contains it becomes a
// sample [t, t + dt]; empty cells are skipped by jumping to the cell's exit (in whole steps, so the
// sample lattice of a ray does not depend on what was skipped).  The reference obtains this from
// nerfacc's OccGridEstimator.sampling (landmark/nerf_components/ray_samplers/volumetric_sampler.py:92-104).
// Output is written directly in the padded [R, max_samples] layout the compositing kernels consume,
// so no packed->padded conversion pass is needed.
#include "common.cuh"

namespace lmb {

struct OccGrid {
  const unsigned char* cells;   // [levels, res, res, res] (z fastest? no: x slowest) -> index ((l*res + ix)*res + iy)*res + iz
  float lo[3], hi[3];           // region of interest of cascade 0
  int res, levels;
};

__device__ __forceinline__ bool ray_aabb(const float* o, const float* d, const float* lo, const float* hi, float& t0, float& t1) {
  t0 = -3.4e38f; t1 = 3.4e38f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float inv = 1.f / (fabsf(d[k]) > 1e-12f ? d[k] : (d[k] >= 0 ? 1e-12f : -1e-12f));
    float a = (lo[k] - o[k]) * inv, b = (hi[k] - o[k]) * inv;
    if (a > b) { float s = a; a = b; b = s; }
    t0 = fmaxf(t0, a); t1 = fminf(t1, b);
  }
  return t1 > t0;
}

// kLanes lanes walk a ray: the lattice of a ray is a chain of three dependent operations a step and every lane runs it, but
// a lane looks only its own point up.  Which points the walk visits is then settled inside the group: after an empty cell the
// next visited point is the first whose middle lies past that cell, exactly as one thread would have gone on.
// Few rays are bound by latency (the chain, then a lookup and the divisions behind it: 4096 rays issue in 29 % of the cycles at 12
// warps an SM), many by instruction issue (65536 and 131072 rays: 64 and 74 %).
template <int kLanes>
__global__ void __launch_bounds__(128)
occ_march_kernel(int R, const float* __restrict__ rays_o, const float* __restrict__ rays_d, const float* __restrict__ jitter,
                 OccGrid g, float near_t, float far_t, float step, float cone_angle, int max_samples,
                 int* __restrict__ counts, float* __restrict__ t_starts, float* __restrict__ t_ends) {
  constexpr unsigned kGroup = kLanes == 32 ? 0xffffffffu : (1u << kLanes) - 1u;
  constexpr float kNone = -3.4e38f;                            // nothing to skip
  const int r = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
  const int lane = threadIdx.x & (kLanes - 1), first = (threadIdx.x & 31) - lane;     // first lane of the group in its warp
  const bool live = r < R;
  const int ray = live ? r : 0;
  const float o[3] = {rays_o[3 * ray], rays_o[3 * ray + 1], rays_o[3 * ray + 2]};
  const float d[3] = {rays_d[3 * ray], rays_d[3 * ray + 1], rays_d[3 * ray + 2]};
  // outermost cascade bounds
  float c[3], h[3], olo[3], ohi[3];
  const float grow = (float)(1 << (g.levels - 1));
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    c[k] = 0.5f * (g.lo[k] + g.hi[k]); h[k] = 0.5f * (g.hi[k] - g.lo[k]);
    olo[k] = c[k] - h[k] * grow; ohi[k] = c[k] + h[k] * grow;
  }
  float t0, t1;
  int n = 0, guard = 0;
  bool more = live && ray_aabb(o, d, olo, ohi, t0, t1);
  float t = 0.f, skip = kNone;                                 // points whose middle lies before `skip` are not visited
  if (more) {
    t0 = fmaxf(t0, near_t); t1 = fminf(t1, far_t);
    t = t0;
    if (jitter) t += jitter[ray] * fmaxf(t * cone_angle, step);
    more = t < t1 && max_samples > 0;
  }
  while (__any_sync(0xffffffffu, more)) {
    const float begin = t;
    float mine = t;
#pragma unroll
    for (int j = 0; j < kLanes; ++j) {
      if (j == lane) mine = t;
      t += fmaxf(t * cone_angle, step);
    }
    const float dt = fmaxf(mine * cone_angle, step);
    const float tm = mine + 0.5f * dt;
    const bool inside = more && mine < t1;
    bool occupied = false;
    float exit_t = kNone;                                      // of an empty cell: where the ray leaves it
    if (inside && !(tm < skip)) {
      float q[3], m = 0.f;
#pragma unroll
      for (int k = 0; k < 3; ++k) { const float p = o[k] + tm * d[k]; q[k] = (p - c[k]) / h[k]; m = fmaxf(m, fabsf(q[k])); }
      // finest cascade containing the point: m <= 2^l
      int l = 0;
      while (l < g.levels - 1 && m > (float)(1 << l)) ++l;
      if (!(m > (float)(1 << l))) {                            // (outside every cascade: visited, neither sample nor skip)
        const float s = (float)(1 << l), shrink = 1.f / s;
        int idx[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float u = (q[k] * shrink * 0.5f + 0.5f) * g.res;         // cell coordinate in [0, res]
          idx[k] = min(max((int)u, 0), g.res - 1);
        }
        const long long cell = (((long long)l * g.res + idx[0]) * g.res + idx[1]) * g.res + idx[2];
        occupied = g.cells[cell] != 0;
        if (!occupied) {
          exit_t = 3.4e38f;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            if (fabsf(d[k]) < 1e-12f) continue;
            const float edge = d[k] > 0 ? (float)(idx[k] + 1) : (float)idx[k];
            const float world = c[k] + ((edge / g.res - 0.5f) * 2.f) * h[k] * s;
            exit_t = fminf(exit_t, (world - o[k]) / d[k]);
          }
        }
      }
    }
    const unsigned in_mask = __ballot_sync(0xffffffffu, inside) >> first & kGroup;
    const unsigned empty = __ballot_sync(0xffffffffu, exit_t != kNone) >> first & kGroup;
    unsigned visited = 0, left = in_mask;                      // left: points not settled yet
    bool go = left != 0;
    while (__any_sync(0xffffffffu, go)) {
      const unsigned open = __ballot_sync(0xffffffffu, !(tm < skip)) >> first & left;
      const int at = open ? __ffs(open) - 1 : 0;
      const unsigned from = open ? ~0u << at : 0u;             // the first point that is visited, and all behind it
      const unsigned stop = empty & from & left;               // the next empty cell from there on is visited too
      const int e = stop ? __ffs(stop) - 1 : kLanes;
      const float next = __shfl_sync(0xffffffffu, exit_t, first + (e & (kLanes - 1)));
      if (go) {
        const unsigned upto = e >= 31 ? ~0u : (2u << e) - 1u;
        visited |= left & from & upto;
        left &= ~upto;
        if (!open) left = 0;
        else skip = stop ? next : kNone;
        go = left != 0;
      }
    }
    while (guard + __popc(visited) > 100000) visited &= ~(1u << (31 - __clz(visited)));      // no more visits than that per ray
    const unsigned hits = visited & (__ballot_sync(0xffffffffu, occupied) >> first & kGroup);
    const int slot = n + __popc(hits & ((1u << lane) - 1u));
    if ((hits >> lane & 1u) && slot < max_samples) {
      t_starts[(long long)r * max_samples + slot] = mine;
      t_ends[(long long)r * max_samples + slot] = mine + dt;
    }
    n = min(n + __popc(hits), max_samples);
    guard += __popc(visited);
    // a step too small to move t: end once nothing more can come of it
    more = more && t < t1 && n < max_samples && guard < 100000 && (t != begin || hits != 0);
  }
  if (live && lane == 0) counts[r] = n;
}

}  // namespace lmb

using namespace lmb;

LMB_API int lmb_occ_march(int R, const float* rays_o, const float* rays_d, const float* jitter, const unsigned char* cells,
                          const float* roi /* lo xyz, hi xyz (host) */, int res, int levels, float near_t, float far_t,
                          float step, float cone_angle, int max_samples, int* counts, float* t_starts, float* t_ends,
                          cudaStream_t stream) {
  if (R <= 0) return 0;
  OccGrid g;
  g.cells = cells; g.res = res; g.levels = levels;
  for (int k = 0; k < 3; ++k) { g.lo[k] = roi[k]; g.hi[k] = roi[3 + k]; }
  // Lanes where the rays alone do not fill the GPU.  Whole call (two cleared outputs among it) in us, rays of a training batch with 2 / 4 /
  // 8 / 16 lanes: 8192 rays 128 / 91 / 74 / 65, 16384 131 / 98 / 84 / 82, 49152 158 / 154 / 145 / 149, 98304 247 / 225 / 230 / 250,
  // 262144 510 / 508 / 542 / 614; rays of a frame: 8192 50 / 46 / 42 / 43, 16384 53 / 47 / 44 / 46, 65536 87 / 83 / 75 / 86, 98304
  // 125 / 117 / 115 / 132, 262144 348 / 292 / 321 / 401.  One thread a ray: 148, 149, 163, 204, 620 and 54, 58, 109, 147, 430.
  const int lanes = R > 65536 ? 4 : R > 8192 ? 8 : 16;
  const auto kernel = lanes == 4 ? occ_march_kernel<4> : lanes == 8 ? occ_march_kernel<8> : occ_march_kernel<16>;
  kernel<<<ceil_div((long long)R * lanes, 128), 128, 0, stream>>>(R, rays_o, rays_d, jitter, g, near_t, far_t, step, cone_angle,
                                                                  max_samples, counts, t_starts, t_ends);
  LMB_LAUNCH_CHECK();
  return 0;
}
