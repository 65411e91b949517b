// 3D Gaussian splatting rasteriser: projection + SH colour, (tile, depth) key generation, per-tile
// ranges, tile alpha-blending, and the backward of all of it.
//
// Functional counterpart of the rasteriser extension the reference calls
// (GaussianRasterizationSettings / GaussianRasterizer with an extra visible_filter;
// benchmarks/nerf/origin_gs/gs_model.py:82-97,148-162,211-220) whose source is not part of the
// reference tree.  The math is the published EWA splatting formulation: 3-D covariance R S S^T R^T,
// perspective Jacobian, 0.3 px low-pass, 3-sigma extent, front-to-back alpha compositing with
// alpha < 1/255 skipped, alpha clamped to 0.99 and termination at T < 1e-4.
// Conventions: matrices are row-vector style ([x y z 1] @ M), 16x16 pixel tiles, channel-first
// image output [3, H, W].  Backward reduces per-Gaussian gradients across the warp with shuffles
// before touching global memory (one atomic per warp and Gaussian instead of one per pixel).
#include "common.cuh"

namespace lmb {

constexpr int kTile = 16;
constexpr int kTilePixels = kTile * kTile;

// Matrices and position stay on the device (35 floats: view, proj, campos); a block copies them to shared memory once, so
// that a frame does not wait for them on the host (three blocking copies, 0.1 ms of a small frame).
struct GSCameraPose {
  float view[16];      // world -> view, row-vector convention (transposed world-to-camera)
  float proj[16];      // world -> clip (view @ projection)
  float campos[3];
};

struct GSCameraInfo {
  float tanfovx, tanfovy;
  int W, H;
  float scale_modifier;
  int sh_degree;       // active degree
  int sh_coeffs;       // coefficients stored per Gaussian ((max_degree + 1)^2)
};

struct GSCamera : GSCameraInfo {
  const float *view, *proj, *campos;
};

__device__ __forceinline__ GSCamera load_camera(const GSCameraInfo& info, const float* __restrict__ pose, GSCameraPose& s) {
  constexpr int n = sizeof(GSCameraPose) / sizeof(float);
  if (threadIdx.x < n) reinterpret_cast<float*>(&s)[threadIdx.x] = pose[threadIdx.x];
  __syncthreads();
  GSCamera cam;
  static_cast<GSCameraInfo&>(cam) = info;
  cam.view = s.view; cam.proj = s.proj; cam.campos = s.campos;
  return cam;
}

__device__ __forceinline__ float3 xform43(const float* m, float3 p) {   // [p 1] @ M, first 3 comps
  return make_float3(m[0] * p.x + m[4] * p.y + m[8] * p.z + m[12], m[1] * p.x + m[5] * p.y + m[9] * p.z + m[13],
                     m[2] * p.x + m[6] * p.y + m[10] * p.z + m[14]);
}
__device__ __forceinline__ float4 xform44(const float* m, float3 p) {
  return make_float4(m[0] * p.x + m[4] * p.y + m[8] * p.z + m[12], m[1] * p.x + m[5] * p.y + m[9] * p.z + m[13],
                     m[2] * p.x + m[6] * p.y + m[10] * p.z + m[14], m[3] * p.x + m[7] * p.y + m[11] * p.z + m[15]);
}

__device__ __forceinline__ void quat_to_rot(float4 q, float* R) {   // q = (w, x, y, z), unit
  const float r = q.x, x = q.y, y = q.z, z = q.w;
  R[0] = 1.f - 2.f * (y * y + z * z); R[1] = 2.f * (x * y - r * z); R[2] = 2.f * (x * z + r * y);
  R[3] = 2.f * (x * y + r * z); R[4] = 1.f - 2.f * (x * x + z * z); R[5] = 2.f * (y * z - r * x);
  R[6] = 2.f * (x * z - r * y); R[7] = 2.f * (y * z + r * x); R[8] = 1.f - 2.f * (x * x + y * y);
}

// Sigma = R diag(s)^2 R^T, upper triangle (xx, xy, xz, yy, yz, zz)
__device__ __forceinline__ void cov3d_from(float3 s, float4 q, float* c) {
  float R[9];
  quat_to_rot(q, R);
  const float sx = s.x * s.x, sy = s.y * s.y, sz = s.z * s.z;
  c[0] = R[0] * R[0] * sx + R[1] * R[1] * sy + R[2] * R[2] * sz;
  c[1] = R[0] * R[3] * sx + R[1] * R[4] * sy + R[2] * R[5] * sz;
  c[2] = R[0] * R[6] * sx + R[1] * R[7] * sy + R[2] * R[8] * sz;
  c[3] = R[3] * R[3] * sx + R[4] * R[4] * sy + R[5] * R[5] * sz;
  c[4] = R[3] * R[6] * sx + R[4] * R[7] * sy + R[5] * R[8] * sz;
  c[5] = R[6] * R[6] * sx + R[7] * R[7] * sy + R[8] * R[8] * sz;
}

// T = J * Wr (2x3), where Wr[i][j] = d view_i / d world_j.  Returns cov2D (a, b, c) before the low-pass.
__device__ __forceinline__ void project_cov(const GSCamera& cam, float3 t, const float* c3, float fx, float fy,
                                            float* T, float& a, float& b, float& c) {
  const float limx = 1.3f * cam.tanfovx, limy = 1.3f * cam.tanfovy;
  const float txz = fminf(limx, fmaxf(-limx, t.x / t.z)) * t.z;
  const float tyz = fminf(limy, fmaxf(-limy, t.y / t.z)) * t.z;
  const float j00 = fx / t.z, j02 = -fx * txz / (t.z * t.z), j11 = fy / t.z, j12 = -fy * tyz / (t.z * t.z);
  const float* v = cam.view;   // Wr[i][j] = v[j*4 + i]
  T[0] = j00 * v[0] + j02 * v[2]; T[1] = j00 * v[4] + j02 * v[6]; T[2] = j00 * v[8] + j02 * v[10];
  T[3] = j11 * v[1] + j12 * v[2]; T[4] = j11 * v[5] + j12 * v[6]; T[5] = j11 * v[9] + j12 * v[10];
  // cov2D = T Sigma T^T
  const float s0 = c3[0] * T[0] + c3[1] * T[1] + c3[2] * T[2];
  const float s1 = c3[1] * T[0] + c3[3] * T[1] + c3[4] * T[2];
  const float s2 = c3[2] * T[0] + c3[4] * T[1] + c3[5] * T[2];
  const float u0 = c3[0] * T[3] + c3[1] * T[4] + c3[2] * T[5];
  const float u1 = c3[1] * T[3] + c3[3] * T[4] + c3[4] * T[5];
  const float u2 = c3[2] * T[3] + c3[4] * T[4] + c3[5] * T[5];
  a = T[0] * s0 + T[1] * s1 + T[2] * s2;
  b = T[3] * s0 + T[4] * s1 + T[5] * s2;
  c = T[3] * u0 + T[4] * u1 + T[5] * u2;
}

__constant__ float kSH_C1 = 0.4886025119029199f;
__constant__ float kSH_C2[5] = {1.0925484305920792f, -1.0925484305920792f, 0.31539156525252005f, -1.0925484305920792f, 0.5462742152960396f};
__constant__ float kSH_C3[7] = {-0.5900435899266435f, 2.890611442640554f, -0.4570457994644658f, 0.3731763325901154f, -0.4570457994644658f, 1.445305721320277f, -0.5900435899266435f};

__device__ __forceinline__ void sh_basis(int deg, float3 d, float* B) {
  const float x = d.x, y = d.y, z = d.z;
  B[0] = 0.28209479177387814f;
  if (deg > 0) {
    B[1] = -kSH_C1 * y; B[2] = kSH_C1 * z; B[3] = -kSH_C1 * x;
    if (deg > 1) {
      const float xx = x * x, yy = y * y, zz = z * z, xy = x * y, yz = y * z, xz = x * z;
      B[4] = kSH_C2[0] * xy; B[5] = kSH_C2[1] * yz; B[6] = kSH_C2[2] * (2.f * zz - xx - yy);
      B[7] = kSH_C2[3] * xz; B[8] = kSH_C2[4] * (xx - yy);
      if (deg > 2) {
        B[9] = kSH_C3[0] * y * (3.f * xx - yy); B[10] = kSH_C3[1] * xy * z; B[11] = kSH_C3[2] * y * (4.f * zz - xx - yy);
        B[12] = kSH_C3[3] * z * (2.f * zz - 3.f * xx - 3.f * yy); B[13] = kSH_C3[4] * x * (4.f * zz - xx - yy);
        B[14] = kSH_C3[5] * z * (xx - yy); B[15] = kSH_C3[6] * x * (xx - 3.f * yy);
      }
    }
  }
}

// d(basis)/d(dir) for the backward of the view-dependent colour
__device__ __forceinline__ void sh_basis_grad(int deg, float3 d, float* Bx, float* By, float* Bz) {
  const float x = d.x, y = d.y, z = d.z;
  Bx[0] = By[0] = Bz[0] = 0.f;
  if (deg > 0) {
    Bx[1] = 0.f; By[1] = -kSH_C1; Bz[1] = 0.f;
    Bx[2] = 0.f; By[2] = 0.f; Bz[2] = kSH_C1;
    Bx[3] = -kSH_C1; By[3] = 0.f; Bz[3] = 0.f;
    if (deg > 1) {
      Bx[4] = kSH_C2[0] * y; By[4] = kSH_C2[0] * x; Bz[4] = 0.f;
      Bx[5] = 0.f; By[5] = kSH_C2[1] * z; Bz[5] = kSH_C2[1] * y;
      Bx[6] = kSH_C2[2] * -2.f * x; By[6] = kSH_C2[2] * -2.f * y; Bz[6] = kSH_C2[2] * 4.f * z;
      Bx[7] = kSH_C2[3] * z; By[7] = 0.f; Bz[7] = kSH_C2[3] * x;
      Bx[8] = kSH_C2[4] * 2.f * x; By[8] = kSH_C2[4] * -2.f * y; Bz[8] = 0.f;
      if (deg > 2) {
        const float xx = x * x, yy = y * y, zz = z * z;
        Bx[9] = kSH_C3[0] * 6.f * x * y; By[9] = kSH_C3[0] * (3.f * xx - 3.f * yy); Bz[9] = 0.f;
        Bx[10] = kSH_C3[1] * y * z; By[10] = kSH_C3[1] * x * z; Bz[10] = kSH_C3[1] * x * y;
        Bx[11] = kSH_C3[2] * -2.f * x * y; By[11] = kSH_C3[2] * (4.f * zz - xx - 3.f * yy); Bz[11] = kSH_C3[2] * 8.f * y * z;
        Bx[12] = kSH_C3[3] * -6.f * x * z; By[12] = kSH_C3[3] * -6.f * y * z; Bz[12] = kSH_C3[3] * (6.f * zz - 3.f * xx - 3.f * yy);
        Bx[13] = kSH_C3[4] * (4.f * zz - 3.f * xx - yy); By[13] = kSH_C3[4] * -2.f * x * y; Bz[13] = kSH_C3[4] * 8.f * x * z;
        Bx[14] = kSH_C3[5] * 2.f * x * z; By[14] = kSH_C3[5] * -2.f * y * z; Bz[14] = kSH_C3[5] * (xx - yy);
        Bx[15] = kSH_C3[6] * (3.f * xx - 3.f * yy); By[15] = kSH_C3[6] * -6.f * x * y; Bz[15] = 0.f;
      }
    }
  }
}

constexpr float kAlphaMin = 1.f / 255.f;
constexpr float kNoBound = 1e9f;      // reach of a record that has no ellipse

// Tiles [x0, x1) x [y0, y1) of a record: the square of the 3-sigma radius, cut to the tiles that hold a pixel within reach.
__device__ __forceinline__ void splat_rect(float4 q0, int r, int tiles_x, int tiles_y, int& x0, int& y0, int& x1, int& y1) {
  x0 = min(tiles_x, max(0, (int)((q0.x - r) / kTile)));
  y0 = min(tiles_y, max(0, (int)((q0.y - r) / kTile)));
  x1 = min(tiles_x, max(0, (int)((q0.x + r + kTile - 1) / kTile)));
  y1 = min(tiles_y, max(0, (int)((q0.y + r + kTile - 1) / kTile)));
  constexpr float inv = 1.f / kTile;
  x0 = max(x0, (int)ceilf((q0.x - q0.z - (kTile - 1)) * inv));
  y0 = max(y0, (int)ceilf((q0.y - q0.w - (kTile - 1)) * inv));
  x1 = max(x0, min(x1, (int)floorf((q0.x + q0.z) * inv) + 1));
  y1 = max(y0, min(y1, (int)floorf((q0.y + q0.w) * inv) + 1));
}

// Rows of a warp's 32 Gaussians (`row` floats each, rows of consecutive Gaussians adjacent) between global and shared memory.
// A warp's rows start on a multiple of 128 bytes from the tensor's base, so they move as float4.  A lane works on one row:
// rows of an odd number of floats stay as they are, which needs no index arithmetic and lets all copies of a warp be in
// flight at once (cp.async); rows of an even number are spread to row + 1, free of bank conflicts.  Rows of Gaussians outside
// `rows` need not be read.
__device__ __forceinline__ void sh_rows_load(const float* __restrict__ g, long long first, int n_rows, int row, uint32_t rows,
                                             float* s) {
  const int lane = threadIdx.x & 31, n4 = n_rows * row / 4;
  const float4* g4 = reinterpret_cast<const float4*>(g + first * row);
  if (row & 1) {
    const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(s);
    const float inv = 1.f / row;
    for (int e = lane; e < n4; e += 32) {
      const int r0 = (int)((4 * e + 0.5f) * inv), r3 = (int)((4 * e + 3.5f) * inv);      // rows of the piece's first and last float
      if ((rows >> r0 | rows >> r3) & 1u)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s0 + 16 * e), "l"(g4 + e) : "memory");
    }
    for (int e = 4 * n4 + lane; e < n_rows * row; e += 32) s[e] = g[first * row + e];
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  const int stride = row + 1;
#pragma unroll 4
  for (int e = lane; e < n4; e += 32) {
    const int r0 = 4 * e / row, r3 = (4 * e + 3) / row;
    if (!((rows >> r0 | rows >> r3) & 1u)) continue;
    const float4 v = __ldg(g4 + e);
    int r = r0, k = 4 * e - r0 * row;
    s[r * stride + k] = v.x; if (++k == row) { k = 0; ++r; }
    s[r * stride + k] = v.y; if (++k == row) { k = 0; ++r; }
    s[r * stride + k] = v.z; if (++k == row) { k = 0; ++r; }
    s[r * stride + k] = v.w;
  }
  for (int e = 4 * n4 + lane; e < n_rows * row; e += 32) s[e / row * stride + e % row] = g[first * row + e];
}

__device__ __forceinline__ void sh_rows_store(float* __restrict__ g, long long first, int n_rows, int row, const float* s) {
  const int lane = threadIdx.x & 31, n4 = n_rows * row / 4;
  float4* g4 = reinterpret_cast<float4*>(g + first * row);
  if (row & 1) {
    const float4* s4 = reinterpret_cast<const float4*>(s);
#pragma unroll 4
    for (int e = lane; e < n4; e += 32) g4[e] = s4[e];
    for (int e = 4 * n4 + lane; e < n_rows * row; e += 32) g[first * row + e] = s[e];
    return;
  }
  const int stride = row + 1;
  for (int e = lane; e < n4; e += 32) {
    int r = 4 * e / row, k = 4 * e - r * row;
    float4 v;
    v.x = s[r * stride + k]; if (++k == row) { k = 0; ++r; }
    v.y = s[r * stride + k]; if (++k == row) { k = 0; ++r; }
    v.z = s[r * stride + k]; if (++k == row) { k = 0; ++r; }
    v.w = s[r * stride + k];
    g4[e] = v;
  }
  for (int e = 4 * n4 + lane; e < n_rows * row; e += 32) g[first * row + e] = s[e / row * stride + e % row];
}

// The coefficients are stored as one tensor or, as a Gaussian model keeps them, as the constant term and the rest; both are
// read in place (joining them first moved 2.3 GB per frame of a 6 M cloud: 1005 us of a 3433 us frame, and 235 us plus the
// split of the gradient in a 1.5 M training step).
struct SHRows {
  int row0, row1;        // floats per row of the first and second tensor (0: there is none)
  float *s0, *s1;        // this warp's rows in shared memory
  float *lane0, *lane1;  // this lane's row of either
};
__host__ __device__ constexpr int sh_warp_floats(int coeffs) { return 32 * (coeffs * 3 + 2); }

__device__ __forceinline__ SHRows sh_layout(float* smem, int coeffs, bool split) {
  SHRows r;
  r.row0 = split ? 3 : coeffs * 3;
  r.row1 = split ? coeffs * 3 - 3 : 0;
  r.s0 = smem + (threadIdx.x >> 5) * sh_warp_floats(coeffs);
  r.s1 = r.s0 + 32 * (r.row0 | 1);
  r.lane0 = r.s0 + (threadIdx.x & 31) * (r.row0 | 1);
  r.lane1 = r.s1 + (threadIdx.x & 31) * (r.row1 | 1);
  if (!split) r.lane1 = r.lane0 + 3;
  return r;              // coefficient 0: lane0[0..2], coefficient k: lane1[3 k - 3 ..]
}

// The pairs of a warp's splats, 32 at a time: f(lane that holds the splat, tile, whether there is a pair) on every lane.  The
// lanes share the pairs evenly, because a lane that walked its own splat alone would wait for an atomic per tile of it.
template <typename F>
__device__ __forceinline__ void for_warp_pairs(uint32_t touched, int x0, int y0, int x1, int tiles_x, F&& f) {
  const int lane = threadIdx.x & 31;
  uint32_t upto = touched;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t below = __shfl_up_sync(0xffffffffu, upto, d);
    if (lane >= d) upto += below;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, upto, 31);
  for (uint32_t base = 0; base < total; base += 32) {
    const uint32_t p = base + lane;
    int owner = 0;                                   // the first lane whose pairs reach past p
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (__shfl_sync(0xffffffffu, upto, owner + step - 1) <= p) owner += step;
    const uint32_t before = __shfl_sync(0xffffffffu, upto - touched, owner);
    const int ox = __shfl_sync(0xffffffffu, x0, owner), oy = __shfl_sync(0xffffffffu, y0, owner);
    const uint32_t wide = (uint32_t)max(__shfl_sync(0xffffffffu, x1, owner) - ox, 1), at = p - before;
    f(owner, (oy + (int)(at / wide)) * tiles_x + ox + (int)(at % wide), p < total);
  }
}

constexpr int kPreThreads = 128;

// Words between two counters: atomics on one 32-byte sector queue (283 -> 128 us in a frame of 6 M).
constexpr int kCounterStride = 8;

// Counters of a tile, a power of two.  The warps take them in turn, or a view whose splats crowd into a few tiles would queue for them
// all the same.  Projection of 6 M Gaussians with one and with several: 1075 -> 332 us at 320 x 180, 2566 -> 348 where they fill 28 tiles
// of 1080p, 325 -> 329 over all of it (the drop 132 -> 120).  Counters are cleared, scanned and written once more, so they stay
// fewer than a sixteenth of the Gaussians.
constexpr int kMaxTileCounters = 32;
static int tile_counters(int N, int n_tiles) {
  int per_tile = 1;
  while (per_tile < kMaxTileCounters && (long long)n_tiles * per_tile * 2 <= N / 16) per_tile *= 2;
  return per_tile;
}
// The counter that a Gaussian's warp takes
__device__ __forceinline__ long long tile_counter(int tile, int per_tile, int gaussian) {
  return ((long long)tile * per_tile + ((gaussian >> 5) & (per_tile - 1))) * kCounterStride;
}

// ---- preprocess ------------------------------------------------------------------------------------------
// visible: optional per-Gaussian byte mask (0 = skip).  shs: [N, sh_coeffs, 3] or null (then colors_pre [N,3]).
// cov3d_pre: optional [N, 6].  Outputs are per Gaussian; radii == 0 marks "not rendered".
// Bound by memory: 44 B of geometry in, 192 B of SH for the Gaussians in view, 56 B out; the SH rows go through shared
// memory because one lane reading its own 192-byte row touches a line per load (6 M Gaussians: 593 -> 299 us).
__global__ void __launch_bounds__(kPreThreads)
gs_preprocess_kernel(int N, const float* __restrict__ means, const float* __restrict__ scales, const float* __restrict__ rots,
                     const float* __restrict__ opac, const float* __restrict__ shs, const float* __restrict__ sh_rest,
                     const float* __restrict__ colors_pre, const float* __restrict__ cov3d_pre,
                     const unsigned char* __restrict__ visible, GSCameraInfo info, const float* __restrict__ pose,
                     int* __restrict__ radii, float4* __restrict__ rec, uint32_t* __restrict__ tiles_touched,
                     uint32_t* __restrict__ tile_counts, int per_tile, int radius_only) {
  extern __shared__ __align__(16) float s_sh[];
  __shared__ GSCameraPose s_pose;
  const GSCamera cam = load_camera(info, pose, s_pose);
  const int i = blockIdx.x * kPreThreads + threadIdx.x;
  const long long first = (long long)blockIdx.x * kPreThreads + (threadIdx.x & ~31);
  if (first >= N) return;                          // whole warps leave; the rest meet at __syncwarp only
  float3 p = make_float3(0.f, 0.f, 0.f);
  float4 q0, q1;
  float depth = 0.f;
  int r = 0;
  uint32_t touched = 0;
  int x0 = 0, y0 = 0, x1 = 0, y1 = 0;
  const int tiles_x = (cam.W + kTile - 1) / kTile, tiles_y = (cam.H + kTile - 1) / kTile;
  if (i < N && (!visible || visible[i])) do {
    p = make_float3(means[3 * i], means[3 * i + 1], means[3 * i + 2]);
    const float3 t = xform43(cam.view, p);
    if (t.z <= 0.2f) break;
    const float4 ph = xform44(cam.proj, p);
    const float pw = 1.f / (ph.w + 1e-7f);
    const float2 ndc = make_float2(ph.x * pw, ph.y * pw);
    float c3[6];
    if (cov3d_pre) {
#pragma unroll
      for (int k = 0; k < 6; ++k) c3[k] = cov3d_pre[6 * (long long)i + k];
    } else {
      const float3 s = make_float3(scales[3 * i] * cam.scale_modifier, scales[3 * i + 1] * cam.scale_modifier,
                                   scales[3 * i + 2] * cam.scale_modifier);
      cov3d_from(s, __ldg(reinterpret_cast<const float4*>(rots) + i), c3);
    }
    const float fx = cam.W / (2.f * cam.tanfovx), fy = cam.H / (2.f * cam.tanfovy);
    float T[6], a, b, c;
    project_cov(cam, t, c3, fx, fy, T, a, b, c);
    a += 0.3f; c += 0.3f;
    const float det = a * c - b * b;
    if (det == 0.f) break;
    const float inv = 1.f / det;
    const float mid = 0.5f * (a + c);
    const float lam = mid + sqrtf(fmaxf(0.1f, mid * mid - det));
    const int rad = (int)ceilf(3.f * sqrtf(lam));
    const float2 pix = make_float2(((ndc.x + 1.f) * cam.W - 1.f) * 0.5f, ((ndc.y + 1.f) * cam.H - 1.f) * 0.5f);
    splat_rect(make_float4(pix.x, pix.y, kNoBound, kNoBound), rad, tiles_x, tiles_y, x0, y0, x1, y1);
    if ((x1 - x0) * (y1 - y0) == 0 || rad <= 0) break;
    r = rad;
    if (radius_only) break;
    const float op = opac[i];
    // alpha >= 1/255  <=>  half the quadratic form <= ln(255 opacity).  The walk evaluates the rounded conic, which has the extent
    // of (a, c) only as far as det = a c - b b keeps its bits: with kappa = a c / det, the determinant, the conic's entries and
    // the terms of the form together lose at most some 1.4e-6 kappa of it (a term of the form is up to kappa times the form).
    // The margins cover that up to a kappa of 270 (a splat 18 pixels long, 0.55 wide, at 45 degrees), the factor on level beyond;
    // from 1e5 on (350 pixels) the square of the radius alone bounds the splat.
    const float kappa = a * c * inv;
    const float level = 2.f * (__logf(255.f * op) + 1e-3f);
    q0 = make_float4(pix.x, pix.y, 0.f, 0.f);
    if (level <= 0.f) {
      x1 = x0;                                     // below 1/255 everywhere
      q0.z = q0.w = -1.f;
    } else if (level > 0.f && det > 0.f && kappa < 1e5f) {
      const float wide = level * (1.f + 2e-6f * kappa);
      q0.z = fminf(sqrtf(wide * a) * 1.0001f + 1e-3f, kNoBound);
      q0.w = fminf(sqrtf(wide * c) * 1.0001f + 1e-3f, kNoBound);
      splat_rect(q0, rad, tiles_x, tiles_y, x0, y0, x1, y1);
    } else {
      q0.z = q0.w = kNoBound;                      // a long needle, or not an ellipse (rounding, not a number)
    }
    q1 = make_float4(c * inv, -b * inv, a * inv, op);
    depth = t.z;
    touched = (uint32_t)((x1 - x0) * (y1 - y0));
  } while (false);
  if (i < N) {
    radii[i] = r;
    if (tiles_touched) tiles_touched[i] = touched;
  }
  if (radius_only) return;
  // A count per tile.  Splats of a warp that share the tile (a distant cloud: all of them) send one sum, or the additions to a
  // few addresses would queue.
  for_warp_pairs(touched, x0, y0, x1, tiles_x, [&](int, int tile, bool on) {
    const int same = __shfl_sync(0xffffffffu, tile, 0);                    // lane 0 always has a pair
    const uint32_t pairs = __ballot_sync(0xffffffffu, on);
    if (__all_sync(0xffffffffu, !on || tile == same)) {
      if ((threadIdx.x & 31) == 0) atomicAdd(tile_counts + tile_counter(same, per_tile, i), (uint32_t)__popc(pairs));
    } else if (on) {
      atomicAdd(tile_counts + tile_counter(tile, per_tile, i), 1u);
    }
  });
  const uint32_t rows = __ballot_sync(0xffffffffu, r > 0);
  if (rows == 0) return;
  float3 col = make_float3(0.f, 0.f, 0.f);
  if (shs) {
    const SHRows s = sh_layout(s_sh, cam.sh_coeffs, sh_rest != nullptr);
    const int n_rows = (int)min(32LL, N - first);
    sh_rows_load(shs, first, n_rows, s.row0, rows, s.s0);
    if (s.row1) sh_rows_load(sh_rest, first, n_rows, s.row1, rows, s.s1);
    __syncwarp();
    float3 d = make_float3(p.x - cam.campos[0], p.y - cam.campos[1], p.z - cam.campos[2]);
    const float n = rsqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
    d.x *= n; d.y *= n; d.z *= n;
    float B[16];
    sh_basis(cam.sh_degree, d, B);
    const int nb = (cam.sh_degree + 1) * (cam.sh_degree + 1);
    const float* sh = s.lane1 - 3;
    col = make_float3(0.5f + B[0] * s.lane0[0], 0.5f + B[0] * s.lane0[1], 0.5f + B[0] * s.lane0[2]);
#pragma unroll
    for (int k = 1; k < 16; ++k)
      if (k < nb) { col.x += B[k] * sh[3 * k]; col.y += B[k] * sh[3 * k + 1]; col.z += B[k] * sh[3 * k + 2]; }
    col = make_float3(fmaxf(col.x, 0.f), fmaxf(col.y, 0.f), fmaxf(col.z, 0.f));
  } else if (r > 0) {
    col = make_float3(colors_pre[3 * i], colors_pre[3 * i + 1], colors_pre[3 * i + 2]);
  }
  if (r > 0) {
    rec[3LL * i] = q0;
    rec[3LL * i + 1] = q1;
    rec[3LL * i + 2] = make_float4(col.x, col.y, col.z, depth);
  }
}

__global__ void __launch_bounds__(256)
gs_make_keys_kernel(int N, const float4* __restrict__ rec, const int* __restrict__ radii, const uint32_t* __restrict__ touched,
                    const uint32_t* __restrict__ offsets, int W, int H, long long capacity, uint64_t* __restrict__ keys,
                    uint32_t* __restrict__ vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N || touched[i] == 0) return;
  const int tiles_x = (W + kTile - 1) / kTile, tiles_y = (H + kTile - 1) / kTile;
  int x0, y0, x1, y1;
  splat_rect(rec[3LL * i], radii[i], tiles_x, tiles_y, x0, y0, x1, y1);
  long long off = offsets[i];
  const uint64_t dbits = (uint64_t)__float_as_uint(rec[3LL * i + 2].w);
  for (int y = y0; y < y1; ++y)
    for (int x = x0; x < x1; ++x) {
      if (off >= capacity) return;
      keys[off] = ((uint64_t)(y * tiles_x + x) << 32) | dbits;
      vals[off] = (uint32_t)i;
      ++off;
    }
}

// ---- pairs in tile and depth order ------------------------------------------------------------------------------
// The pairs of a tile are counted with the projection, a scan over the tiles gives every tile its range, the pairs are dropped
// into it in any order, and one block sorts a tile by (depth, Gaussian).  A pair is written twice and read once; the sort of all
// pairs by (tile, depth) moved each of them six times and stays for views with a tile that no block can hold.  A frame of 6 M
// Gaussians (1080p): scan of the splats' counts, keys, six passes and ranges 590 us, now count 30, scan 12, drop 120, sort 200 us;
// 400 k anchors 260 -> 110; 60 k at 801 x 603 67 -> 22.  The drop is bound by the atomics on the
// tiles' cursors.

// A block scans a chunk of the n counters: the place of the next pair of each takes the place of its count, and every tile gets its
// range; totals: {pairs, pairs of the fullest tile}.  Chunks before this one: their sums, in the spare word behind their first counter.
constexpr int kScanBlock = 1024, kScanPer = 8, kScanChunk = kScanBlock * kScanPer;

__global__ void __launch_bounds__(kScanBlock)
gs_tile_sums_kernel(int n, uint32_t* __restrict__ counts, uint32_t* __restrict__ totals) {
  __shared__ uint32_t s_sum[32];
  const int tid = threadIdx.x, base = blockIdx.x * kScanChunk;
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int i = base + k * kScanBlock + tid;
    sum += i < n ? counts[(long long)i * kCounterStride] : 0u;
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if ((tid & 31) == 0) s_sum[tid >> 5] = sum;
  __syncthreads();
  if (tid >= 32) return;
  sum = __reduce_add_sync(0xffffffffu, s_sum[tid]);
  if (tid == 0) counts[(long long)base * kCounterStride + 1] = sum;
  if (tid == 0 && blockIdx.x == 0) totals[1] = 0;
}

__global__ void __launch_bounds__(kScanBlock)
gs_tile_scan_kernel(int n, int per_tile, uint32_t* __restrict__ counts, uint2* __restrict__ ranges, uint32_t* __restrict__ totals) {
  __shared__ uint32_t s_sum[32], s_max[32], s_at[kScanChunk + kScanChunk / kScanPer + 1];      // a spare word after every kScanPer
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, base = blockIdx.x * kScanChunk;
  uint32_t before = 0, mine = 0;
  if (warp == 0) {
    for (int c = lane; c < (int)blockIdx.x; c += 32) before += counts[(long long)c * kScanChunk * kCounterStride + 1];
    before = __reduce_add_sync(0xffffffffu, before);
  }
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int i = k * kScanBlock + tid;
    s_at[i + i / kScanPer] = base + i < n ? counts[(long long)(base + i) * kCounterStride] : 0u;
  }
  __syncthreads();
  uint32_t* at = s_at + tid * (kScanPer + 1);
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) mine += at[k];
  uint32_t incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t below = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += below;
  }
  if (lane == 31) s_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = s_sum[lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t below = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= d) w += below;
    }
    __syncwarp();
    s_sum[lane] = w + before;
    s_max[lane] = before;
  }
  __syncthreads();
  uint32_t next = (warp ? s_sum[warp - 1] : s_max[0]) + incl - mine;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) { const uint32_t v = at[k]; at[k] = next; next += v; }
  if (tid == kScanBlock - 1) at[kScanPer + 1] = next;                 // where the next chunk begins
  __syncthreads();
  uint32_t most = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int i = k * kScanBlock + tid;
    if (base + i >= n) continue;
    const uint32_t start = s_at[i + i / kScanPer];
    counts[(long long)(base + i) * kCounterStride] = start;
    if (i & (per_tile - 1)) continue;
    const int e = i + per_tile;                                       // the first counter of the next tile
    const uint32_t end = s_at[e + e / kScanPer];
    ranges[(base + i) / per_tile] = make_uint2(start, end);
    most = max(most, end - start);
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0) s_max[warp] = most;
  __syncthreads();
  if (warp == 0) {
    most = __reduce_max_sync(0xffffffffu, s_max[lane]);
    if (lane == 0) {
      if (gridDim.x == 1) totals[1] = most;
      else atomicMax(totals + 1, most);
      if (blockIdx.x == gridDim.x - 1) totals[0] = s_sum[31];
    }
  }
}

__global__ void __launch_bounds__(256)
gs_drop_pairs_kernel(int N, const float4* __restrict__ rec, const int* __restrict__ radii, const uint32_t* __restrict__ touched, int W,
                     int H, long long capacity, int per_tile, uint32_t* __restrict__ cursors, uint64_t* __restrict__ keys) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int tiles_x = (W + kTile - 1) / kTile, tiles_y = (H + kTile - 1) / kTile;
  const uint32_t pairs = i < N ? touched[i] : 0u;
  int x0 = 0, y0 = 0, x1 = 0, y1 = 0;
  uint32_t depth = 0;
  if (pairs) {
    splat_rect(rec[3LL * i], radii[i], tiles_x, tiles_y, x0, y0, x1, y1);
    depth = __float_as_uint(rec[3LL * i + 2].w);
  }
  const uint32_t first = (uint32_t)i & ~31u;                               // the warp's first Gaussian
  for_warp_pairs(pairs, x0, y0, x1, tiles_x, [&](int owner, int tile, bool on) {
    const uint64_t key = (uint64_t)__shfl_sync(0xffffffffu, depth, owner) << 32 | (first + owner);
    if (!on) return;
    const uint32_t at = atomicAdd(cursors + tile_counter(tile, per_tile, i), 1u);
    if (at < capacity) keys[at] = key;
  });
}

__device__ __forceinline__ void order(uint64_t& a, uint64_t& b) {
  const bool swap = b < a;
  const uint64_t t = a;
  a = swap ? b : a;
  b = swap ? t : b;
}

// Bitonic sort of the pairs of a tile that holds more than `least` and at most 8 kThreads of them, by (depth, Gaussian) - the
// order in which a stable sort by depth leaves pairs that were written Gaussian by Gaussian.  A merge begins with the mirror image
// (i with i ^ (k - 1)), so that all comparisons put the smaller key first and warps past the last key have nothing to do.  A
// thread holds 8 consecutive keys: strides up to 4 stay in the thread, up to 128 in the warp, wider ones (3 of the 55 steps of
// 1024 keys) go through shared memory.  Bound by the barriers of those and by instruction issue (6 M Gaussians, tiles of 257 to 2048
// pairs: 56 % of the cycles).
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
gs_sort_tiles_kernel(const uint2* __restrict__ ranges, const uint64_t* __restrict__ keys, uint32_t* __restrict__ vals, int least) {
  extern __shared__ __align__(16) uint64_t s_keys[];        // [8][kThreads]
  const uint2 range = ranges[blockIdx.x];
  const int n = (int)(range.y - range.x), tid = threadIdx.x;
  if (n <= least || n > 8 * kThreads) return;
  const int holders = (n + 7) / 8;                           // threads that hold keys
  const int threads = (holders + 31) & ~31;                  // their warps
  const bool active = tid < threads;
  uint64_t key[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {                              // any order will do
    const int at = e * holders + tid;
    key[e] = tid < holders && at < n ? keys[range.x + at] : ~0ull;
  }
  if (active) {
#pragma unroll
    for (int k = 2; k <= 8; k <<= 1) {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (!(e & k >> 1)) order(key[e], key[e ^ (k - 1)]);
#pragma unroll
      for (int j = k >> 2; j > 0; j >>= 1)
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (!(e & j)) order(key[e], key[e + j]);
    }
  }
  for (int k = 16; k < 16 * holders; k <<= 1) {
    for (int j = k >> 1; j >= 256; j >>= 1) {
      const bool mirror = 2 * j == k;
      const int partner = mirror ? tid ^ (k / 8 - 1) : tid ^ (j / 8);
      __syncthreads();
      if (active) {
#pragma unroll
        for (int e = 0; e < 8; ++e) s_keys[e * kThreads + tid] = key[e];
      }
      __syncthreads();
      if (active && partner < threads) {
        const bool low = partner > tid;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const uint64_t other = s_keys[(mirror ? 7 - e : e) * kThreads + partner];
          key[e] = (other < key[e]) == low ? other : key[e];
        }
      }
    }
    if (active) {
      if (k <= 256) {
        uint64_t other[8];
        const bool low = !(tid & k / 16);
#pragma unroll
        for (int e = 0; e < 8; ++e) other[e] = __shfl_xor_sync(0xffffffffu, key[7 - e], k / 8 - 1);
#pragma unroll
        for (int e = 0; e < 8; ++e) key[e] = (other[e] < key[e]) == low ? other[e] : key[e];
      }
      for (int j = min(k >> 2, 128); j >= 8; j >>= 1) {
        const bool low = !(tid & j / 8);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const uint64_t other = __shfl_xor_sync(0xffffffffu, key[e], j / 8);
          key[e] = (other < key[e]) == low ? other : key[e];
        }
      }
#pragma unroll
      for (int j = 4; j > 0; j >>= 1)
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (!(e & j)) order(key[e], key[e + j]);
    }
  }
  // out through shared memory, so that a warp stores consecutive values
  uint32_t* s_vals = reinterpret_cast<uint32_t*>(s_keys);
  __syncthreads();
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (tid * 8 + e < n) s_vals[tid * 8 + e] = (uint32_t)key[e];
  __syncthreads();
  for (int at = tid; at < n; at += kThreads) vals[range.x + at] = s_vals[at];
}

// ---- tile blending --------------------------------------------------------------------------------------------
// A block blends one 16x16 tile, a warp one 8x4 part of it.  The tile's records are staged 256 at a time together with a
// byte that says which of the 8 warps they reach; every warp then walks only the records that reach its own pixels.
// Projected Gaussians of a large scene are small (radius about 3 pixels on average in a 6 M cloud at 1080p), so a record
// reaches 1.3 - 1.6 of the 8 warps and the walk is that much shorter than one over the whole tile list.  The kernels are
// bound by the instructions of the walk: forward 1994 -> 539 us (6 M Gaussians, 1080p), backward 1439 -> 529 us (1.5 M)
// against every pixel evaluating every record of its tile.
struct TileWarp {
  int px, py;            // this lane's pixel
  int tile_px, tile_py;  // the tile's first pixel
};

__device__ __forceinline__ TileWarp tile_warp() {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  TileWarp t;
  t.tile_px = blockIdx.x * kTile; t.tile_py = blockIdx.y * kTile;
  t.px = t.tile_px + (w & 1) * 8 + (lane & 7);
  t.py = t.tile_py + (w >> 1) * 4 + (lane >> 3);
  return t;
}

// bit w: the record's reach touches warp w's 8x4 pixels
__device__ __forceinline__ uint32_t reach_mask(float4 q0, const TileWarp& t) {
  const float lx = q0.x - q0.z - t.tile_px, hx = q0.x + q0.z - t.tile_px;
  const float ly = q0.y - q0.w - t.tile_py, hy = q0.y + q0.w - t.tile_py;
  const uint32_t cols = (lx <= 7.f && hx >= 0.f ? 1u : 0u) | (lx <= 15.f && hx >= 8.f ? 2u : 0u);
  uint32_t m = 0;
#pragma unroll
  for (int r = 0; r < 4; ++r)
    if (ly <= 4.f * r + 3.f && hy >= 4.f * r) m |= cols << (2 * r);
  return m;
}

__global__ void __launch_bounds__(kTilePixels, 8)
gs_render_fwd_kernel(const uint2* __restrict__ ranges, const uint32_t* __restrict__ point_list, int W, int H,
                     const float4* __restrict__ rec, const float* __restrict__ bg, float* __restrict__ out_color,
                     float* __restrict__ out_alpha, float* __restrict__ final_T, uint32_t* __restrict__ n_contrib) {
  __shared__ float2 s_xy[kTilePixels];
  __shared__ float4 s_co[kTilePixels];
  __shared__ float4 s_rgb[kTilePixels];
  __shared__ unsigned char s_mask[kTilePixels];
  const TileWarp tw = tile_warp();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const bool inside = tw.px < W && tw.py < H;
  const float2 pixf = make_float2((float)tw.px, (float)tw.py);
  const uint2 range = ranges[blockIdx.y * gridDim.x + blockIdx.x];
  bool done = !inside;
  float T = 1.f, C[3] = {0.f, 0.f, 0.f};
  uint32_t last = 0;
  uint32_t next = range.x + tid < range.y ? point_list[range.x + tid] : 0u;
  for (uint32_t base = range.x; base < range.y; base += kTilePixels) {
    if (!__syncthreads_or(!done)) break;
    uint32_t mask = 0;
    if (base + tid < range.y) {
      const float4 q0 = __ldg(rec + 3LL * next);
      s_xy[tid] = make_float2(q0.x, q0.y);
      s_co[tid] = __ldg(rec + 3LL * next + 1);
      s_rgb[tid] = __ldg(rec + 3LL * next + 2);
      mask = reach_mask(q0, tw);
    }
    s_mask[tid] = (unsigned char)mask;
    const uint32_t ahead = base + kTilePixels + tid;
    if (ahead < range.y) next = point_list[ahead];
    __syncthreads();
    for (int g = 0; g < kTilePixels; g += 32) {
      if (__all_sync(0xffffffffu, done)) break;
      uint32_t m = __ballot_sync(0xffffffffu, s_mask[g + lane] >> w & 1u);
      while (m) {
        const int j = g + __ffs(m) - 1;
        m &= m - 1;
        const float2 xy = s_xy[j];
        const float4 co = s_co[j];
        const float2 d = make_float2(xy.x - pixf.x, xy.y - pixf.y);
        const float power = -0.5f * (co.x * d.x * d.x + co.z * d.y * d.y) - co.y * d.x * d.y;
        const float alpha = fminf(0.99f, co.w * __expf(power));
        if (done || power > 0.f || alpha < kAlphaMin) continue;
        const float test_T = T * (1.f - alpha);
        if (test_T < 1e-4f) { done = true; continue; }
        const float wgt = alpha * T;
        const float4 c = s_rgb[j];
        C[0] += c.x * wgt; C[1] += c.y * wgt; C[2] += c.z * wgt;
        T = test_T;
        last = base - range.x + j + 1;
      }
    }
  }
  if (inside) {
    const long long pix = (long long)tw.py * W + tw.px;
    final_T[pix] = T;
    out_alpha[pix] = 1.f - T;
    n_contrib[pix] = last;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) out_color[(long long)ch * H * W + pix] = C[ch] + T * bg[ch];
  }
}

// Sum of v[0..7] over the warp: lane L ends with the total of v[L >> 2] (halving the number of values while doubling the
// lanes that share one: 4 + 2 + 1 + 2 shuffles instead of 8 x 5).
__device__ __forceinline__ float warp_sum8(const float (&v)[8]) {
  const int lane = threadIdx.x & 31;
  float a[4], b[2], c;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float keep = lane & 16 ? v[4 + k] : v[k], send = lane & 16 ? v[k] : v[4 + k];
    a[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float keep = lane & 8 ? a[2 + k] : a[k], send = lane & 8 ? a[k] : a[2 + k];
    b[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  const float keep = lane & 4 ? b[1] : b[0], send = lane & 4 ? b[0] : b[1];
  c = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// Gradient record of a Gaussian, 12 floats: {mean x, y, conic a, b}, {conic c, opacity, r, g}, {b, -, -, -}.  A warp adds
// its nine sums with one request (nine lanes, consecutive addresses).  The walk starts at the last record that any pixel of
// the tile blended: what lies behind it was never reached by the forward pass.
constexpr int kGradRow = 12;

__global__ void __launch_bounds__(kTilePixels, 5)
gs_render_bwd_kernel(const uint2* __restrict__ ranges, const uint32_t* __restrict__ point_list, int W, int H,
                     const float* __restrict__ bg, const float4* __restrict__ rec, const float* __restrict__ final_T,
                     const uint32_t* __restrict__ n_contrib, const float* __restrict__ dL_dpix, float* __restrict__ grad) {
  __shared__ uint32_t s_id[kTilePixels];
  __shared__ float2 s_xy[kTilePixels];
  __shared__ float4 s_co[kTilePixels];
  __shared__ float4 s_rgb[kTilePixels];
  __shared__ unsigned char s_mask[kTilePixels];
  __shared__ int s_last[kTilePixels / 32];
  const TileWarp tw = tile_warp();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const bool inside = tw.px < W && tw.py < H;
  const long long pix = (long long)tw.py * W + tw.px;
  const float2 pixf = make_float2((float)tw.px, (float)tw.py);
  const uint2 range = ranges[blockIdx.y * gridDim.x + blockIdx.x];
  const float T_final = inside ? final_T[pix] : 0.f;
  float T = T_final;
  const int last = inside ? (int)n_contrib[pix] : 0;
  const int warp_last = __reduce_max_sync(0xffffffffu, last);
  if (lane == 0) s_last[w] = warp_last;
  __syncthreads();
  int count = 0;
#pragma unroll
  for (int k = 0; k < kTilePixels / 32; ++k) count = max(count, s_last[k]);
  float accum[3] = {0.f, 0.f, 0.f}, dpix[3] = {0.f, 0.f, 0.f}, last_color[3] = {0.f, 0.f, 0.f};
  float last_alpha = 0.f;
  if (inside) {
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) dpix[ch] = dL_dpix[(long long)ch * H * W + pix];
  }
  const float bg_dot = bg[0] * dpix[0] + bg[1] * dpix[1] + bg[2] * dpix[2];
  const float ddelx_dx = 0.5f * W, ddely_dy = 0.5f * H;
  uint32_t next = tid < count ? point_list[range.x + count - 1 - tid] : 0u;
  for (int left = count; left > 0; left -= kTilePixels) {       // records left..1 of the list, back to front
    __syncthreads();
    uint32_t mask = 0;
    if (tid < left) {
      const float4 q0 = __ldg(rec + 3LL * next);
      s_id[tid] = next;
      s_xy[tid] = make_float2(q0.x, q0.y);
      s_co[tid] = __ldg(rec + 3LL * next + 1);
      s_rgb[tid] = __ldg(rec + 3LL * next + 2);
      mask = reach_mask(q0, tw);
    }
    s_mask[tid] = (unsigned char)mask;
    const int ahead = left - kTilePixels - 1 - tid;
    if (ahead >= 0) next = point_list[range.x + ahead];
    __syncthreads();
    for (int g = 0; g < kTilePixels; g += 32) {
      uint32_t m = __ballot_sync(0xffffffffu, (s_mask[g + lane] >> w & 1u) && left - (g + lane) <= warp_last);
      while (m) {
        const int j = g + __ffs(m) - 1;
        m &= m - 1;
        bool active = left - j <= last;
        const float2 xy = s_xy[j];
        const float4 co = s_co[j];
        const float2 d = make_float2(xy.x - pixf.x, xy.y - pixf.y);
        const float power = -0.5f * (co.x * d.x * d.x + co.z * d.y * d.y) - co.y * d.x * d.y;
        const float G = __expf(power);
        const float alpha = fminf(0.99f, co.w * G);
        active = active && power <= 0.f && alpha >= kAlphaMin;
        if (!__any_sync(0xffffffffu, active)) continue;
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, v8 = 0.f;
        if (active) {
          const float4 c4 = s_rgb[j];
          const float col[3] = {c4.x, c4.y, c4.z};
          T = T / (1.f - alpha);
          const float dchannel_dcolor = alpha * T;
          float dL_dalpha = 0.f;
#pragma unroll
          for (int ch = 0; ch < 3; ++ch) {
            accum[ch] = last_alpha * last_color[ch] + (1.f - last_alpha) * accum[ch];
            last_color[ch] = col[ch];
            dL_dalpha += (col[ch] - accum[ch]) * dpix[ch];
          }
          dL_dalpha *= T;
          last_alpha = alpha;
          dL_dalpha += (-T_final / (1.f - alpha)) * bg_dot;
          const float free = co.w * G <= 0.99f ? 1.f : 0.f;       // the clamp passes no gradient
          const float dL_dG = co.w * dL_dalpha * free;
          const float gdx = G * d.x, gdy = G * d.y;
          v[0] = dL_dG * (-gdx * co.x - gdy * co.y) * ddelx_dx;
          v[1] = dL_dG * (-gdy * co.z - gdx * co.y) * ddely_dy;
          v[2] = -0.5f * gdx * d.x * dL_dG;
          v[3] = -0.5f * gdx * d.y * dL_dG;
          v[4] = -0.5f * gdy * d.y * dL_dG;
          v[5] = G * dL_dalpha * free;
          v[6] = dchannel_dcolor * dpix[0];
          v[7] = dchannel_dcolor * dpix[1];
          v8 = dchannel_dcolor * dpix[2];
        }
        const float total = warp_sum8(v), total8 = warp_sum(v8);
        float* row = grad + (long long)s_id[j] * kGradRow;
        if ((lane & 3) == 0 || lane == 1) atomicAdd(row + (lane == 1 ? 8 : lane >> 2), lane == 1 ? total8 : total);
      }
    }
  }
}

// ---- preprocess backward -----------------------------------------------------------------------------------------
// Every output row is written, zeros for Gaussians that were not rendered, so the caller allocates without clearing.
// Bound by memory (384 B of SH rows in and out per Gaussian); 503 -> 159 us at 1.5 M with the rows staged.
__global__ void __launch_bounds__(kPreThreads)
gs_preprocess_bwd_kernel(int N, const float* __restrict__ means, const float* __restrict__ scales, const float* __restrict__ rots,
                         const float* __restrict__ shs, const float* __restrict__ sh_rest, const float* __restrict__ cov3d_pre,
                         const int* __restrict__ radii, GSCameraInfo info, const float* __restrict__ pose,
                         const float4* __restrict__ grad, float* __restrict__ dL_dmeans,
                         float* __restrict__ dL_dmeans2D, float* __restrict__ dL_dopacity, float* __restrict__ dL_dscales,
                         float* __restrict__ dL_drots, float* __restrict__ dL_dshs,
                         float* __restrict__ dL_dsh_rest, float* __restrict__ dL_dcolors_pre) {
  extern __shared__ __align__(16) float s_sh[];
  __shared__ GSCameraPose s_pose;
  const GSCamera cam = load_camera(info, pose, s_pose);
  const int i = blockIdx.x * kPreThreads + threadIdx.x;
  const long long first = (long long)blockIdx.x * kPreThreads + (threadIdx.x & ~31);
  if (first >= N) return;
  const bool on = i < N && radii[i] > 0;
  const uint32_t rows = __ballot_sync(0xffffffffu, on);
  float3 p = make_float3(0.f, 0.f, 0.f), dmean = p, dscale = p;
  float4 g0 = make_float4(0.f, 0.f, 0.f, 0.f), g1 = g0, g2 = g0, dq = g0;
  float dL_dcov[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (on) {
    g0 = __ldg(grad + 3LL * i); g1 = __ldg(grad + 3LL * i + 1); g2 = __ldg(grad + 3LL * i + 2);
    p = make_float3(means[3 * i], means[3 * i + 1], means[3 * i + 2]);
  }
  if (on) {
    const float3 t = xform43(cam.view, p);
    const float fx = cam.W / (2.f * cam.tanfovx), fy = cam.H / (2.f * cam.tanfovy);
    float c3[6];
    if (cov3d_pre) {
#pragma unroll
      for (int k = 0; k < 6; ++k) c3[k] = cov3d_pre[6 * (long long)i + k];
    } else {
      cov3d_from(make_float3(scales[3 * i] * cam.scale_modifier, scales[3 * i + 1] * cam.scale_modifier,
                             scales[3 * i + 2] * cam.scale_modifier), __ldg(reinterpret_cast<const float4*>(rots) + i), c3);
    }
    float T[6], a, b, c;
    project_cov(cam, t, c3, fx, fy, T, a, b, c);
    a += 0.3f; c += 0.3f;
    const float denom = a * c - b * b;
    const float denom2inv = 1.f / (denom * denom + 1e-7f);
    const float gcx = g0.z, gcy = g0.w, gcz = g1.x;
    float dL_da = 0.f, dL_db = 0.f, dL_dc = 0.f;
    float dT[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (denom2inv != 0.f) {
      // conic = (c, -b, a) / denom
      dL_da = denom2inv * (-c * c * gcx + 2.f * b * c * gcy + (denom - a * c) * gcz);
      dL_dc = denom2inv * (-a * a * gcz + 2.f * a * b * gcy + (denom - a * c) * gcx);
      dL_db = denom2inv * 2.f * (b * c * gcx - (denom + 2.f * b * b) * gcy + a * b * gcz);
      // cov2D = T Sigma T^T  ->  d/dSigma
      dL_dcov[0] = T[0] * T[0] * dL_da + T[0] * T[3] * dL_db + T[3] * T[3] * dL_dc;
      dL_dcov[3] = T[1] * T[1] * dL_da + T[1] * T[4] * dL_db + T[4] * T[4] * dL_dc;
      dL_dcov[5] = T[2] * T[2] * dL_da + T[2] * T[5] * dL_db + T[5] * T[5] * dL_dc;
      dL_dcov[1] = 2.f * T[0] * T[1] * dL_da + (T[0] * T[4] + T[1] * T[3]) * dL_db + 2.f * T[3] * T[4] * dL_dc;
      dL_dcov[2] = 2.f * T[0] * T[2] * dL_da + (T[0] * T[5] + T[2] * T[3]) * dL_db + 2.f * T[3] * T[5] * dL_dc;
      dL_dcov[4] = 2.f * T[2] * T[1] * dL_da + (T[1] * T[5] + T[2] * T[4]) * dL_db + 2.f * T[4] * T[5] * dL_dc;
      // d/dT
      const float S0[3] = {c3[0], c3[1], c3[2]}, S1[3] = {c3[1], c3[3], c3[4]}, S2[3] = {c3[2], c3[4], c3[5]};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float st0 = S0[k] * T[0] + S1[k] * T[1] + S2[k] * T[2];   // (Sigma T0^T)_k
        const float st1 = S0[k] * T[3] + S1[k] * T[4] + S2[k] * T[5];
        dT[k] = 2.f * st0 * dL_da + st1 * dL_db;
        dT[3 + k] = 2.f * st1 * dL_dc + st0 * dL_db;
      }
    }
    // T = J Wr ; J entries: j00 = fx/tz, j02 = -fx*txz/tz^2, j11 = fy/tz, j12 = -fy*tyz/tz^2
    const float* v = cam.view;
    const float dJ00 = v[0] * dT[0] + v[4] * dT[1] + v[8] * dT[2];
    const float dJ02 = v[2] * dT[0] + v[6] * dT[1] + v[10] * dT[2];
    const float dJ11 = v[1] * dT[3] + v[5] * dT[4] + v[9] * dT[5];
    const float dJ12 = v[2] * dT[3] + v[6] * dT[4] + v[10] * dT[5];
    const float limx = 1.3f * cam.tanfovx, limy = 1.3f * cam.tanfovy;
    const float rx = t.x / t.z, ry = t.y / t.z;
    const float txz = fminf(limx, fmaxf(-limx, rx)) * t.z, tyz = fminf(limy, fmaxf(-limy, ry)) * t.z;
    const float x_grad_mul = (rx < -limx || rx > limx) ? 0.f : 1.f;
    const float y_grad_mul = (ry < -limy || ry > limy) ? 0.f : 1.f;
    const float tz = 1.f / t.z, tz2 = tz * tz, tz3 = tz2 * tz;
    const float dL_dtx = x_grad_mul * -fx * tz2 * dJ02;
    const float dL_dty = y_grad_mul * -fy * tz2 * dJ12;
    const float dL_dtz = -fx * tz2 * dJ00 - fy * tz2 * dJ11 + (2.f * fx * txz) * tz3 * dJ02 + (2.f * fy * tyz) * tz3 * dJ12;
    // view = [p 1] @ V -> d p_j = sum_i V[j*4+i] d t_i
    dmean = make_float3(v[0] * dL_dtx + v[1] * dL_dty + v[2] * dL_dtz, v[4] * dL_dtx + v[5] * dL_dty + v[6] * dL_dtz,
                               v[8] * dL_dtx + v[9] * dL_dty + v[10] * dL_dtz);
    // screen-space mean gradient through the projection
    {
      const float4 mh = xform44(cam.proj, p);
      const float mw = 1.f / (mh.w + 1e-7f);
      const float* m = cam.proj;
      const float gx = g0.x, gy = g0.y;
      const float mul1 = (m[0] * p.x + m[4] * p.y + m[8] * p.z + m[12]) * mw * mw;
      const float mul2 = (m[1] * p.x + m[5] * p.y + m[9] * p.z + m[13]) * mw * mw;
      dmean.x += (m[0] * mw - m[3] * mul1) * gx + (m[1] * mw - m[3] * mul2) * gy;
      dmean.y += (m[4] * mw - m[7] * mul1) * gx + (m[5] * mw - m[7] * mul2) * gy;
      dmean.z += (m[8] * mw - m[11] * mul1) * gx + (m[9] * mw - m[11] * mul2) * gy;
    }
    if (dL_dscales) {
      // Sigma = M M^T with M = R diag(s): dL/dM = 2 * dSigma_sym * M
      const float3 s = make_float3(scales[3 * i] * cam.scale_modifier, scales[3 * i + 1] * cam.scale_modifier,
                                   scales[3 * i + 2] * cam.scale_modifier);
      const float4 q0 = __ldg(reinterpret_cast<const float4*>(rots) + i);
      float R[9];
      quat_to_rot(q0, R);
      // symmetric dSigma with off-diagonals halved (each appears twice in the full matrix)
      const float D[9] = {dL_dcov[0], 0.5f * dL_dcov[1], 0.5f * dL_dcov[2], 0.5f * dL_dcov[1], dL_dcov[3], 0.5f * dL_dcov[4],
                          0.5f * dL_dcov[2], 0.5f * dL_dcov[4], dL_dcov[5]};
      const float sv[3] = {s.x, s.y, s.z};
      float dM[9];   // dL/dM, M[r][c] = R[r][c] * s[c]
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
          float acc = 0.f;
#pragma unroll
          for (int k = 0; k < 3; ++k) acc += D[r * 3 + k] * R[k * 3 + cc] * sv[cc];
          dM[r * 3 + cc] = 2.f * acc;
        }
      float ds[3], dR[9];
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        ds[cc] = (R[cc] * dM[cc] + R[3 + cc] * dM[3 + cc] + R[6 + cc] * dM[6 + cc]) * cam.scale_modifier;
#pragma unroll
        for (int r = 0; r < 3; ++r) dR[r * 3 + cc] = dM[r * 3 + cc] * sv[cc];
      }
      dscale = make_float3(ds[0], ds[1], ds[2]);
      const float r = q0.x, x = q0.y, y = q0.z, z = q0.w;
      dq.x = 2.f * (-z * dR[1] + y * dR[2] + z * dR[3] - x * dR[5] - y * dR[6] + x * dR[7]);
      dq.y = 2.f * (y * dR[1] + z * dR[2] + y * dR[3] - 2.f * x * dR[4] - r * dR[5] + z * dR[6] + r * dR[7] - 2.f * x * dR[8]);
      dq.z = 2.f * (-2.f * y * dR[0] + x * dR[1] + r * dR[2] + x * dR[3] + z * dR[5] - r * dR[6] + z * dR[7] - 2.f * y * dR[8]);
      dq.w = 2.f * (-2.f * z * dR[0] - r * dR[1] + x * dR[2] + r * dR[3] - 2.f * z * dR[4] + y * dR[5] + x * dR[6] + y * dR[7]);
    }
  }
  if (shs) {
    const SHRows s = sh_layout(s_sh, cam.sh_coeffs, sh_rest != nullptr);
    const int n_rows = (int)min(32LL, N - first);
    if (rows) {
      sh_rows_load(shs, first, n_rows, s.row0, rows, s.s0);
      if (s.row1) sh_rows_load(sh_rest, first, n_rows, s.row1, rows, s.s1);
    }
    __syncwarp();
    float *sh0 = s.lane0, *sh = s.lane1 - 3;
    if (on) {
      const float3 dir0 = make_float3(p.x - cam.campos[0], p.y - cam.campos[1], p.z - cam.campos[2]);
      const float n2 = dir0.x * dir0.x + dir0.y * dir0.y + dir0.z * dir0.z;
      const float invn = rsqrtf(n2);
      const float3 d = make_float3(dir0.x * invn, dir0.y * invn, dir0.z * invn);
      float B[16];
      sh_basis(cam.sh_degree, d, B);
      const int nb = (cam.sh_degree + 1) * (cam.sh_degree + 1);
      // colour clamped at zero: recomputed with the forward kernel's sums
      float3 v = make_float3(0.5f + B[0] * sh0[0], 0.5f + B[0] * sh0[1], 0.5f + B[0] * sh0[2]);
#pragma unroll
      for (int k = 1; k < 16; ++k)
        if (k < nb) { v.x += B[k] * sh[3 * k]; v.y += B[k] * sh[3 * k + 1]; v.z += B[k] * sh[3 * k + 2]; }
      const float3 g = make_float3(v.x < 0.f ? 0.f : g1.z, v.y < 0.f ? 0.f : g1.w, v.z < 0.f ? 0.f : g2.x);
      float Bx[16], By[16], Bz[16];
      sh_basis_grad(cam.sh_degree, d, Bx, By, Bz);
      float3 ddir = make_float3(0.f, 0.f, 0.f);               // the constant term does not depend on the direction
      sh0[0] = B[0] * g.x; sh0[1] = B[0] * g.y; sh0[2] = B[0] * g.z;
#pragma unroll
      for (int k = 1; k < 16; ++k)
        if (k < nb) {
          const float t = sh[3 * k] * g.x + sh[3 * k + 1] * g.y + sh[3 * k + 2] * g.z;
          ddir.x += Bx[k] * t; ddir.y += By[k] * t; ddir.z += Bz[k] * t;
          sh[3 * k] = B[k] * g.x; sh[3 * k + 1] = B[k] * g.y; sh[3 * k + 2] = B[k] * g.z;
        }
      for (int k = 3 * nb; k < cam.sh_coeffs * 3; ++k) sh[k] = 0.f;
      // backward of normalisation: (I - d d^T) / |dir0|
      const float dot = d.x * ddir.x + d.y * ddir.y + d.z * ddir.z;
      dmean.x += (ddir.x - d.x * dot) * invn; dmean.y += (ddir.y - d.y * dot) * invn; dmean.z += (ddir.z - d.z * dot) * invn;
    } else {
      sh0[0] = sh0[1] = sh0[2] = 0.f;
      for (int k = 3; k < cam.sh_coeffs * 3; ++k) sh[k] = 0.f;
    }
    __syncwarp();
    sh_rows_store(dL_dshs, first, n_rows, s.row0, s.s0);
    if (s.row1) sh_rows_store(dL_dsh_rest, first, n_rows, s.row1, s.s1);
  }
  if (i >= N) return;
  dL_dmeans[3 * i] = dmean.x; dL_dmeans[3 * i + 1] = dmean.y; dL_dmeans[3 * i + 2] = dmean.z;
  dL_dmeans2D[3 * i] = g0.x; dL_dmeans2D[3 * i + 1] = g0.y; dL_dmeans2D[3 * i + 2] = 0.f;
  dL_dopacity[i] = g1.y;
  if (dL_dcolors_pre) { dL_dcolors_pre[3 * i] = g1.z; dL_dcolors_pre[3 * i + 1] = g1.w; dL_dcolors_pre[3 * i + 2] = g2.x; }
  if (dL_dscales) {
    dL_dscales[3 * i] = dscale.x; dL_dscales[3 * i + 1] = dscale.y; dL_dscales[3 * i + 2] = dscale.z;
    reinterpret_cast<float4*>(dL_drots)[i] = dq;
  }
}

}  // namespace lmb

using namespace lmb;

// Float4-read arrays (rots, shs, sh_rest and their gradients) start on 16 bytes.  pose: device, {view, proj, campos}.
// tiles_touched: [N].  sh_rest null: shs holds [N, sh_coeffs, 3], otherwise shs [N, 1, 3] and sh_rest [N, sh_coeffs - 1, 3].
static int preprocess(int N, const float* means, const float* scales, const float* rots, const float* opac,
                              const float* shs, const float* sh_rest, const float* colors_pre, const float* cov3d_pre,
                              const unsigned char* visible, const GSCameraInfo* cam, const float* pose, int* radii, float* rec,
                              uint32_t* tiles_touched, uint32_t* tile_counts, int per_tile, int radius_only,
                              cudaStream_t stream) {
  if (N <= 0) return 0;
  const size_t smem = shs && !radius_only ? (size_t)(kPreThreads / 32) * sh_warp_floats(cam->sh_coeffs) * sizeof(float) : 0;
  gs_preprocess_kernel<<<ceil_div(N, kPreThreads), kPreThreads, smem, stream>>>(N, means, scales, rots, opac, shs, sh_rest,
      colors_pre, cov3d_pre, visible, *cam, pose, radii, (float4*)rec, tiles_touched, tile_counts, per_tile, radius_only);
  LMB_LAUNCH_CHECK();
  return 0;
}

static int n_tiles_of(int W, int H) { return ((W + kTile - 1) / kTile) * ((H + kTile - 1) / kTile); }

// Words of tile_cursors for a tile.
LMB_API int lmb_gs_tile_words(int N, int W, int H) { return tile_counters(N, n_tiles_of(W, H)) * kCounterStride; }

static int render_fwd(const uint32_t* ranges, const uint32_t* point_list, int W, int H, const float* rec, const float* bg,
                      float* out_color, float* out_alpha, float* final_T, uint32_t* n_contrib, cudaStream_t stream) {
  dim3 grid((W + kTile - 1) / kTile, (H + kTile - 1) / kTile);
  gs_render_fwd_kernel<<<grid, kTilePixels, 0, stream>>>((const uint2*)ranges, point_list, W, H, (const float4*)rec, bg,
                                                         out_color, out_alpha, final_T, n_contrib);
  LMB_LAUNCH_CHECK();
  return 0;
}

LMB_API long long lmb_scan_scratch_bytes(long long n);
LMB_API int lmb_exclusive_scan_u32(const uint32_t* in, uint32_t* out, long long n, void* scratch, cudaStream_t stream);
LMB_API long long lmb_radix_sort_scratch_bytes(long long max_n);
LMB_API int lmb_radix_sort_pairs(uint64_t* keys, uint32_t* vals, const int* count_ptr, long long max_n, int begin_bit, int end_bit,
                                 void* scratch, cudaStream_t stream);

// A frame is two calls around the two values that the host must know, the number of (splat, tile) pairs and that of the fullest
// tile: a small frame spends its time in calls and allocations.
// First call: records, radii, the range of every tile (ranges) and where its pairs go (tile_cursors, [tiles, lmb_gs_tile_words], of which
// the first word of every 8 counts and the first of all is the tile's start; one draw uses them up); totals: [2].  visible_filter passes radius_only and none of these.  See preprocess for the other arrays.
LMB_API int lmb_gs_project(int N, const float* means, const float* scales, const float* rots, const float* opac, const float* shs,
                           const float* sh_rest, const float* colors_pre, const float* cov3d_pre, const unsigned char* visible,
                           const GSCameraInfo* cam, const float* pose, int* radii, float* rec, uint32_t* tiles_touched,
                           uint32_t* tile_cursors, uint32_t* ranges, uint32_t* totals, int radius_only, cudaStream_t stream) {
  const int n_tiles = n_tiles_of(cam->W, cam->H);
  const int per_tile = tile_counters(N, n_tiles), counters = n_tiles * per_tile;
  if (!radius_only) LMB_CUDA_TRY(cudaMemsetAsync(tile_cursors, 0, (size_t)counters * kCounterStride * 4, stream));
  const int rc = preprocess(N, means, scales, rots, opac, shs, sh_rest, colors_pre, cov3d_pre, visible, cam, pose, radii, rec,
                            tiles_touched, tile_cursors, per_tile, radius_only, stream);
  if (rc || radius_only) return rc;
  const int chunks = ceil_div(counters, kScanChunk);
  if (chunks > 1) {
    gs_tile_sums_kernel<<<chunks, kScanBlock, 0, stream>>>(counters, tile_cursors, totals);
    LMB_LAUNCH_CHECK();
  }
  gs_tile_scan_kernel<<<chunks, kScanBlock, 0, stream>>>(counters, per_tile, tile_cursors, (uint2*)ranges, totals);
  LMB_LAUNCH_CHECK();
  return 0;
}

// The fullest tile that a block sorts: 64 KB of shared memory.  A view with a fuller one pays for the counts beside the sort of all pairs,
// which gives it the ranges too: 6 M Gaussians at 960 x 540 1515 -> 1550 - 1599 us a frame, at 320 x 180 3160 -> 3190, in 28 tiles 10.9 ->
// 11.05 ms, 400 k at 320 x 180 700 -> 705.
constexpr uint32_t kTileSortMax = 8192;

static long long draw_work_bytes(int N, long long total) {
  const long long scan = lmb_scan_scratch_bytes(N), sort = lmb_radix_sort_scratch_bytes(total);
  return ((scan > sort ? scan : sort) + 255) & ~255LL;
}

// Bytes of scratch of the second call: none where every tile is sorted by a block, else the sums of the touched tiles and what
// their scan and the sort of all pairs need.
LMB_API long long lmb_gs_sort_scratch_bytes(int N, long long total, long long most) {
  if (most <= kTileSortMax) return 0;
  return draw_work_bytes(N, total) + (long long)N * 4;
}

template <int kThreads>
static int sort_tiles(int n_tiles, const uint32_t* ranges, const uint64_t* keys, uint32_t* vals, int least, cudaStream_t stream) {
  constexpr int smem = 8 * kThreads * sizeof(uint64_t);
  if (smem > 48 * 1024)
    LMB_CUDA_TRY(cudaFuncSetAttribute(gs_sort_tiles_kernel<kThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  gs_sort_tiles_kernel<kThreads><<<n_tiles, kThreads, smem, stream>>>((const uint2*)ranges, keys, vals, least);
  LMB_LAUNCH_CHECK();
  return 0;
}

// Second call: the `total` pairs in tile and depth order (vals) and the image; `most` pairs in the fullest tile.  keys: [total];
// tiles_touched, tile_cursors, ranges: of the first call; scratch: lmb_gs_sort_scratch_bytes; final_T, n_contrib: [H, W], kept
// for the backward.
LMB_API int lmb_gs_draw(int N, const float* rec, const int* radii, uint32_t* tiles_touched, uint32_t* tile_cursors, int W, int H,
                        long long total, long long most, uint64_t* keys, uint32_t* vals, void* scratch, const uint32_t* ranges,
                        const float* bg, float* out_color, float* out_alpha, float* final_T, uint32_t* n_contrib, cudaStream_t stream) {
  const int n_tiles = n_tiles_of(W, H);
  int rc = 0, tile_bits = 1;
  while ((1LL << tile_bits) < n_tiles) ++tile_bits;
  if (total > 0 && most > kTileSortMax) {
    uint32_t* offsets = (uint32_t*)((unsigned char*)scratch + draw_work_bytes(N, total));
    rc = lmb_exclusive_scan_u32(tiles_touched, offsets, N, scratch, stream);
    if (rc) return rc;
    gs_make_keys_kernel<<<ceil_div(N, 256), 256, 0, stream>>>(N, (const float4*)rec, radii, tiles_touched, offsets, W, H, total, keys, vals);
    LMB_LAUNCH_CHECK();
    rc = lmb_radix_sort_pairs(keys, vals, nullptr, total, 0, 32 + tile_bits, scratch, stream);
  } else if (total > 0) {
    gs_drop_pairs_kernel<<<ceil_div(N, 256), 256, 0, stream>>>(N, (const float4*)rec, radii, tiles_touched, W, H, total,
                                                                tile_counters(N, n_tiles), tile_cursors, keys);
    LMB_LAUNCH_CHECK();
    // a warp per tile of up to 256 pairs, 8 warps up to 2048, 16 and 32 beyond; a class without tiles costs a launch at most
    rc = sort_tiles<32>(n_tiles, ranges, keys, vals, 0, stream);
    if (!rc && most > 256) rc = sort_tiles<256>(n_tiles, ranges, keys, vals, 256, stream);
    if (!rc && most > 2048) rc = sort_tiles<512>(n_tiles, ranges, keys, vals, 2048, stream);
    if (!rc && most > 4096) rc = sort_tiles<1024>(n_tiles, ranges, keys, vals, 4096, stream);
  }
  if (!rc) rc = render_fwd(ranges, vals, W, H, rec, bg, out_color, out_alpha, final_T, n_contrib, stream);
  return rc;
}

// grad: [N, 12] floats, zeroed by the caller
LMB_API int lmb_gs_render_bwd(const uint32_t* ranges, const uint32_t* point_list, int W, int H, const float* bg,
                              const float* rec, const float* final_T, const uint32_t* n_contrib, const float* dL_dpix,
                              float* grad, cudaStream_t stream) {
  dim3 grid((W + kTile - 1) / kTile, (H + kTile - 1) / kTile);
  gs_render_bwd_kernel<<<grid, kTilePixels, 0, stream>>>((const uint2*)ranges, point_list, W, H, bg, (const float4*)rec, final_T,
                                                         n_contrib, dL_dpix, grad);
  LMB_LAUNCH_CHECK();
  return 0;
}

// dL_dscales / dL_drots and dL_dcolors_pre may be null
LMB_API int lmb_gs_preprocess_bwd(int N, const float* means, const float* scales, const float* rots, const float* shs,
                                  const float* sh_rest, const float* cov3d_pre, const int* radii, const GSCameraInfo* cam,
                                  const float* pose, const float* grad,
                                  float* dL_dmeans, float* dL_dmeans2D, float* dL_dopacity, float* dL_dscales, float* dL_drots,
                                  float* dL_dshs, float* dL_dsh_rest, float* dL_dcolors_pre, cudaStream_t stream) {
  if (N <= 0) return 0;
  const size_t smem = shs ? (size_t)(kPreThreads / 32) * sh_warp_floats(cam->sh_coeffs) * sizeof(float) : 0;
  gs_preprocess_bwd_kernel<<<ceil_div(N, kPreThreads), kPreThreads, smem, stream>>>(N, means, scales, rots, shs, sh_rest, cov3d_pre,
      radii, *cam, pose, (const float4*)grad, dL_dmeans, dL_dmeans2D, dL_dopacity, dL_dscales, dL_drots, dL_dshs, dL_dsh_rest,
      dL_dcolors_pre);
  LMB_LAUNCH_CHECK();
  return 0;
}
