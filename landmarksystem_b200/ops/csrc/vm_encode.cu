// VM (vector-matrix) feature-grid lookup for GridNeRF-style fields, forward and backward.
//
// A sample carries block-local coordinates (x, y, z) in [-1, 1] and the index b of the spatial
// block that owns it.  For every resolution level l the feature is
//     bilinear(plane_l[b], x, y)  *  linear(line_l[b], z)          (element-wise over C channels)
// with align_corners=True / zero-padding semantics, and levels are concatenated: out[n, l*C + c].
// This is the math of the reference's 5-D/4-D F.grid_sample pair followed by the product
// (landmark/nerf_components/model_components/fields/encodings/tensor_vm_encoding.py:129-197) and of
// its channels-last kernel (landmark/ops/kernel/densityappfeature/grid_sampler_3d_ndhwc_kernel.cu:206-369),
// re-designed around the memory system: planes are stored channels-last [B, H, W, C] so one texel
// is one or three 32-byte sectors, each thread moves 8 channels with a single 16-byte load, and the
// plane * line product and the level concat are fused so no intermediate ever reaches HBM.
#include "common.cuh"

namespace lmb {

struct VMLevels {
  const void* plane[kMaxLevels];  // [B, H, W, C]
  const void* line[kMaxLevels];   // [B, Z, C]
  float* gplane[kMaxLevels];      // fp32 gradient accumulators, same shapes (backward only)
  float* gline[kMaxLevels];
  int H[kMaxLevels], W[kMaxLevels], Z[kMaxLevels];
  int L, C, B;
};

struct Corner2 {
  int i0, i1;
  float w0, w1;  // weights already zeroed for out-of-range taps
};

__device__ __forceinline__ Corner2 taps(float u, int size) {
  // u in [-1, 1] -> continuous index in [0, size-1] (align_corners=True); zero padding outside.
  float f = (u + 1.f) * 0.5f * (float)(size - 1);
  float fl = floorf(f);
  int i0 = (int)fl;
  float t = f - fl;
  Corner2 c;
  c.i0 = i0; c.i1 = i0 + 1;
  c.w0 = (i0 >= 0 && i0 < size) ? 1.f - t : 0.f;
  c.w1 = (c.i1 >= 0 && c.i1 < size) ? t : 0.f;
  c.i0 = min(max(c.i0, 0), size - 1);
  c.i1 = min(max(c.i1, 0), size - 1);
  return c;
}

// ---- eight channels of a sample ----------------------------------------------------------------------------------
// The forward lookups are bound by instruction issue (79 % of the slots, L1 at half of its throughput), so they keep to few
// instructions: pairs of channels in one fma.rn.f32x2 (the same roundings as two scalar ones), addresses as a 32 x 32 -> 64 bit
// multiply-add on byte strides, one unsigned comparison for "inside", and what depends on the level alone taken out of the loop
// over samples where there is one level.  1080p frame: density 7.29 -> 5.23 ms, colour features 6.66 -> 5.86; 8192 rays of 128 samples
// on 4096^2 texels: density 51.5 -> 41 us, on 1371^2 38 -> 23.  Four blocks an SM instead of five: colour features of a 320 x 180
// preview 181 against 165 us.  Three levels (512^2 to 2048^2, 1 Mi samples): density 107 -> 80 us in bf16 and 126 -> 108 in fp32, 48
// channels 225 -> 209 and 363 -> 343; their backwards as before (480 -> 473, 1590 -> 1592).
struct P8 { unsigned long long v[4]; };       // pairs of fp32

__device__ __forceinline__ unsigned long long pair_of(float lo, float hi) {
  unsigned long long p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
  return p;
}
__device__ __forceinline__ float2 halves_of(unsigned long long p) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(p));
  return f;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
template <typename T>
__device__ __forceinline__ P8 load_pairs(const char* p) {
  P8 r;
  if constexpr (sizeof(T) == 2) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) r.v[i] = pair_of(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
  } else {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    r.v[0] = pair_of(a.x, a.y); r.v[1] = pair_of(a.z, a.w); r.v[2] = pair_of(b.x, b.y); r.v[3] = pair_of(b.z, b.w);
  }
  return r;
}

struct Level {
  const char *plane, *line;
  float w, h, z;                  // last index along x, y and the line
  uint32_t W, H, Z, cell, row;    // sizes, bytes of a texel and of a row
  unsigned long long block, line_block;
};
template <typename T>
__device__ __forceinline__ Level level_of(const VMLevels& lv, int l) {
  Level v;
  v.plane = reinterpret_cast<const char*>(lv.plane[l]); v.line = reinterpret_cast<const char*>(lv.line[l]);
  v.W = lv.W[l]; v.H = lv.H[l]; v.Z = lv.Z[l];
  v.w = (float)(lv.W[l] - 1); v.h = (float)(lv.H[l] - 1); v.z = (float)(lv.Z[l] - 1);
  v.cell = (uint32_t)lv.C * sizeof(T);
  v.row = v.W * v.cell;
  v.block = (unsigned long long)v.row * v.H;
  v.line_block = (unsigned long long)v.cell * v.Z;
  return v;
}

struct Tap2 { uint32_t i0, i1; float w0, w1; };
// taps() with the size's last index as a float; the same values
__device__ __forceinline__ Tap2 taps_of(float u, uint32_t size, float last) {
  const float f = (u + 1.f) * 0.5f * last;
  const float fl = floorf(f);
  const int i = (int)fl;
  const float t = f - fl;
  Tap2 c;
  c.w0 = (uint32_t)i < size ? 1.f - t : 0.f;
  c.w1 = (uint32_t)(i + 1) < size ? t : 0.f;
  c.i0 = min(max(i, 0), (int)size - 1);
  c.i1 = min(max(i + 1, 0), (int)size - 1);
  return c;
}

// The two factors of channels 8 ch .. 8 ch + 7 of block b: bilinear(plane) and linear(line)
template <typename T>
__device__ __forceinline__ void factors8(const Level& v, const float4& q, int b, int ch, P8& pv, P8& lv, Tap2& cx, Tap2& cy, Tap2& cz) {
  cx = taps_of(q.x, v.W, v.w); cy = taps_of(q.y, v.H, v.h); cz = taps_of(q.z, v.Z, v.z);
  const uint32_t at = (uint32_t)ch * 8 * sizeof(T);
  const char* pl = v.plane + (unsigned long long)(uint32_t)b * v.block + at;
  const char* ln = v.line + (unsigned long long)(uint32_t)b * v.line_block + at;
  const char *x0 = pl + (unsigned long long)cx.i0 * v.cell, *x1 = pl + (unsigned long long)cx.i1 * v.cell;
  const P8 p00 = load_pairs<T>(x0 + (unsigned long long)cy.i0 * v.row), p01 = load_pairs<T>(x1 + (unsigned long long)cy.i0 * v.row);
  const P8 p10 = load_pairs<T>(x0 + (unsigned long long)cy.i1 * v.row), p11 = load_pairs<T>(x1 + (unsigned long long)cy.i1 * v.row);
  const P8 l0 = load_pairs<T>(ln + (unsigned long long)cz.i0 * v.cell), l1 = load_pairs<T>(ln + (unsigned long long)cz.i1 * v.cell);
  const float a = cy.w0 * cx.w0, b01 = cy.w0 * cx.w1, c = cy.w1 * cx.w0, d = cy.w1 * cx.w1;
  const unsigned long long w00 = pair_of(a, a), w01 = pair_of(b01, b01), w10 = pair_of(c, c), w11 = pair_of(d, d);
  const unsigned long long z0 = pair_of(cz.w0, cz.w0), z1 = pair_of(cz.w1, cz.w1);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    pv.v[i] = fma2(w11, p11.v[i], fma2(w10, p10.v[i], fma2(w01, p01.v[i], mul2(w00, p00.v[i]))));
    lv.v[i] = fma2(z1, l1.v[i], mul2(z0, l0.v[i]));
  }
}

template <typename T>
__device__ __forceinline__ P8 lookup8(const Level& v, const float4& q, int b, int ch) {
  P8 pv, lv;
  Tap2 cx, cy, cz;
  factors8<T>(v, q, b, ch, pv, lv, cx, cy, cz);
#pragma unroll
  for (int i = 0; i < 4; ++i) pv.v[i] = mul2(pv.v[i], lv.v[i]);
  return pv;
}

__device__ __forceinline__ void red_add_pairs(float* addr, const P8& g, float w) {
  const unsigned long long ww = pair_of(w, w);
  const float2 a = halves_of(mul2(g.v[0], ww)), b = halves_of(mul2(g.v[1], ww)), c = halves_of(mul2(g.v[2], ww)),
               d = halves_of(mul2(g.v[3], ww));
  red_add_v4(addr, a.x, a.y, b.x, b.y);
  red_add_v4(addr + 4, c.x, c.y, d.x, d.y);
}

// Gradients dp of the plane factor and dl of the line factor to the taps' texels
__device__ __forceinline__ void scatter8(const VMLevels& lv, int l, const Level& v, int b, int ch, const Tap2& cx, const Tap2& cy,
                                         const Tap2& cz, const P8& dp, const P8& dl) {
  const uint32_t C = lv.C, row = v.W * C;
  float* gp = lv.gplane[l] + (unsigned long long)(uint32_t)b * ((unsigned long long)row * v.H) + ch * 8;
  float* gl = lv.gline[l] + (unsigned long long)(uint32_t)b * ((unsigned long long)C * v.Z) + ch * 8;
  float *x0 = gp + (unsigned long long)cx.i0 * C, *x1 = gp + (unsigned long long)cx.i1 * C;
  const float w00 = cy.w0 * cx.w0, w01 = cy.w0 * cx.w1, w10 = cy.w1 * cx.w0, w11 = cy.w1 * cx.w1;
  if (w00 != 0.f) red_add_pairs(x0 + (unsigned long long)cy.i0 * row, dp, w00);
  if (w01 != 0.f) red_add_pairs(x1 + (unsigned long long)cy.i0 * row, dp, w01);
  if (w10 != 0.f) red_add_pairs(x0 + (unsigned long long)cy.i1 * row, dp, w10);
  if (w11 != 0.f) red_add_pairs(x1 + (unsigned long long)cy.i1 * row, dp, w11);
  if (cz.w0 != 0.f) red_add_pairs(gl + (unsigned long long)cz.i0 * C, dl, cz.w0);
  if (cz.w1 != 0.f) red_add_pairs(gl + (unsigned long long)cz.i1 * C, dl, cz.w1);
}

__device__ __forceinline__ void store_pairs(float* p, const P8& r) {
  const float2 a = halves_of(r.v[0]), b = halves_of(r.v[1]), c = halves_of(r.v[2]), d = halves_of(r.v[3]);
  reinterpret_cast<float4*>(p)[0] = make_float4(a.x, a.y, b.x, b.y);
  reinterpret_cast<float4*>(p)[1] = make_float4(c.x, c.y, d.x, d.y);
}
__device__ __forceinline__ void store_pairs(__nv_bfloat16* p, const P8& r) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = halves_of(r.v[i]);
    const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

// Optional 16-column tail of every output row: the viewing direction of the row's ray (3 values) followed by 13 zeros,
// written by the row's first thread as two 16-byte stores.  The colour head reads the direction from there, so the
// row leaves this kernel complete and no separate pass has to patch three 2-byte values into every 320-byte row.
struct DirTail {
  const float* dirs;   // [rays, 3]; null: no tail
  const int* idx;      // row -> flat sample index (ray = idx / samples_per_ray); null: row n reads dirs[n]
  int samples_per_ray;
  int col;             // first tail column, a multiple of 8
};

template <typename T, typename OutT, bool kOne>
__global__ void __launch_bounds__(256, 5)
vm_encode_fwd_kernel(const float4* __restrict__ coords, const int* __restrict__ count_ptr, long long max_n,
                     const __grid_constant__ VMLevels lv, OutT* __restrict__ out, int out_stride, DirTail tail, DivBy by_groups) {
  const int CH = lv.C >> 3;
  const long long n_valid = resolve_count(count_ptr, max_n);
  const bool few = n_valid * CH <= 0x7FFFFFFF;
  // grid-stride: the grid is capped, so a launch sized for a worst-case row capacity costs nothing when
  // the device-side count is small
  for (long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x; tid < n_valid * CH;
       tid += (long long)gridDim.x * blockDim.x) {
  const long long n = few ? (long long)by_groups((uint32_t)tid) : tid / CH;
  int ch = (int)(tid - n * CH);
  float4 q = __ldg(coords + n);
  int b = (int)q.w;
  if (tail.dirs != nullptr && ch == 0) {
    const float* d = tail.dirs + (tail.idx != nullptr ? (long long)(tail.idx[n] / tail.samples_per_ray) : n) * 3;
    F8 a, z;
#pragma unroll
    for (int i = 0; i < 8; ++i) { a.v[i] = 0.f; z.v[i] = 0.f; }
    a.v[0] = d[0]; a.v[1] = d[1]; a.v[2] = d[2];
    store8(out + n * out_stride + tail.col, a);
    store8(out + n * out_stride + tail.col + 8, z);
  }
  if (b < 0 || b >= lv.B) {
    F8 z;
#pragma unroll
    for (int i = 0; i < 8; ++i) z.v[i] = 0.f;
    for (int l = 0; l < lv.L; ++l) store8(out + n * out_stride + l * lv.C + ch * 8, z);
    continue;
  }
  for (int l = 0; l < (kOne ? 1 : lv.L); ++l)
    store_pairs(out + n * out_stride + l * lv.C + ch * 8, lookup8<T>(level_of<T>(lv, kOne ? 0 : l), q, b, ch));
  }
}

// Backward: recompute the taps and both interpolants, then push d(plane) and d(line) with
// 16-byte vector reductions into the fp32 accumulators.
template <typename T, typename GT, bool kOne>
__global__ void __launch_bounds__(256)
vm_encode_bwd_kernel(const float4* __restrict__ coords, const int* __restrict__ count_ptr, long long max_n,
                     const __grid_constant__ VMLevels lv, const GT* __restrict__ dout, int out_stride, DivBy by_groups) {
  const int CH = lv.C >> 3;
  const long long n_valid = resolve_count(count_ptr, max_n);
  const bool few = n_valid * CH <= 0x7FFFFFFF;
  for (long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x; tid < n_valid * CH;
       tid += (long long)gridDim.x * blockDim.x) {
    const long long n = few ? (long long)by_groups((uint32_t)tid) : tid / CH;
    const int ch = (int)(tid - n * CH);
    const float4 q = __ldg(coords + n);
    const int b = (int)q.w;
    if (b < 0 || b >= lv.B) continue;
    for (int l = 0; l < (kOne ? 1 : lv.L); ++l) {
      const Level v = level_of<T>(lv, kOne ? 0 : l);
      const P8 g = load_pairs<GT>(reinterpret_cast<const char*>(dout + n * out_stride + l * lv.C + ch * 8));
      P8 pv, lf;
      Tap2 cx, cy, cz;
      factors8<T>(v, q, b, ch, pv, lf, cx, cy, cz);
      bool any = false;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 h = halves_of(g.v[i]);
        any |= h.x != 0.f || h.y != 0.f;
        lf.v[i] = mul2(g.v[i], lf.v[i]);
        pv.v[i] = mul2(g.v[i], pv.v[i]);
      }
      if (any) scatter8(lv, kOne ? 0 : l, v, b, ch, cx, cy, cz, lf, pv);
    }
  }
}

// ---- atomic-free (deterministic) backward ------------------------------------------------------------------
// Samples are sorted by the texel cell they fall into; one thread owns a whole run of equal cells, sums the run in
// registers in sorted (stable) order and adds the four corner sums to the gradient plane with plain loads and stores.
// Neighbouring cells share corners, so cells are 4-coloured by the parity of (x0, y0) and the colours run as separate
// launches: within a launch no two runs touch the same texel.  Lines are handled the same way with cells sorted by z0,
// two colours, and a warp per run (fixed lane assignment and shuffle tree).  The result is bit-reproducible; the
// default backward (16-byte reductions into L2) is faster and differs only in summation order.
constexpr unsigned long long kNoKey = ~0ull;

__global__ void __launch_bounds__(256)
vm_sort_keys_kernel(const float4* __restrict__ coords, const int* __restrict__ count_ptr, long long max_n, int B, int H, int W, int Z,
                    unsigned long long* __restrict__ pkeys, unsigned* __restrict__ pvals, unsigned long long* __restrict__ zkeys,
                    unsigned* __restrict__ zvals) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= max_n) return;
  const long long n_valid = resolve_count(count_ptr, max_n);
  unsigned long long pk = kNoKey, zk = kNoKey;
  if (n < n_valid) {
    const float4 q = __ldg(coords + n);
    const int b = (int)q.w;
    if (b >= 0 && b < B) {
      const float fx = (q.x + 1.f) * 0.5f * (float)(W - 1), fy = (q.y + 1.f) * 0.5f * (float)(H - 1);
      const float fz = (q.z + 1.f) * 0.5f * (float)(Z - 1);
      const int x0 = min(max((int)floorf(fx), -1), W - 1), y0 = min(max((int)floorf(fy), -1), H - 1);
      const int z0 = min(max((int)floorf(fz), -1), Z - 1);
      pk = ((unsigned long long)b * (H + 1) + (y0 + 1)) * (W + 1) + (x0 + 1);
      zk = (unsigned long long)b * (Z + 1) + (z0 + 1);
    }
  }
  pkeys[n] = pk; pvals[n] = (unsigned)n;
  zkeys[n] = zk; zvals[n] = (unsigned)n;
}

__device__ __forceinline__ void rmw_add8(float* p, const F8& a) {
  float4* q = reinterpret_cast<float4*>(p);
  float4 u = q[0], v = q[1];
  u.x += a.v[0]; u.y += a.v[1]; u.z += a.v[2]; u.w += a.v[3];
  v.x += a.v[4]; v.y += a.v[5]; v.z += a.v[6]; v.w += a.v[7];
  q[0] = u; q[1] = v;
}

template <typename T, typename GT>
__global__ void __launch_bounds__(256)
vm_bwd_sorted_plane_kernel(const float4* __restrict__ coords, VMLevels lv, int l, const GT* __restrict__ dout, int out_stride,
                           const unsigned long long* __restrict__ keys, const unsigned* __restrict__ vals, long long max_n,
                           int colour) {
  const int CH = lv.C >> 3;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long i = tid / CH;
  const int ch = (int)(tid - i * CH);
  if (i >= max_n) return;
  const unsigned long long key = keys[i];
  if (key == kNoKey || (i > 0 && keys[i - 1] == key)) return;          // not the head of a run
  const int H = lv.H[l], W = lv.W[l], Z = lv.Z[l];
  const int x0p = (int)(key % (unsigned long long)(W + 1));
  const unsigned long long t = key / (unsigned long long)(W + 1);
  const int y0p = (int)(t % (unsigned long long)(H + 1));
  const int b = (int)(t / (unsigned long long)(H + 1));
  if (((x0p & 1) | ((y0p & 1) << 1)) != colour) return;
  F8 a00, a01, a10, a11;
#pragma unroll
  for (int k = 0; k < 8; ++k) a00.v[k] = a01.v[k] = a10.v[k] = a11.v[k] = 0.f;
  const T* ln = reinterpret_cast<const T*>(lv.line[l]) + ((long long)b * Z) * lv.C + ch * 8;
  for (long long j = i; j < max_n && keys[j] == key; ++j) {
    const long long n = vals[j];
    const float4 q = __ldg(coords + n);
    const Corner2 cx = taps(q.x, W), cy = taps(q.y, H), cz = taps(q.z, Z);
    const F8 l0 = load8(ln + (long long)cz.i0 * lv.C), l1 = load8(ln + (long long)cz.i1 * lv.C);
    const F8 g = load8(dout + n * out_stride + l * lv.C + ch * 8);
    const float w00 = cy.w0 * cx.w0, w01 = cy.w0 * cx.w1, w10 = cy.w1 * cx.w0, w11 = cy.w1 * cx.w1;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float dp = g.v[k] * (cz.w0 * l0.v[k] + cz.w1 * l1.v[k]);
      a00.v[k] += dp * w00; a01.v[k] += dp * w01; a10.v[k] += dp * w10; a11.v[k] += dp * w11;
    }
  }
  const int x0 = x0p - 1, y0 = y0p - 1;
  float* gp = lv.gplane[l] + ((long long)b * H * W) * lv.C + ch * 8;
  const bool xa = x0 >= 0, xb = x0 + 1 < W, ya = y0 >= 0, yb = y0 + 1 < H;
  if (ya && xa) rmw_add8(gp + ((long long)y0 * W + x0) * lv.C, a00);
  if (ya && xb) rmw_add8(gp + ((long long)y0 * W + x0 + 1) * lv.C, a01);
  if (yb && xa) rmw_add8(gp + ((long long)(y0 + 1) * W + x0) * lv.C, a10);
  if (yb && xb) rmw_add8(gp + ((long long)(y0 + 1) * W + x0 + 1) * lv.C, a11);
}

__device__ __forceinline__ long long lower_bound_u64(const unsigned long long* a, long long n, unsigned long long v) {
  long long lo = 0, hi = n;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (a[mid] < v) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// one warp per (z cell, channel group)
template <typename T, typename GT>
__global__ void __launch_bounds__(256)
vm_bwd_sorted_line_kernel(const float4* __restrict__ coords, VMLevels lv, int l, const GT* __restrict__ dout, int out_stride,
                          const unsigned long long* __restrict__ keys, const unsigned* __restrict__ vals, long long max_n,
                          int colour) {
  const int CH = lv.C >> 3;
  const int H = lv.H[l], W = lv.W[l], Z = lv.Z[l];
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long cell = warp / CH;
  const int ch = (int)(warp - cell * CH);
  if (cell >= (long long)lv.B * (Z + 1)) return;
  const int z0p = (int)(cell % (Z + 1));
  if ((z0p & 1) != colour) return;
  const int b = (int)(cell / (Z + 1));
  const long long start = lower_bound_u64(keys, max_n, (unsigned long long)cell);
  const long long end = lower_bound_u64(keys, max_n, (unsigned long long)cell + 1);
  F8 a0, a1;
#pragma unroll
  for (int k = 0; k < 8; ++k) a0.v[k] = a1.v[k] = 0.f;
  const T* pl = reinterpret_cast<const T*>(lv.plane[l]) + ((long long)b * H * W) * lv.C + ch * 8;
  for (long long j = start + lane; j < end; j += 32) {
    const long long n = vals[j];
    const float4 q = __ldg(coords + n);
    const Corner2 cx = taps(q.x, W), cy = taps(q.y, H), cz = taps(q.z, Z);
    const F8 p00 = load8(pl + ((long long)cy.i0 * W + cx.i0) * lv.C), p01 = load8(pl + ((long long)cy.i0 * W + cx.i1) * lv.C);
    const F8 p10 = load8(pl + ((long long)cy.i1 * W + cx.i0) * lv.C), p11 = load8(pl + ((long long)cy.i1 * W + cx.i1) * lv.C);
    const F8 g = load8(dout + n * out_stride + l * lv.C + ch * 8);
    const float w00 = cy.w0 * cx.w0, w01 = cy.w0 * cx.w1, w10 = cy.w1 * cx.w0, w11 = cy.w1 * cx.w1;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float dl = g.v[k] * (w00 * p00.v[k] + w01 * p01.v[k] + w10 * p10.v[k] + w11 * p11.v[k]);
      a0.v[k] += dl * cz.w0; a1.v[k] += dl * cz.w1;
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k)
    for (int o = 16; o > 0; o >>= 1) {
      a0.v[k] += __shfl_xor_sync(0xffffffffu, a0.v[k], o);
      a1.v[k] += __shfl_xor_sync(0xffffffffu, a1.v[k], o);
    }
  if (lane != 0 || start == end) return;
  const int z0 = z0p - 1;
  float* gl = lv.gline[l] + ((long long)b * Z) * lv.C + ch * 8;
  if (z0 >= 0) rmw_add8(gl + (long long)z0 * lv.C, a0);
  if (z0 + 1 < Z) rmw_add8(gl + (long long)(z0 + 1) * lv.C, a1);
}

// ---- fused density head --------------------------------------------------------------------------
// sigma = act(relu?(sum_c w_c * feature_c)): the lookup, the 1-wide linear layer (or plain channel sum)
// and the activation of the reference's density path (benchmarks/nerf/gridnerf/gridnerf.py:177-197,
// compute_densityfeature + feature2density) in one kernel; the [N, L*C] feature matrix is never written.
// The C/8 threads of a sample are adjacent lanes (C/8 must be a power of two <= 32).
struct DensityHead {
  const float* w;     // [L*C] weights of the 1-wide linear layer, or nullptr for a plain sum
  int inner_relu;     // relu between the linear layer and the activation
  int act;            // 0 relu, 1 softplus(x + shift)
  float shift;
};

// Spatial-block model parallelism: the rows of an owner's batch came from other GPUs (all-to-all dispatch); row n
// belongs to rank route_src[n], which expects its density at slot route_slot[n] of its landing buffer dest[src].
// With a route the density kernel stores sigma there itself (a peer store over NVLink) - the "combine" half of the
// exchange costs no kernel of its own.
struct DensityRoute {
  const int* src;     // nullptr: no route
  const int* slot;
  float* dest[8];
};

template <typename T, bool kOne>
__global__ void __launch_bounds__(256, 5)
vm_density_fwd_kernel(const float4* __restrict__ coords, const int* __restrict__ count_ptr, long long max_n,
                      const __grid_constant__ VMLevels lv, DensityHead head, float* __restrict__ sigma, float* __restrict__ pre,
                      const __grid_constant__ DensityRoute route) {
  const int CH = lv.C >> 3, ch_bits = __ffs(CH) - 1;                  // a power of two
  const long long n_valid = resolve_count(count_ptr, max_n);
  // grid-stride with a trip count that is uniform per block (the shuffles below need whole warps)
  for (long long base = (long long)blockIdx.x * blockDim.x; base < n_valid * CH; base += (long long)gridDim.x * blockDim.x) {
  const long long tid = base + threadIdx.x;
  const long long n = tid >> ch_bits;
  const int ch = (int)tid & (CH - 1);
  const bool live = n < n_valid;
  float acc = 0.f;
  if (live) {
    const float4 q = __ldg(coords + n);
    const int b = (int)q.w;
    if (b >= 0 && b < lv.B) {
      for (int l = 0; l < (kOne ? 1 : lv.L); ++l) {
        const P8 f = lookup8<T>(level_of<T>(lv, kOne ? 0 : l), q, b, ch);
        const float* w = head.w ? head.w + l * lv.C + ch * 8 : nullptr;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 v = halves_of(f.v[i]);
          acc += v.x * (w ? __ldg(w + 2 * i) : 1.f);
          acc += v.y * (w ? __ldg(w + 2 * i + 1) : 1.f);
        }
      }
    }
  }
  for (int o = CH >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (live && ch == 0) {
    const float r = head.inner_relu ? fmaxf(acc, 0.f) : acc;
    const float x = r + head.shift;
    const float sg = head.act == 0 ? fmaxf(r, 0.f) : (x > 20.f ? x : log1pf(__expf(x)));
    sigma[n] = sg;
    pre[n] = acc;
    if (route.src != nullptr) route.dest[route.src[n]][route.slot[n]] = sg;
  }
  }
}

// dsigma [N] -> plane / line gradient accumulators (as vm_encode_bwd) and dw [L*C].  With one level a thread's channels are the same
// for all of its samples: their sums stay in registers and meet in shared memory once; the grid is kept small for that.  8192 rays of
// 128 samples on 4096^2 texels 115 -> 101 us, on 1371^2 97 -> 65; what is left are the reductions into the planes.
template <typename T, bool kOne>
__global__ void __launch_bounds__(256)
vm_density_bwd_kernel(const float4* __restrict__ coords, const int* __restrict__ count_ptr, long long max_n,
                      const __grid_constant__ VMLevels lv, DensityHead head, const float* __restrict__ dsigma,
                      const float* __restrict__ pre, float* __restrict__ dw) {
  extern __shared__ float dw_sh[];               // [L*C]
  const int CH = lv.C >> 3, ch_bits = __ffs(CH) - 1;                  // a power of two
  const int n_w = lv.L * lv.C;
  const bool weights = head.w != nullptr && dw != nullptr;
  for (int i = threadIdx.x; i < n_w; i += blockDim.x) dw_sh[i] = 0.f;
  __syncthreads();
  const long long n_valid = resolve_count(count_ptr, max_n);
  const int lane = threadIdx.x & 31;
  float sums[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) sums[i] = 0.f;
  // lanes with the same channel group are CH apart: fold them, then one shared-memory atomic per warp
  auto fold = [&](int l) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float v = sums[i];
      for (int o = CH; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane < CH) atomicAdd(&dw_sh[l * lv.C + (lane & (CH - 1)) * 8 + i], v);
    }
  };
  for (long long base = (long long)blockIdx.x * blockDim.x; base < n_valid * CH; base += (long long)gridDim.x * blockDim.x) {
    const long long tid = base + threadIdx.x;
    const long long n = tid >> ch_bits;
    const int ch = (int)tid & (CH - 1);
    bool live = n < n_valid;
    float4 q = make_float4(0.f, 0.f, 0.f, -1.f);
    float dz = 0.f;
    if (live) {
      q = __ldg(coords + n);
      const int b = (int)q.w;
      live = b >= 0 && b < lv.B;
      if (live) {
        const float z = pre[n];
        const float r = head.inner_relu ? fmaxf(z, 0.f) : z;
        const float dact = head.act == 0 ? (r > 0.f ? 1.f : 0.f) : __fdividef(1.f, 1.f + __expf(-(r + head.shift)));
        dz = dsigma[n] * dact * ((head.inner_relu && z <= 0.f) ? 0.f : 1.f);
      }
    }
    for (int l = 0; l < (kOne ? 1 : lv.L); ++l) {
      if (!kOne) {
#pragma unroll
        for (int i = 0; i < 8; ++i) sums[i] = 0.f;
      }
      if (live && dz != 0.f) {
        const int b = (int)q.w;
        const Level v = level_of<T>(lv, kOne ? 0 : l);
        P8 pv, lf;
        Tap2 cx, cy, cz;
        factors8<T>(v, q, b, ch, pv, lf, cx, cy, cz);
        const float* w = head.w ? head.w + l * lv.C + ch * 8 : nullptr;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = halves_of(mul2(pv.v[i], lf.v[i]));
          sums[2 * i] += dz * f.x; sums[2 * i + 1] += dz * f.y;
          const unsigned long long g = pair_of(dz * (w ? __ldg(w + 2 * i) : 1.f), dz * (w ? __ldg(w + 2 * i + 1) : 1.f));
          lf.v[i] = mul2(g, lf.v[i]);
          pv.v[i] = mul2(g, pv.v[i]);
        }
        scatter8(lv, kOne ? 0 : l, v, b, ch, cx, cy, cz, lf, pv);
      }
      if (!kOne && weights) fold(l);
    }
  }
  if (!weights) return;
  if (kOne) fold(0);
  __syncthreads();
  for (int i = threadIdx.x; i < n_w; i += blockDim.x)
    if (dw_sh[i] != 0.f) atomicAdd(dw + i, dw_sh[i]);
}

}  // namespace lmb

using namespace lmb;

// enough blocks to fill the GPU several times over, never more than the work needs
static int capped_grid(long long work_items, int threads) {
  const long long want = (work_items + threads - 1) / threads;
  const long long cap = 148LL * 64;
  return (int)(want < cap ? (want > 0 ? want : 1) : cap);
}

// param_dtype / io_dtype: 0 = fp32, 1 = bf16.
// tail_dirs (may be null): see DirTail; tail_col must be a multiple of 8 with tail_col + 16 <= the row stride.
LMB_API int lmb_vm_encode_fwd(const float* coords, const int* count_ptr, long long max_n, const VMLevels* levels,
                              int param_dtype, void* out, int out_dtype, int out_stride, const float* tail_dirs,
                              const int* tail_idx, int tail_samples_per_ray, int tail_col, cudaStream_t stream) {
  if (max_n <= 0) return 0;
  if (levels->C % 8 != 0 || levels->L < 1 || levels->L > kMaxLevels) return (int)cudaErrorInvalidValue;
  const int CH = levels->C / 8;
  const int threads = 256;
  const int blocks = capped_grid(max_n * CH, threads);
  const float4* c4 = reinterpret_cast<const float4*>(coords);
  const int stride = out_stride > 0 ? out_stride : levels->L * levels->C;
  const DirTail tail{tail_dirs, tail_idx, tail_samples_per_ray > 0 ? tail_samples_per_ray : 1, tail_col};
  if (tail_dirs != nullptr && (tail_col % 8 != 0 || tail_col < levels->L * levels->C || tail_col + 16 > stride))
    return (int)cudaErrorInvalidValue;
#define LAUNCH(T, O) (levels->L == 1 ? vm_encode_fwd_kernel<T, O, true> : vm_encode_fwd_kernel<T, O, false>)<<<blocks, threads, 0, stream>>>(c4, count_ptr, max_n, *levels, (O*)out, stride, tail, DivBy(levels->C >> 3))
  if (param_dtype == 0 && out_dtype == 0) LAUNCH(float, float);
  else if (param_dtype == 0 && out_dtype == 1) LAUNCH(float, __nv_bfloat16);
  else if (param_dtype == 1 && out_dtype == 0) LAUNCH(__nv_bfloat16, float);
  else LAUNCH(__nv_bfloat16, __nv_bfloat16);
#undef LAUNCH
  LMB_LAUNCH_CHECK();
  return 0;
}

LMB_API int lmb_vm_encode_bwd(const float* coords, const int* count_ptr, long long max_n, const VMLevels* levels,
                              int param_dtype, const void* dout, int dout_dtype, int dout_stride, cudaStream_t stream) {
  if (max_n <= 0) return 0;
  if (levels->C % 8 != 0 || levels->L < 1 || levels->L > kMaxLevels) return (int)cudaErrorInvalidValue;
  const int CH = levels->C / 8;
  const int threads = 256;
  const int blocks = capped_grid(max_n * CH, threads);
  const float4* c4 = reinterpret_cast<const float4*>(coords);
#define LAUNCH(T, G) (levels->L == 1 ? vm_encode_bwd_kernel<T, G, true> : vm_encode_bwd_kernel<T, G, false>)<<<blocks, threads, 0, stream>>>( \
    c4, count_ptr, max_n, *levels, (const G*)dout, dout_stride > 0 ? dout_stride : levels->L * levels->C, DivBy(levels->C >> 3))
  if (param_dtype == 0 && dout_dtype == 0) LAUNCH(float, float);
  else if (param_dtype == 0 && dout_dtype == 1) LAUNCH(float, __nv_bfloat16);
  else if (param_dtype == 1 && dout_dtype == 0) LAUNCH(__nv_bfloat16, float);
  else LAUNCH(__nv_bfloat16, __nv_bfloat16);
#undef LAUNCH
  LMB_LAUNCH_CHECK();
  return 0;
}

static bool density_shape_ok(const VMLevels* lv) {
  const int CH = lv->C / 8;
  return lv->C % 8 == 0 && lv->L >= 1 && lv->L <= kMaxLevels && CH >= 1 && CH <= 32 && (CH & (CH - 1)) == 0;
}

// sigma, pre: fp32 [max_n]; w: fp32 [L*C] or null (plain channel sum); act: 0 relu, 1 softplus(x + shift)
// route_src / route_slot / dest_table (all null, or int [max_n] x 2 and `world` landing-buffer addresses): see DensityRoute
LMB_API int lmb_vm_density_fwd(const float* coords, const int* count_ptr, long long max_n, const VMLevels* levels,
                               int param_dtype, const float* w, int inner_relu, int act, float shift, float* sigma, float* pre,
                               const int* route_src, const int* route_slot, const long long* dest_table, int world,
                               cudaStream_t stream) {
  if (max_n <= 0) return 0;
  if (!density_shape_ok(levels) || (route_src != nullptr && (dest_table == nullptr || world > 8))) return (int)cudaErrorInvalidValue;
  const DensityHead head{w, inner_relu, act, shift};
  DensityRoute route;
  route.src = route_src; route.slot = route_slot;
  for (int i = 0; i < 8; ++i) route.dest[i] = (route_src != nullptr && i < world) ? (float*)dest_table[i] : nullptr;
  const int blocks = capped_grid(max_n * (levels->C / 8), 256);
  const float4* c4 = reinterpret_cast<const float4*>(coords);
  const bool one = levels->L == 1;
  const auto kernel = param_dtype == 0 ? (one ? vm_density_fwd_kernel<float, true> : vm_density_fwd_kernel<float, false>)
                                       : (one ? vm_density_fwd_kernel<__nv_bfloat16, true> : vm_density_fwd_kernel<__nv_bfloat16, false>);
  kernel<<<blocks, 256, 0, stream>>>(c4, count_ptr, max_n, *levels, head, sigma, pre, route);
  LMB_LAUNCH_CHECK();
  return 0;
}

// dw: fp32 [L*C] accumulator (may be null when w is null)
LMB_API int lmb_vm_density_bwd(const float* coords, const int* count_ptr, long long max_n, const VMLevels* levels,
                               int param_dtype, const float* w, int inner_relu, int act, float shift, const float* dsigma,
                               const float* pre, float* dw, cudaStream_t stream) {
  if (max_n <= 0) return 0;
  if (!density_shape_ok(levels)) return (int)cudaErrorInvalidValue;
  const DensityHead head{w, inner_relu, act, shift};
  const int blocks = capped_grid(max_n * (levels->C / 8), 256);
  const size_t smem = sizeof(float) * levels->L * levels->C;
  const float4* c4 = reinterpret_cast<const float4*>(coords);
  const bool one = levels->L == 1;
  const auto kernel = param_dtype == 0 ? (one ? vm_density_bwd_kernel<float, true> : vm_density_bwd_kernel<float, false>)
                                       : (one ? vm_density_bwd_kernel<__nv_bfloat16, true> : vm_density_bwd_kernel<__nv_bfloat16, false>);
  kernel<<<one && blocks > 148 * 8 ? 148 * 8 : blocks, 256, smem, stream>>>(c4, count_ptr, max_n, *levels, head, dsigma, pre, dw);
  LMB_LAUNCH_CHECK();
  return 0;
}

extern "C" int lmb_radix_sort_pairs(uint64_t* keys, uint32_t* vals, const int* count_ptr, long long max_n, int begin_bit, int end_bit,
                                    void* scratch, cudaStream_t stream);

static int bits_for(unsigned long long n_keys) {      // enough bits that the all-ones "no key" sorts after every real key
  int bits = 1;
  while ((1ull << bits) <= n_keys) ++bits;
  return bits;
}

// Deterministic backward.  pkeys / zkeys: uint64 [max_n]; pvals / zvals: uint32 [max_n]; sort_scratch: lmb_radix_sort_scratch_bytes(max_n).
LMB_API int lmb_vm_encode_bwd_sorted(const float* coords, const int* count_ptr, long long max_n, const VMLevels* levels,
                                     int param_dtype, const void* dout, int dout_dtype, int dout_stride, uint64_t* pkeys,
                                     uint32_t* pvals, uint64_t* zkeys, uint32_t* zvals, void* sort_scratch, cudaStream_t stream) {
  if (max_n <= 0) return 0;
  if (levels->C % 8 != 0 || levels->L < 1 || levels->L > kMaxLevels) return (int)cudaErrorInvalidValue;
  const int CH = levels->C / 8;
  const float4* c4 = reinterpret_cast<const float4*>(coords);
  const int stride = dout_stride > 0 ? dout_stride : levels->L * levels->C;
  for (int l = 0; l < levels->L; ++l) {
    const int H = levels->H[l], W = levels->W[l], Z = levels->Z[l], B = levels->B;
    vm_sort_keys_kernel<<<ceil_div(max_n, 256), 256, 0, stream>>>(c4, count_ptr, max_n, B, H, W, Z, (unsigned long long*)pkeys, pvals,
                                                                 (unsigned long long*)zkeys, zvals);
    LMB_LAUNCH_CHECK();
    int rc = lmb_radix_sort_pairs(pkeys, pvals, nullptr, max_n, 0, bits_for((unsigned long long)B * (H + 1) * (W + 1)), sort_scratch, stream);
    if (rc) return rc;
    rc = lmb_radix_sort_pairs(zkeys, zvals, nullptr, max_n, 0, bits_for((unsigned long long)B * (Z + 1)), sort_scratch, stream);
    if (rc) return rc;
    const int pblocks = ceil_div(max_n * CH, 256);
    const int lblocks = ceil_div((long long)B * (Z + 1) * CH * 32, 256);
#define LAUNCH(T, G)                                                                                                              \
    for (int colour = 0; colour < 4; ++colour)                                                                                    \
      vm_bwd_sorted_plane_kernel<T, G><<<pblocks, 256, 0, stream>>>(c4, *levels, l, (const G*)dout, stride,                       \
                                                                   (const unsigned long long*)pkeys, pvals, max_n, colour);      \
    for (int colour = 0; colour < 2; ++colour)                                                                                    \
      vm_bwd_sorted_line_kernel<T, G><<<lblocks, 256, 0, stream>>>(c4, *levels, l, (const G*)dout, stride,                        \
                                                                  (const unsigned long long*)zkeys, zvals, max_n, colour);
    if (param_dtype == 0 && dout_dtype == 0) { LAUNCH(float, float) }
    else if (param_dtype == 0 && dout_dtype == 1) { LAUNCH(float, __nv_bfloat16) }
    else if (param_dtype == 1 && dout_dtype == 0) { LAUNCH(__nv_bfloat16, float) }
    else { LAUNCH(__nv_bfloat16, __nv_bfloat16) }
#undef LAUNCH
    LMB_LAUNCH_CHECK();
  }
  return 0;
}
